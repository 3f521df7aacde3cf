"""Products on the warp-level tensor path for the shapes and block types that the TMA kernels do not
take, at its edges: rows of one block and of a piece and a bit, row groups that are not full, more
row groups than a wave, batches around a pass of 8 and of 16, tensors at an address that is only
even, each store.

The bound: every weight is s * q + o with q and the products q * x exact, so a sum is off by what its
float additions and the scalings round, at most (k + 8) * 2^-23 of the sum of the magnitudes
|s q x| + |o x| (2^-23: an addition on the tensor path may truncate)."""
import numpy as np
import pytest

import _blocks
from _util import GUARD, dev, torch_mod

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import aotx_b200
    c = aotx_b200.Q8Context(0)
    yield c
    assert c.device_status() == 0
    c.close()


@pytest.fixture(scope="module")
def decoder(tmp_path_factory):
    return _blocks.HostDecoder(tmp_path_factory.mktemp("decoder"))


def at_offset(w, offset):
    """The bytes on the device, `offset` bytes past a 256-byte boundary."""
    torch = torch_mod()
    room = torch.zeros(w.size + 512, dtype=torch.uint8, device="cuda")
    skip = (-room.data_ptr()) % 256 + offset
    room[skip:skip + w.size] = torch.from_numpy(w).cuda()
    return room[skip:skip + w.size]


@pytest.mark.parametrize("kind", [8, 2, 3, 6, 7, 12, 13, 14])
@pytest.mark.parametrize("n,runs,m,offset", [(1, 1, 1, 0), (17, 3, 8, 4), (33, 37, 9, 8), (4800, 9, 17, 0), (40, 8, 5, 2)])
def test_product(ctx, decoder, kind, n, runs, m, offset):
    torch = torch_mod()
    k = runs * (256 if kind >= 10 else 32)
    rng = np.random.Generator(np.random.PCG64(n + kind))
    rows = min(n, 64)                       # decoded once, repeated down the tensor
    some = _blocks.random_rows(kind, rows, k, rng).reshape(rows, -1)
    w_host = np.resize(some, (n, some.shape[1])) if n > rows else some
    values = torch.from_numpy(np.resize(decoder.rows(kind, some.reshape(-1), rows, k), (n, k))).cuda().double()
    w = at_offset(np.ascontiguousarray(w_host).reshape(-1), offset)
    for x_kind in (torch.float16, torch.bfloat16):
        x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(x_kind).cuda()
        y = torch.full((m + 1, n), GUARD, device="cuda")
        ctx.set_path(1 if kind == 8 else 0)
        ctx.matmul(w, n, k, x, y=y[:m], type=kind)
        ctx.set_path(0)
        want = x.double() @ values.T
        # the magnitudes of scale and offset parts are at most a few times the largest weight of the row
        bound = (k + 8) * 2.0 ** -23 * 4.0 * x.double().abs() @ (values.abs().amax(dim=1, keepdim=True).expand(n, k)).T + 1e-30
        assert bool(((y[:m].double() - want).abs() <= bound).all())
        assert bool((y[m] == GUARD).all())
        half = torch.empty((m, n), device="cuda", dtype=torch.bfloat16)
        ctx.set_path(1 if kind == 8 else 0)
        ctx.matmul(w, n, k, x, y=half, type=kind)
        ctx.set_path(0)
        assert torch.equal(half, y[:m].bfloat16())


@pytest.mark.parametrize("n,k,m", [(18, 96, 3), (5002, 2912, 11)])
def test_fused_stores(ctx, n, k, m):
    import aotx_b200
    torch = torch_mod()
    w = aotx_b200.synth_q8_0_device(n, k, 5)
    x = dev(np.random.Generator(np.random.PCG64(6)).standard_normal((m, k)).astype(np.float16))
    y = ctx.matmul(w, n, k, x)
    live = torch.tensor([m - 1], dtype=torch.int32, device="cuda")
    base = torch.randn(m, n, device="cuda")
    r = base.clone()
    ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_ADD, m=m, m_dev=live, y=r)
    assert torch.equal(r[:m - 1], base[:m - 1] + y[:m - 1]) and torch.equal(r[m - 1:], base[m - 1:])
    g = ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_SWIGLU).double()
    gate, up = y[:, 0::2].double(), y[:, 1::2].double()
    unit = gate / (1.0 + torch.exp(-gate)) * up
    assert bool(((g - unit).abs() <= 2.0 ** -20 * unit.abs() + 1e-12).all())   # expf and three float roundings


# one piece per thread up to 591 * 1024 pieces of 8 weights, four from there on; a last block that is full, and not
@pytest.mark.parametrize("rows,k", [(1, 32), (2327, 2080), (2332, 2080), (592, 8192), (593, 8192), (1999, 4064)])
def test_dequant_exact_on_both_sides_of_the_line(ctx, rows, k):
    import aotx_b200
    torch = torch_mod()
    w = aotx_b200.synth_q8_0_device(rows, k, rows)
    raw = w.view(-1, 34)
    d = raw[:, :2].contiguous().view(torch.float16)
    want = (raw[:, 2:].contiguous().view(torch.int8).half() * d).view(rows, k)    # rounded once, like the kernel
    assert torch.equal(ctx.dequant(w, k, 0, rows), want)
    # a result that starts between 16-byte boundaries, and nothing written around it
    store = torch.full((rows * k + 4,), GUARD, device="cuda", dtype=torch.float16)
    ctx.dequant(w, k, 0, rows, out=store[2:2 + rows * k].view(rows, k))
    assert torch.equal(store[2:2 + rows * k].view(rows, k), want)
    assert bool((store[:2] == store[-1]).all()) and bool((store[-2:] == GUARD).all())


@pytest.mark.parametrize("kind,n,k,m", [(8, 33, 1184, 7), (8, 50, 96, 12), (12, 40, 512, 5), (13, 17, 256, 8), (2, 18, 160, 3)])
def test_x_between_16_byte_boundaries(ctx, kind, n, k, m):
    """The two ways to load x take the same weights into the same sums."""
    torch = torch_mod()
    w = dev(_blocks.random_rows(kind, n, k, np.random.Generator(np.random.PCG64(n))).reshape(-1))
    room = torch.randn(m * k + 4, device="cuda").half()
    shifted = room[4:].view(m, k)                 # 8 bytes past a boundary
    ctx.set_path(1 if kind == 8 else 0)
    a = ctx.matmul(w, n, k, shifted, type=kind)
    b = ctx.matmul(w, n, k, shifted.clone(), type=kind)
    ctx.set_path(0)
    assert torch.equal(a, b)
