"""Products of up to 5 rows at the sizes where the kernel that takes whole rows of w can go wrong, and at the edges of its
range: tiles of 11 rows and of sixteen and the sizes next to them, the least and the largest depth and the ones next to them,
segments that eight warps do not share evenly, rows of x on both sides of its last, a live batch, each store.

The bound: k additions in any order are off by at most k * 2^-23 times the sum of the magnitudes, and half a step of the
type that is stored.  (test_gpu_s_sum_errors.py holds the same kernel to the 2-norm that its chains give.)"""
import ctypes

import pytest

from _util import torch_mod

pytestmark = pytest.mark.gpu

PLACES = 296   # blocks at a time


def served(n, k, m, epilogue=0):
    """Whether the library's rule gives the product to that kernel, on 148 SMs."""
    import aotx_b200.library as library
    rule = ctypes.CDLL(library.LIB_PATH)._ZN2q811rows_heightEjjjjj
    return rule(n, k, m, 148, epilogue) != 0


@pytest.fixture(scope="module")
def ctx():
    import aotx_b200
    c = aotx_b200.Q8Context(0)
    yield c
    assert c.device_status() == 0
    c.close()


def data(ctx, n, k, m, dtype):
    import aotx_b200
    torch = torch_mod()
    w = aotx_b200.synth_q8_0_device(n, k, n + m)
    x = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n + k + m)).to(dtype)
    wd, xd = ctx.dequant(w, k, 0, n).double(), x.half().double()
    return w, x, xd @ wd.T, k * 2.0 ** -23 * (xd.abs() @ wd.abs().T) + 1e-30


# (rows of w, served with depths up to 4096, served above)
ROWS = [(10 * PLACES, False, False), (10 * PLACES + 1, True, False), (3333, True, False), (4095, True, False), (4096, True, False),
        (4097, True, True), (4600, True, True), (16 * PLACES, True, True), (16 * PLACES + 1, False, False)]
# (depth, rows of x, whether the rule takes them)
DEPTHS = [(1792, 4, False), (2048, 1, True), (2304, 4, True), (4096, 3, True), (4352, 1, True), (9216, 2, True), (16384, 1, True),
          (16384, 4, True), (16640, 2, False), (2048, 5, False)]


@pytest.mark.parametrize("n,shallow,deep", ROWS)
@pytest.mark.parametrize("k,m,taken", DEPTHS)
def test_edges_of_the_tiles(ctx, n, shallow, deep, k, m, taken):
    assert served(n, k, m) == (taken and (shallow if k <= 4096 else deep))
    torch = torch_mod()
    w, x, want, bound = data(ctx, n, k, m, torch.float16)
    first = None
    for _ in range(3):
        y = torch.full((m + 1, n), 7.0, device="cuda")
        ctx.matmul(w, n, k, x, y=y)
        assert first is None or torch.equal(first, y)
        first = y
    assert bool(((y[:m].double() - want).abs() <= bound).all())
    assert bool((y[m:] == 7.0).all())


@pytest.mark.parametrize("m", [1, 4, 5])
@pytest.mark.parametrize("n,k", [(3072, 2048), (4096, 4096), (4609, 9216), (16 * PLACES, 16384)])
@pytest.mark.parametrize("x_type,y_type,step", [("float16", "float16", 2.0 ** -11), ("bfloat16", "bfloat16", 2.0 ** -8),
                                                ("bfloat16", "float32", 0.0)])
def test_types_and_batches(ctx, n, k, m, x_type, y_type, step):
    torch = torch_mod()
    assert served(n, k, m) == (m <= 4)
    w, x, want, bound = data(ctx, n, k, m, getattr(torch, x_type))
    got = ctx.matmul(w, n, k, x, y_dtype=getattr(torch, y_type)).double()
    assert bool(((got - want).abs() <= bound + step * (want.abs() + bound) + 2.0 ** -24).all())


@pytest.mark.parametrize("n,k,m", [(2962, 2304, 2), (3458, 2816, 3), (4736, 2048, 1), (4096, 4096, 4), (14 * PLACES, 14336, 4),
                                   (16 * PLACES, 16384, 1)])
def test_stores_and_live_batch(ctx, n, k, m):
    import aotx_b200
    torch = torch_mod()
    assert served(n, k, m, aotx_b200.EPILOGUE_ADD) and served(n, k, m, aotx_b200.EPILOGUE_SWIGLU)
    w, x, want, bound = data(ctx, n, k, m, torch.float16)
    for live in sorted({m, m - 1, 0}):
        word = torch.tensor([live], dtype=torch.int32, device="cuda")
        y = torch.full((m, n), 3.0, device="cuda")
        ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_ADD, m=m, m_dev=word, y=y)
        assert bool(((y.double() - 3.0 - want).abs() <= bound + 2.0 ** -23 * (want.abs() + 3.0))[:live].all())
        assert bool((y[live:] == 3.0).all())
        z = torch.full((m, n // 2), 3.0, device="cuda")
        ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_SWIGLU, m=m, m_dev=word, y=z)
        gate, up = want[:, 0::2], want[:, 1::2]
        unit = gate / (1 + torch.exp(-gate)) * up
        # |silu'| is at most 1.1, and |silu| at most the gate's magnitude; both factors' errors, and roundings
        off = 1.1 * bound[:, 0::2] * (up.abs() + bound[:, 1::2]) + gate.abs() * bound[:, 1::2] + 2.0 ** -20 * unit.abs() + 1e-30
        assert bool(((z.double() - unit).abs() <= off)[:live].all())
        assert bool((z[live:] == 3.0).all())
