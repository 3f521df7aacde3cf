"""Products of small batches at the sizes where the kernel that serves them can go wrong: the edges
of its token tiles (8, 16), row tiles that are not full, one segment of depth and many, one
cluster per row tile (few rows) and tiles cut between blocks (many), each of its stores.

The bound: products of two binary16 values are exact in float, and k float additions in any order
are off by at most k * 2^-23 times the sum of the magnitudes (2^-23: an addition may truncate)."""
import pytest

from _util import GUARD, torch_mod

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import aotx_b200
    c = aotx_b200.Q8Context(0)
    yield c
    assert c.device_status() == 0
    c.close()


def sums(ctx, w, n, k, x):
    """The exact products in float64 and the bound of their float sums."""
    wd = ctx.dequant(w, k, 0, n).double()
    xd = x.double()
    return xd @ wd.T, k * 2.0 ** -23 * (xd.abs() @ wd.abs().T) + 1e-30


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 256), (129, 256), (1023, 2048), (9473, 512), (20011, 768)])
def test_every_store(ctx, n, k, m):
    import aotx_b200
    torch = torch_mod()
    w = aotx_b200.synth_q8_0_device(n, k, n + k + m)
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    want, bound = sums(ctx, w, n, k, x)
    y = torch.full((m + 1, n), GUARD, device="cuda")
    ctx.matmul(w, n, k, x, y=y[:m])
    assert bool(((y[:m].double() - want).abs() <= bound).all()) and bool((y[m] == GUARD).all())
    # 16-bit results are the same float sums, rounded once
    for kind in (torch.float16, torch.bfloat16):
        z = torch.full((m + 1, n), GUARD, device="cuda", dtype=kind)
        ctx.matmul(w, n, k, x, y=z[:m])
        assert torch.equal(z[:m], y[:m].to(kind)), "the same float sums, rounded"
        assert bool((z[m] == torch.tensor(GUARD, dtype=kind)).all())
    # bfloat16 activations inside the range that binary16 holds exactly give the same sums
    xb = x.bfloat16()
    exact = xb.half()
    assert torch.equal(ctx.matmul(w, n, k, xb), ctx.matmul(w, n, k, exact)) or bool((exact.float() != xb.float()).any())
    # residual add, and only the live rows
    live = torch.tensor([max(1, m - 1)], dtype=torch.int32, device="cuda")
    base = torch.randn(m, n, device="cuda", generator=gen)
    r = base.clone()
    ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_ADD, m=m, m_dev=live, y=r)
    rows = max(1, m - 1)
    assert torch.equal(r[:rows], base[:rows] + y[:rows]) and torch.equal(r[rows:], base[rows:])
    if n > 1:
        even = n // 2 * 2
        g = ctx.matmul_fused(w, even, k, x, aotx_b200.EPILOGUE_SWIGLU)
        gate, up = y[:m, 0:even:2].double(), y[:m, 1:even:2].double()
        unit = gate / (1.0 + torch.exp(-gate)) * up
        # the sums may be cut at other places over `even` rows: both within the bound of exact ones;
        # silu has a slope of at most 1.1, and four float roundings follow
        slack = 2.2 * (bound[:, 0:even:2] * up.abs() + bound[:, 1:even:2] * (gate.abs() + 1.0)) + 2.0 ** -21 * unit.abs() + 1e-12
        assert bool(((g.double() - unit).abs() <= slack).all())
