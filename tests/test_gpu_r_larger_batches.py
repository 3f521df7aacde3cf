"""Products of 17 rows and more at the sizes where the kernels that serve them can go wrong: the edges of
the regimes (17, 128, 129 rows) and of the token tiles (256), row tiles that are not full, one segment of
depth and many, clusters that share a tile (few rows of w), whole tiles in turns, tiles cut into units
(among more than two blocks too), each store.

The bounds: products of two binary16 values are exact in float and k float additions in any order are off
by at most k * 2^-23 times the sum of the magnitudes (2^-23: an addition may truncate).  bfloat16 x above
128 rows: the weights are rounded to bfloat16 as well, 2^-8 of a weight at most."""
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


def sums(ctx, w, n, k, x, extra=0.0):
    """The exact products in float64 and the bound of their float sums."""
    wd = ctx.dequant(w, k, 0, n).double()
    xd = x.double()
    return xd @ wd.T, (k * 2.0 ** -23 + extra) * (xd.abs() @ wd.abs().T) + 1e-30


# rows of w: a partial tile; one tile; a cluster of four's, of two's; two turns; cut into units; and deep
# enough that one tile has several holders
SHAPES = [(1, 256, 17), (130, 1024, 33), (1023, 2048, 128), (9990, 512, 40), (20004, 768, 64), (60001, 256, 100),
          (77, 1536, 129), (300, 5120, 257), (2049, 1024, 300), (19456, 512, 512), (40962, 256, 700)]


@pytest.mark.parametrize("n,k,m", SHAPES)
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
        assert torch.equal(z[:m], y[:m].to(kind))
        assert bool((z[m] == torch.tensor(GUARD, dtype=kind)).all())
    # bfloat16 activations
    xb = x.bfloat16()
    want_b, bound_b = sums(ctx, w, n, k, xb, extra=2.0 ** -8 if m > 128 else 2.0 ** -11)
    assert bool(((ctx.matmul(w, n, k, xb).double() - want_b).abs() <= bound_b).all())
    # residual add, and only the live rows
    for rows in sorted({0, m // 2, m - 1}):
        live = torch.tensor([rows], dtype=torch.int32, device="cuda")
        base = torch.randn(m, n, device="cuda", generator=gen)
        r = base.clone()
        ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_ADD, m=m, m_dev=live, y=r)
        # (other live tiles: the sums may be cut at other places)
        assert bool(((r[:rows] - base[:rows]).double() - want[:rows]).abs().le(bound[:rows] + 2.0 ** -22 * (base[:rows].abs() + want[:rows].abs())).all())
        assert torch.equal(r[rows:], base[rows:])
    if n > 1:
        even = n // 2 * 2
        for kind, eps in ((torch.float32, 2.0 ** -21), (torch.float16, 2.0 ** -10)):
            g = torch.full((m + 1, even // 2), GUARD, device="cuda", dtype=kind)
            ctx.matmul_fused(w, even, k, x, aotx_b200.EPILOGUE_SWIGLU, m=m, y=g[:m])
            gate, up = y[:m, 0:even:2].double(), y[:m, 1:even:2].double()
            unit = gate / (1.0 + torch.exp(-gate)) * up
            # silu has a slope of at most 1.1; four float roundings, and the one to binary16 (or to its
            # smallest step, 2^-24)
            slack = 2.2 * (bound[:, 0:even:2] * up.abs() + bound[:, 1:even:2] * (gate.abs() + 1.0)) + eps * unit.abs() + 2.0 ** -24
            assert bool(((g[:m].double() - unit).abs() <= slack).all())
            assert bool((g[m] == torch.tensor(GUARD, dtype=kind)).all())
