"""Products above 128 rows whose tiles are cut between pairs of SMs, where the way a cut tile is finished changes: few
holders (the one that began it), many (all of them, each a run of its rows of x), more than a warp has lanes, rows of x
that are no multiple of a run, tiles that are not full, and a live batch with fewer tiles than the whole one.

The bound: k additions in any order are off by at most k * 2^-23 times the sum of the magnitudes."""
import pytest

from _util import torch_mod

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import aotx_b200
    c = aotx_b200.Q8Context(0)
    yield c
    assert c.device_status() == 0
    c.close()


@pytest.mark.parametrize("n,k,m", [(1000, 2048, 200), (256, 16384, 150), (130, 16384, 257), (2560, 2560, 300), (1024, 4096, 301),
                                   (5000, 1024, 161), (19456, 2560, 300), (2048, 9728, 133), (300, 256, 700)])
@pytest.mark.parametrize("epilogue", ["store", "add", "gated"])
def test_cut_tiles(ctx, n, k, m, epilogue):
    import aotx_b200
    torch = torch_mod()
    gen = torch.Generator(device="cuda").manual_seed(n + m)
    w = aotx_b200.synth_q8_0_device(n, k, n + m)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    wd, xd = ctx.dequant(w, k, 0, n).double(), x.double()
    want, bound = xd @ wd.T, k * 2.0 ** -23 * (xd.abs() @ wd.abs().T) + 1e-30
    for live in sorted({m, m - 1, 129, 128, 1, 0}):
        word = torch.tensor([live], dtype=torch.int32, device="cuda")
        if epilogue == "gated":
            first = None
            for _ in range(2):
                y = torch.full((m, n // 2), 3.0, device="cuda")
                ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_SWIGLU, m=m, m_dev=word, y=y)
                assert first is None or torch.equal(first, y)
                first = y
            gate, up = want[:live, 0::2], want[:live, 1::2]
            silu = gate / (1 + torch.exp(-gate))
            # |silu'| is at most 1.1, and |silu| at most the gate's magnitude; both factors' errors, and roundings
            off = 1.1 * bound[:live, 0::2] * (up.abs() + bound[:live, 1::2]) + gate.abs() * bound[:live, 1::2] + 2.0 ** -20 * (silu * up).abs()
            assert bool(((y[:live].double() - silu * up).abs() <= off + 1e-30).all())
            assert bool((y[live:] == 3.0).all())
            continue
        y = torch.full((m, n), 3.0, device="cuda")
        if epilogue == "add":
            ctx.matmul_fused(w, n, k, x, aotx_b200.EPILOGUE_ADD, m=m, m_dev=word, y=y)
            got, slack = y.double() - 3.0, 2.0 ** -23 * (want.abs() + 3.0)
        else:
            ctx.matmul(w, n, k, x, m=m, m_dev=word, y=y)
            got, slack = y.double(), 0.0
        assert bool(((got - want).abs() <= bound + slack)[:live].all())
        assert bool((y[live:] == 3.0).all())
