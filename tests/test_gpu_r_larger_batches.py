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
SHAPES = [(20004, 512, 113), (1, 256, 17), (130, 1024, 33), (1023, 2048, 128), (9990, 512, 40), (20004, 768, 64), (60001, 256, 100),
          (77, 1536, 129), (300, 5120, 257), (2049, 1024, 300), (19456, 512, 512), (40962, 256, 700),
          (20004, 512, 192), (20004, 512, 325), (1500, 2048, 370), (2049, 1024, 576)]


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


# pairs: fewer than blocks; one step of a warp and one more; more than a warp keeps in registers (4096)
@pytest.mark.parametrize("tokens,experts,used,hidden,ffn", [(1, 16, 2, 256, 256), (33, 8, 4, 512, 256),
                                                            (700, 16, 6, 1024, 512), (1100, 128, 4, 256, 256)])
def test_routed_experts_sorted_by_many_blocks(ctx, tokens, experts, used, hidden, ffn):
    """The sort and gather over many blocks and the product of gate and up in one launch, with a live batch,
    selections outside the table and an expert that most tokens choose."""
    import aotx_b200
    torch = torch_mod()
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    wg = aotx_b200.synth_q8_0_device(experts * ffn, hidden, 1)
    wu = aotx_b200.synth_q8_0_device(experts * ffn, hidden, 2)
    wd = aotx_b200.synth_q8_0_device(experts * hidden, ffn, 3)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).half()
    ids = torch.stack([torch.randperm(experts, device="cuda", generator=gen)[:used] for _ in range(tokens)]).int()
    ids[: tokens * 3 // 4, 0] = 0                 # (a pair twice is a pair like any other)
    ids[tokens // 2, used - 1] = experts + 5      # outside the table: adds nothing
    prob = torch.rand(tokens, experts, device="cuda", generator=gen)
    live = tokens - tokens // 3
    out = torch.full((tokens, hidden), GUARD, device="cuda")
    ctx.moe_ffn(wg, wu, wd, experts, hidden, ffn, x, prob, ids, tokens_dev=torch.tensor([live], dtype=torch.int32, device="cuda"),
                out=out)
    gate_w, up_w = (ctx.dequant(w, hidden, 0, experts * ffn).double().view(experts, ffn, hidden) for w in (wg, wu))
    down_w = ctx.dequant(wd, ffn, 0, experts * hidden).double().view(experts, hidden, ffn)
    want = torch.zeros(tokens, hidden, device="cuda", dtype=torch.float64)
    bound = torch.zeros_like(want)
    for e in range(experts):
        for t, r in (ids[:live] == e).nonzero().tolist():
            xd = x[t].double()
            gate, up = gate_w[e] @ xd, up_w[e] @ xd
            unit = gate / (1.0 + torch.exp(-gate)) * up
            # act: the float sums' errors through the unit (slope at most 1.1), and one rounding to binary16
            eg, eu = (hidden * 2.0 ** -23 * (w[e].abs() @ xd.abs()) for w in (gate_w, up_w))
            err = 2.2 * (eg * up.abs() + eu * (gate.abs() + 1.0)) + 2.0 ** -10 * unit.abs() + 2.0 ** -24
            p = prob[t, e].double()
            want[t] += p * (down_w[e] @ unit)
            bound[t] += p * (down_w[e].abs() @ (err + (ffn + used + 2) * 2.0 ** -23 * unit.abs()))
    assert bool(((out[:live].double() - want[:live]).abs() <= bound[:live] * 1.001 + 1e-30).all())
    assert bool((out[live:] == GUARD).all())
