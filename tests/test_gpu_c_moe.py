"""Routed experts on the device against the oracle (cases of tests/expert_test.cu)."""
import numpy as np
import pytest

from _util import GUARD, dev, dev_weights, torch_mod
from oracle.binding import SEED, row_bytes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import aotx_b200
    c = aotx_b200.Q8Context(0)
    yield c
    c.close()


def _route_fixture(tokens, experts, precision):
    """Router rows and inputs of tests/expert_test.cu:66-89."""
    hidden = 32
    router = np.zeros((experts, hidden), np.float32)
    for e in range(experts):
        pos = np.float32(e) / np.float32(max(experts - 1, 1))
        for d in range(hidden):
            router[e, d] = (np.float32(1.0002) if e == 2 else np.float32(1.0)) if precision \
                else np.float32((d % 5) - 2) * np.float32(0.0012345)
        if not precision:
            router[e, 0] = np.float32(3.0) * pos
            router[e, 1] = np.float32(-3.0) * pos * pos
    router[1] = router[0]
    x = np.zeros((tokens, hidden), np.float16)
    for t in range(tokens):
        for d in range(hidden):
            x[t, d] = 1.0 if precision else (((t * 7 + d * 3) % 13) - 6) / 16.0
        if not precision:
            x[t, 0] = np.float32(2.0) * np.float32(t) / np.float32(tokens) + np.float32(0.007)
            x[t, 1] = 1.0
    return router, x


@pytest.mark.parametrize("tokens", [1, 64])
@pytest.mark.parametrize("experts,used,precision", [(7, 1, 0), (7, 3, 0), (7, 7, 0), (64, 8, 0),
                                                    (256, 256, 0), (3, 1, 1)])
def test_route(ctx, oracle, tokens, experts, used, precision):
    torch = torch_mod()
    router, x = _route_fixture(tokens, experts, precision)
    cap = tokens + 2
    prob = torch.full((cap, experts), GUARD, dtype=torch.float32, device="cuda")
    ids = torch.full((cap, used), -1, dtype=torch.int32, device="cuda")
    xd = dev(np.concatenate([x, np.zeros((2, 32), np.float16)]))
    ctx.moe_route(xd, dev(router), used, tokens=tokens, prob=prob, ids=ids)
    torch.cuda.synchronize()
    got_p = prob.cpu().numpy()
    got_i = ids.cpu().numpy().view(np.uint32)
    want_p, want_i = oracle.route(x.view(np.uint16), router, used)
    assert np.isfinite(got_p[:tokens]).all()
    assert np.abs(got_p[:tokens] - want_p).max() < 2e-6
    assert np.array_equal(got_i[:tokens], want_i)
    assert np.array_equal(got_i[:tokens], oracle.rank(got_p[:tokens], used))
    assert (got_p[tokens:] == GUARD).all() and (got_i[tokens:] == 0xFFFFFFFF).all()
    mass = np.take_along_axis(got_p[:tokens], got_i[:tokens].astype(np.int64), 1).sum(1)
    if used == experts:
        assert np.abs(mass - 1.0).max() < 2e-5
    else:
        assert (mass < 0.999).all()


# (a live count on the device: the kernels with tiles take only what the host has counted)
@pytest.mark.parametrize("tokens,experts,used,hidden,live", [
    (149, 17, 3, 32, 149),        # rows of one step
    (153, 33, 4, 160, 150),       # eight tokens to a cluster of four blocks; a last group cut by the live count
    (300, 128, 8, 2048, 297),     # the same, full rounds of a row
    (593, 16, 2, 1120, 592),      # a block for all experts
    (601, 5, 5, 288, 1),          # the same, one live token
    (1203, 250, 9, 1056, 1203)])  # groups one behind the other
def test_route_of_many_tokens(ctx, oracle, tokens, experts, used, hidden, live):
    torch = torch_mod()
    rng = np.random.Generator(np.random.PCG64(tokens + experts))
    router = rng.standard_normal((experts, hidden)).astype(np.float32) / np.float32(np.sqrt(hidden))
    router[experts - 1] = router[0]           # the same sums: the lower index first
    x = rng.standard_normal((tokens, hidden)).astype(np.float16)
    prob = torch.full((tokens, experts), GUARD, dtype=torch.float32, device="cuda")
    ids = torch.full((tokens, used), -1, dtype=torch.int32, device="cuda")
    ctx.moe_route(dev(x), dev(router), used, tokens=tokens, tokens_dev=dev(np.array([live], np.int32)), prob=prob, ids=ids)
    torch.cuda.synchronize()
    got_p = prob.cpu().numpy()
    got_i = ids.cpu().numpy().view(np.uint32)
    want_p, want_i = oracle.route(x[:live].view(np.uint16), router, used)
    assert np.abs(got_p[:live] - want_p).max() < 2e-6
    assert np.array_equal(got_i[:live], oracle.rank(got_p[:live], used))
    assert np.array_equal(got_i[:live], want_i)
    assert np.array_equal(got_p[:live, experts - 1], got_p[:live, 0])
    assert (got_p[live:] == GUARD).all() and (got_i[live:] == 0xFFFFFFFF).all()
    assert ctx.device_status() == 0


def _off_boundary(t, values):
    """A copy that starts `values` elements after a 16-byte boundary, which the router's tiles do not take."""
    flat = torch_mod().empty(t.numel() + values, dtype=t.dtype, device="cuda")
    return flat[values:].view(t.shape).copy_(t)


# Every form of the tiles (tokens to a group, experts to a block, one block of an SM or two) and every size of cluster, with a
# last group and a last block that are not full, and the sizes next to a line; beside them the kernels that take rows off a
# boundary, for more than 148 tokens clusters of four blocks, and one block for all experts where rows are long or tokens
# many and experts at most 64.  (Which form it is follows from how many clusters run at the same time, here as on a B200 with 15
# clusters of seven.)
@pytest.mark.parametrize("tokens,experts,used,hidden", [
    (149, 17, 3, 32), (153, 33, 4, 160), (180, 72, 5, 4096),                           # groups of 4, clusters of 1, 2, 3
    (1000, 17, 2, 544), (592, 64, 6, 288), (300, 96, 8, 640), (257, 100, 8, 2048),     # groups of 8, clusters of 1, 2, 3, 4
    (200, 136, 8, 512), (161, 192, 7, 1056),                                           # clusters of 5, 6
    (593, 64, 6, 288), (361, 96, 8, 640), (297, 128, 8, 2048), (220, 136, 8, 512),     # groups of 16, clusters of 2, 3, 4, 5
    (200, 192, 7, 1056), (149, 200, 8, 1024), (150, 256, 3, 992),          # clusters of 6, 7, 8
    (256, 224, 8, 4096), (256, 256, 8, 2048),                                          # two blocks to an SM, groups of 8
    (1203, 250, 9, 1056), (1185, 48, 4, 256),                                          # groups of 16
    (150, 48, 3, 4128), (1201, 20, 4, 96),                                             # beside one block for all experts
    (593, 16, 2, 1120), (1300, 14, 2, 288)])                                           # a block for all of few experts, 8 and 16 tokens
def test_router_tiles_give_the_floats_of_the_other_kernels(ctx, tokens, experts, used, hidden):
    torch = torch_mod()
    gen = torch.Generator(device="cuda").manual_seed(tokens * 7 + experts)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).half()
    router = torch.randn(experts, hidden, device="cuda", generator=gen) / hidden ** 0.5
    router[experts - 1] = router[0]
    prob = torch.full((tokens + 1, experts), GUARD, dtype=torch.float32, device="cuda")
    ids = torch.full((tokens + 1, used), -1, dtype=torch.int32, device="cuda")
    ctx.moe_route(x, router, used, tokens=tokens, prob=prob, ids=ids)
    for x_other, router_other in ((_off_boundary(x, 4), router), (x, _off_boundary(router, 1))):
        want_p, want_i = ctx.moe_route(x_other, router_other, used)
        assert torch.equal(prob[:tokens].view(torch.int32), want_p.view(torch.int32))
        assert torch.equal(ids[:tokens], want_i)
    assert bool((prob[tokens:] == GUARD).all()) and bool((ids[tokens:] == -1).all())
    assert ctx.device_status() == 0


# more than 148 tokens, rows of no multiple of 32 values: clusters of four, and one block for all experts
@pytest.mark.parametrize("tokens,experts,hidden", [(149, 33, 1000), (300, 128, 2040), (160, 20, 4100), (1100, 64, 500)])
def test_router_of_other_widths(ctx, oracle, tokens, experts, hidden):
    torch = torch_mod()
    rng = np.random.Generator(np.random.PCG64(tokens + hidden))
    router = rng.standard_normal((experts, hidden)).astype(np.float32) / np.float32(np.sqrt(hidden))
    x = rng.standard_normal((tokens, hidden)).astype(np.float16)
    prob, ids = ctx.moe_route(dev(x), dev(router), 4)
    torch.cuda.synchronize()
    want_p, want_i = oracle.route(x.view(np.uint16), router, 4)
    assert np.abs(prob.cpu().numpy() - want_p).max() < 2e-6
    assert np.array_equal(ids.cpu().numpy().view(np.uint32), want_i)


def _route_us(ctx, x, router, used, live):
    torch = torch_mod()
    tokens, experts = x.shape[0], router.shape[0]
    prob = torch.empty(tokens, experts, device="cuda")
    ids = torch.empty(tokens, used, dtype=torch.int32, device="cuda")
    count = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    ctx.moe_route(x, router, used, tokens_dev=count, prob=prob, ids=ids)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(10):
            ctx.moe_route(x, router, used, tokens_dev=count, prob=prob, ids=ids)
    graph.replay()
    times = []
    for _ in range(7):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        for _ in range(4):
            graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(begin.elapsed_time(end) * 1000.0 / 40.0)
    return min(times)


# The rule between the router's kernels: rows on a boundary may take another kernel than rows off it, not a slower one.  A
# fifth is more than two runs of one kernel differ by.
@pytest.mark.parametrize("tokens,experts,hidden,live", [
    (2048, 8, 2048, 64), (2048, 32, 2048, 8),      # few of the most are live: 2.0 and 1.5 of the others' time on tiles
    (256, 224, 4096, None),                        # 16 clusters, of which 15 run at the same time alone on their SMs: 1.6
    (1024, 8, 4096, None), (593, 2, 6144, None), (200, 17, 8192, None), (592, 24, 5120, None)])   # one block for all experts: 1.3 to 2.2
def test_router_on_a_boundary_is_not_slower(ctx, tokens, experts, hidden, live):
    torch = torch_mod()
    gen = torch.Generator(device="cuda").manual_seed(tokens + experts)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).half()
    router = torch.randn(experts, hidden, device="cuda", generator=gen) / hidden ** 0.5
    on = _route_us(ctx, x, router, min(8, experts), live)
    off = _route_us(ctx, _off_boundary(x, 4), router, min(8, experts), live)
    assert on <= 1.2 * off, (on, off)


def _moe_case(oracle, tokens, experts, used, hidden, ffn, seed):
    import aotx_b200
    wg = aotx_b200.synth_q8_0(experts * ffn, hidden, seed)
    wu = aotx_b200.synth_q8_0(experts * ffn, hidden, seed + 1)
    wd = aotx_b200.synth_q8_0(experts * hidden, ffn, seed + 2)
    rng = np.random.Generator(np.random.PCG64(seed + 3))
    # scales of the benchmark's distribution give outputs near 1e-4; a unit-size input keeps
    # every intermediate inside the half range
    x = rng.standard_normal((tokens, hidden)).astype(np.float16)
    router = rng.standard_normal((experts, hidden)).astype(np.float32) / np.float32(np.sqrt(hidden))
    return wg, wu, wd, x, router


@pytest.mark.parametrize("tokens,experts,used,hidden,ffn", [(1, 5, 3, 512, 64), (64, 5, 3, 512, 96),
                                                            (33, 16, 4, 256, 256), (200, 7, 2, 512, 256),
                                                            (64, 128, 8, 2048, 768)])
def test_moe_ffn_matches_oracle(ctx, oracle, tokens, experts, used, hidden, ffn):
    torch = torch_mod()
    wg, wu, wd, x, router = _moe_case(oracle, tokens, experts, used, hidden, ffn, 40 + tokens)
    xd = dev(x)
    prob, ids = ctx.moe_route(xd, dev(router), used)
    out = torch.full((tokens + 2, hidden), GUARD, dtype=torch.float32, device="cuda")
    ctx.moe_ffn(dev_weights(wg), dev_weights(wu), dev_weights(wd), experts, hidden, ffn, xd, prob,
                ids, tokens=tokens, out=out[:tokens])
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    p = prob.cpu().numpy()
    i = ids.cpu().numpy().view(np.uint32)
    want = oracle.moe_ffn(wg, wu, wd, experts, hidden, ffn, x.view(np.uint16), p, i)
    ok, err, bound = oracle.within_bound(got[:tokens], want.astype(np.float64))
    assert ok, (err, bound)
    assert oracle.diff(got[:tokens], want.astype(np.float64))[0] == 0
    assert (got[tokens:] == GUARD).all()


def test_selection_outside_the_expert_table_adds_nothing(ctx, oracle):
    """The selections come from the caller: one that names no expert is left out of the products
    (no kernel indexes a tensor with it) and adds nothing to its token's sum, on the grouped
    tensor-core path and on the per-pair path.  The reference has no such case: its selections
    come from its own router (cuda/model/experts.cu:10-75)."""
    import aotx_b200
    torch = torch_mod()
    tokens, experts, used, hidden, ffn = 24, 6, 2, 256, 256
    wg, wu, wd, x, router = _moe_case(oracle, tokens, experts, used, hidden, ffn, 77)
    xd = dev(x)
    prob, ids = ctx.moe_route(xd, dev(router), used)
    p = prob.cpu().numpy()
    i = ids.cpu().numpy().view(np.uint32)
    want = oracle.moe_ffn(wg, wu, wd, experts, hidden, ffn, x.view(np.uint16), p, i)
    first = oracle.moe_ffn(wg, wu, wd, experts, hidden, ffn, x.view(np.uint16), p, np.ascontiguousarray(i[:, :1]))
    want[3] = first[3]
    bad = i.copy()
    bad[3, 1] = 0xFFFFFFFF
    bad_dev = dev(bad.view(np.int32))
    dwg, dwu, dwd = dev_weights(wg), dev_weights(wu), dev_weights(wd)
    for path in (0, aotx_b200.PATH_GENERAL):
        ctx.set_path(path)
        try:
            out = ctx.moe_ffn(dwg, dwu, dwd, experts, hidden, ffn, xd, prob, bad_dev)
        finally:
            ctx.set_path(0)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        ok, err, bound = oracle.within_bound(got, want.astype(np.float64))
        assert ok, (path, err, bound)
    assert ctx.device_status() == 0


def test_ordered_sum_bit_exact(ctx, oracle):
    """The rank-ordered weighted sum equals the oracle bit for bit, rows past the batch stay
    untouched (tests/expert_test.cu:164-195)."""
    torch = torch_mod()
    rng = np.random.Generator(np.random.PCG64(3))
    for tokens, hidden, experts, used in ((1, 32, 7, 1), (9, 96, 11, 5), (64, 32, 7, 7)):
        proj = rng.standard_normal((tokens, used, hidden)).astype(np.float32)
        prob = rng.random((tokens, experts)).astype(np.float32)
        ids = np.stack([rng.permutation(experts)[:used] for _ in range(tokens)]).astype(np.uint32)
        want = oracle.ordered_sum(np.ascontiguousarray(proj.transpose(1, 0, 2)), prob, ids)
        out = torch.full((tokens + 2, hidden), GUARD, dtype=torch.float32, device="cuda")
        ctx.moe_combine(dev(proj), dev(prob), dev(ids.view(np.int32)), out=out[:tokens])
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[:tokens].view(np.uint32), want.view(np.uint32))
        assert (got[tokens:] == GUARD).all()


def test_grouped_path_equals_per_pair_path_at_full_size(ctx, oracle):
    """The benchmark's routed-expert shape (512 tokens, 128 experts, top 8, 2048 -> 768 -> 2048):
    the grouped tensor-core path and the per-pair path give the same result within the product
    bound, and the same selections feed both."""
    import aotx_b200
    torch = torch_mod()
    tokens, experts, used, hidden, ffn = 512, 128, 8, 2048, 768
    wg, wu, wd, x, router = _moe_case(oracle, tokens, experts, used, hidden, ffn, 900)
    xd = dev(x)
    prob, ids = ctx.moe_route(xd, dev(router), used)
    dwg, dwu, dwd = dev_weights(wg), dev_weights(wu), dev_weights(wd)
    outs = []
    for path in (aotx_b200.PATH_TENSOR, aotx_b200.PATH_GENERAL):
        ctx.set_path(path)
        try:
            outs.append(ctx.moe_ffn(dwg, dwu, dwd, experts, hidden, ffn, xd, prob, ids).cpu().numpy())
        finally:
            ctx.set_path(0)
    torch.cuda.synchronize()
    a, b = outs
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= 1e-2 * np.abs(b).max() + 1e-3
    counts = np.bincount(ids.cpu().numpy().reshape(-1), minlength=experts)
    assert counts.sum() == tokens * used and counts.max() > 32
    assert ctx.device_status() == 0


# A block for all experts of four tokens: few experts (149, 301, 2500 tokens), long rows of up to 47 (150); clusters that share
# them (148); tiles (1024, 1025).
@pytest.mark.parametrize("tokens,experts,hidden", [(149, 8, 512), (148, 8, 512), (301, 16, 2048), (150, 33, 4128), (1025, 64, 512),
                                                   (1024, 64, 512), (2500, 3, 96)])
def test_router_on_both_sides_of_the_line(tokens, experts, hidden):
    import aotx_b200
    torch = torch_mod()
    ctx = aotx_b200.Q8Context(0)
    used = min(experts, 3)
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).half()
    router = torch.randn(experts, hidden, device="cuda", generator=gen) / hidden ** 0.5
    prob, ids = ctx.moe_route(x, router, used)
    want = torch.softmax(x.double() @ router.double().T, dim=1)
    # the logits' float sums, and a softmax of at most `experts` terms
    slack = hidden * 2.0 ** -23 * (x.double().abs() @ router.double().abs().T).amax(dim=1, keepdim=True) * 2.0 + experts * 2.0 ** -23
    assert bool(((prob.double() - want).abs() <= slack * want + 1e-30).all())
    order = torch.sort(prob, dim=1, descending=True, stable=True)[1][:, :used]
    assert torch.equal(ids.long(), order)
    ctx.close()
