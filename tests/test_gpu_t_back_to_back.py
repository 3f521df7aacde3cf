"""Launches right behind launches: blocks of a launch without work of their own, whose places the next launch
takes at once.  Every result is the one that the same calls give one at a time."""
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


def in_turn_and_alone(ctx, calls, repeats=20):
    """Every call gives a tensor.  The calls behind one another without a wait, against each by itself."""
    torch = torch_mod()
    alone = []
    for call in calls:
        alone.append(call().clone())
        torch.cuda.synchronize()
    for _ in range(repeats):
        together = [call() for call in calls]
        torch.cuda.synchronize()
        for got, want in zip(together, alone):
            assert torch.equal(got, want)


# more places than pieces: one row tile, a few of them, few segments; and a live batch that leaves tiles empty
@pytest.mark.parametrize("n,k,m,live", [(100, 512, 200, 200), (700, 256, 300, 300), (256, 1024, 2048, 3), (40, 256, 64, 64),
                                        (1000, 1024, 128, 128)])
def test_products_with_blocks_that_have_no_work(ctx, n, k, m, live):
    import aotx_b200
    torch = torch_mod()
    ws = [aotx_b200.synth_q8_0_device(n, k, seed) for seed in range(4)]
    x = torch.randn(m, k, device="cuda").half()
    few = torch.tensor([live], dtype=torch.int32, device="cuda")
    ys = [torch.zeros(m, n, device="cuda") for _ in ws]
    in_turn_and_alone(ctx, [lambda w=w, y=y: ctx.matmul(w, n, k, x, m_dev=few, y=y) for w, y in zip(ws, ys)])


def test_routed_steps_with_fewer_tiles_than_blocks(ctx):
    import aotx_b200
    torch = torch_mod()
    experts, used, hidden, ffn, tokens = 64, 2, 512, 256, 40
    gen = torch.Generator(device="cuda").manual_seed(1)
    wg, wu = (aotx_b200.synth_q8_0_device(experts * ffn, hidden, s) for s in (1, 2))
    wd = aotx_b200.synth_q8_0_device(experts * hidden, ffn, 3)
    x = torch.randn(tokens, hidden, device="cuda", generator=gen).half()
    prob = torch.rand(tokens, experts, device="cuda", generator=gen)
    calls = []
    # every token on the same two experts; on none that exists; on any
    for ids in (torch.tensor([[3, 9]] * tokens), torch.full((tokens, used), experts + 1),
                torch.randint(0, experts, (tokens, used), generator=torch.Generator().manual_seed(2))):
        ids = ids.int().cuda()
        out = torch.zeros(tokens, hidden, device="cuda")
        work = ctx.moe_workspace(tokens, used, hidden, ffn)
        calls.append(lambda ids=ids, out=out, work=work: ctx.moe_ffn(wg, wu, wd, experts, hidden, ffn, x, prob, ids, out=out,
                                                                     workspace=work))
    in_turn_and_alone(ctx, calls)


def test_results_that_the_next_launch_reads(ctx):
    """Launches start before the one before them has ended and read its results: y of one product is x of the next, two
    buffers in turn, through the kernels of every regime and of the other block types, the conversion of bfloat16 x,
    the router and the routed step.  The same as with every launch by itself."""
    import aotx_b200
    import numpy as np
    import _blocks
    from _util import dev
    torch = torch_mod()
    k = 1024
    gen = torch.Generator(device="cuda").manual_seed(7)
    q8 = [aotx_b200.synth_q8_0_device(k, k, s) for s in range(3)]
    other = {t: dev(_blocks.random_rows(t, k, k, np.random.Generator(np.random.PCG64(t))).reshape(-1)) for t in (2, 12, 14)}
    experts, used, ffn = 16, 2, 256
    wg, wu = (aotx_b200.synth_q8_0_device(experts * ffn, k, s) for s in (4, 5))
    wd = aotx_b200.synth_q8_0_device(experts * k, ffn, 6)
    router = torch.randn(experts, k, device="cuda", generator=gen) / k ** 0.5
    results = []
    for m in (3, 12, 40, 200):
        for kind in (torch.float16, torch.bfloat16):
            start = torch.randn(m, k, device="cuda", generator=gen).to(kind)
            a, b = torch.empty_like(start), torch.empty_like(start)
            out = torch.empty(m, k, device="cuda")
            work = ctx.moe_workspace(m, used, k, ffn)

            def chain():
                a.copy_(start)
                ctx.matmul(q8[0], k, k, a, y=b)
                ctx.matmul(other[2], k, k, b, y=a, type=2)
                ctx.matmul(other[12], k, k, a, y=b, type=12)
                ctx.matmul(q8[1], k, k, b, y=a)
                ctx.set_path(1)
                ctx.matmul(q8[2], k, k, a, y=b)
                ctx.set_path(0)
                ctx.matmul(other[14], k, k, b, y=a, type=14)
                if kind == torch.float16:
                    prob, ids = ctx.moe_route(a, router, used)
                    ctx.moe_ffn(wg, wu, wd, experts, k, ffn, a, prob, ids, out=out, workspace=work)
                    return a.clone(), out.clone()
                return (a.clone(),)

            ctx.set_overlap(False)
            alone = chain()
            torch.cuda.synchronize()
            ctx.set_overlap(True)
            for _ in range(10):
                for got, want in zip(chain(), alone):
                    assert torch.equal(got, want)
            results.append(alone[0].float().abs().max().item())
    assert all(0.0 < r < 60000.0 for r in results)      # nothing died away or left the range of binary16


# whole rows of w per block, both its depths; bfloat16 x that becomes binary16 in the kernel, in clusters and whole tiles;
# the pairs' cut tiles of many holders and of few
@pytest.mark.parametrize("n,k,m", [(3072, 3072, 1), (4096, 2048, 4), (4700, 9216, 3), (1024, 1024, 24), (28672, 1024, 24),
                                   (28672, 1024, 60), (1000, 2048, 200), (2560, 2560, 300)])
@pytest.mark.parametrize("kind", ["float16", "bfloat16"])
def test_results_that_the_same_kernel_reads(ctx, n, k, m, kind):
    """Back and forth between two buffers, k to n and n to k: each product reads what the launch before it wrote."""
    import aotx_b200
    torch = torch_mod()
    kind = getattr(torch, kind)
    n = n // 256 * 256
    there, back = aotx_b200.synth_q8_0_device(n, k, 1), aotx_b200.synth_q8_0_device(k, n, 2)
    start = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)).to(kind)
    a, b = torch.empty_like(start), torch.empty(m, n, device="cuda", dtype=kind)

    def chain():
        a.copy_(start)
        for _ in range(3):
            ctx.matmul(there, n, k, a, y=b)
            ctx.matmul(back, k, n, b, y=a)
        return a.clone(), b.clone()

    ctx.set_overlap(False)
    alone = chain()
    torch.cuda.synchronize()
    ctx.set_overlap(True)
    for _ in range(10):
        for got, want in zip(chain(), alone):
            assert torch.equal(got, want)
    assert all(0.0 < t.float().abs().max().item() < 60000.0 for t in alone)
