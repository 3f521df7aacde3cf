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
