"""How exact the float sums of a product are, against float64.

A tensor-core MMA adds sixteen products to a running sum and truncates the result: half a unit in the last
place of the sum, towards zero, each time.  So what the error of a product grows with is the number of MMAs
that go one after the other into one accumulator.  Over a chain of L of them the running sum of random
products has 2/3 of its final size on average, a float is 0.72 of the next power of two, and the losses
towards zero add up: at most 0.4 * L * 2^-24 of the result in the 2-norm, and the ordinary roundings beside
them, 1.5 * 2^-24.

`chain` is the longest chain the kernels may use at that shape: the depth of a block's run where the
(row tile, segment) units of the tensor are dealt evenly to all places for a block, over two blocks per SM
and four accumulators in turn (up to 16 rows), two (up to 32), one block per SM and one accumulator above."""
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


@pytest.mark.parametrize("n,k,m,chain", [(4096, 4096, 1, 8), (3072, 4096, 4, 8), (4600, 14336, 1, 28),
                                         (4736, 16384, 4, 32), (5000, 1024, 8, 4), (2048, 14336, 16, 28), (28672, 4096, 8, 40),
                                         # accumulators in turn: in clusters of four with one slab and with two, of two,
                                         # whole tiles in turns; runs, of one segment and of several
                                         (4096, 4096, 24, 16), (6144, 4096, 32, 32), (14336, 4096, 20, 44), (28672, 4096, 32, 77),
                                         (4096, 4096, 48, 55), (512, 16384, 64, 28), (300, 4096, 128, 16), (2048, 14336, 100, 94),
                                         # pairs of SMs: two accumulators; few tiles, whose units are dealt evenly
                                         (20000, 4096, 100, 188), (5000, 1024, 160, 18), (2560, 2560, 300, 45), (1000, 2048, 200, 16)])
def test_error_of_the_sums(ctx, n, k, m, chain):
    import aotx_b200
    torch = torch_mod()
    w = aotx_b200.synth_q8_0_device(n, k, n + m)
    x = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)).half()
    want = x.double() @ ctx.dequant(w, k, 0, n).double().T
    off = ((ctx.matmul(w, n, k, x).double() - want).norm() / want.norm()).item()
    assert off <= (1.5 + 0.4 * chain) * 2.0 ** -24
