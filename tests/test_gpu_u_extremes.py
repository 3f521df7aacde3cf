"""What becomes of values at the ends of the number range: gates far below and above zero, infinities, sums that
are finite though the sums of their whole-number form are not."""
import numpy as np
import pytest

import _blocks
from _util import dev, torch_mod

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import aotx_b200
    c = aotx_b200.Q8Context(0)
    yield c
    assert c.device_status() == 0
    c.close()


def same_kind(got, want):
    """Finite, infinite of the same sign, or not a number, in the same places."""
    torch = torch_mod()
    return bool((torch.isnan(got) == torch.isnan(want)).all()) and torch.equal(got.isinf(), want.isinf()) \
        and torch.equal(got[got.isinf()], want[want.isinf()])


GATES = [0.0, 1.0, -1.0, 20.0, -50.0, -87.0, -88.0, -88.5, -89.0, -90.0, -100.0, -110.0, -200.0, -1000.0, -60000.0, 60000.0, 100.0,
         float("inf"), float("-inf"), float("nan"), -1e10, 1e10, -1e30, 1e30]


# the general path; up to 16 rows; whole rows of w per block; clusters, units and turns of the kernel for 17 to 128 rows, a
# width that is no multiple of four; pairs of SMs: cut tiles of few holders and of many
@pytest.mark.parametrize("n,m,path,k", [(256, 24, 1, 256), (5000, 8, 1, 256), (256, 8, 0, 256), (40000, 16, 0, 256), (4000, 4, 0, 2048),
                                        (4600, 3, 0, 5120), (256, 24, 0, 256), (9000, 100, 0, 256), (12006, 32, 0, 256),
                                        (40000, 64, 0, 256), (60002, 100, 0, 256), (512, 200, 0, 256), (20002, 300, 0, 256),
                                        (512, 200, 0, 4096)])
@pytest.mark.parametrize("kind", ["float16", "bfloat16"])
def test_gates_at_the_limits(ctx, n, m, path, k, kind):
    """Rows of weights that are 1 in the first place: gate and up are the x in that place.  The unit is the float
    expression g / (1 + exp(-g)) * g within four roundings; what lies below the smallest normal float may be zero."""
    import aotx_b200
    torch = torch_mod()
    kind = getattr(torch, kind)
    raw = torch.zeros(n, k // 32, 34, dtype=torch.uint8, device="cuda")
    raw[:, :, :2] = torch.tensor([1.0], dtype=torch.float16).view(torch.uint8).cuda()
    raw[:, 0, 2] = 1
    gates = torch.tensor(GATES)
    if kind == torch.float16 or (path == 0 and m <= 128):
        gates = gates[gates.isnan() | gates.isinf() | (gates.abs() <= 65504.0)]      # x is binary16 there
    if kind == torch.bfloat16 and path == 0 and m <= 128:
        gates = gates[gates.isfinite()]                                               # and saturates
    for at in range(0, len(gates), m):
        some = gates[at:at + m].to(kind)
        x = torch.zeros(m, k, device="cuda", dtype=kind)
        x[:len(some), 0] = some.cuda()
        ctx.set_path(path)
        got = ctx.matmul_fused(raw.view(-1), n, k, x, aotx_b200.EPILOGUE_SWIGLU)[:len(some)]
        ctx.set_path(0)
        g = some.float().cuda()
        want = (g / (1.0 + torch.exp(-g)) * g)[:, None].expand_as(got)
        assert same_kind(got, want)
        fine = want.isfinite()
        assert bool(((got - want).abs() <= 2.0 ** -20 * want.abs() + 2.0 ** -120)[fine].all())


@pytest.fixture(scope="module")
def decoder(tmp_path_factory):
    return _blocks.HostDecoder(tmp_path_factory.mktemp("decoder"))


@pytest.mark.parametrize("type", [8, 2, 3, 6, 7, 12, 13, 14])
@pytest.mark.parametrize("m", [4, 20])
@pytest.mark.parametrize("kind", ["float16", "bfloat16"])
def test_infinities_and_large_x(ctx, decoder, type, m, kind):
    """A finite weight times an infinite x is infinite with the sign of the product (or, for a weight of zero, not a
    number), and a sum that fits a float is finite, whatever the scales and offsets of the format."""
    torch = torch_mod()
    kind = getattr(torch, kind)
    n, k = 70, 1024
    w = _blocks.random_rows(type, n, k, np.random.Generator(np.random.PCG64(type)))
    weights = torch.from_numpy(decoder.rows(type, w, n, k)).double().cuda()
    x = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)).to(kind)
    x[0, 5], x[1, 40], x[2, 300] = float("inf"), float("-inf"), float("nan")
    if kind == torch.bfloat16:
        x[3] = 0.0
        x[3, 64:128] = 3e36       # whole numbers times it leave the float range
    want = x.double() @ weights.T
    ctx.set_path(1 if type == 8 else 0)
    got = ctx.matmul(dev(w), n, k, x, type=type)
    ctx.set_path(0)
    assert same_kind(got, want.float())
    fine = want.isfinite()
    bound = (k + 8) * 2.0 ** -23 * 4.0 * (x.double().abs() @ weights.abs().amax(dim=1, keepdim=True).expand(n, k).T)
    assert bool(((got.double() - want).abs() <= bound)[fine].all())
