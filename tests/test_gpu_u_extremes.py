"""What becomes of values at the ends of the number range: gates far below and above zero, infinities."""
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


def same_kind(got, want):
    """Finite, infinite of the same sign, or not a number, in the same places."""
    torch = torch_mod()
    return bool((torch.isnan(got) == torch.isnan(want)).all()) and torch.equal(got.isinf(), want.isinf()) \
        and torch.equal(got[got.isinf()], want[want.isinf()])


GATES = [0.0, 1.0, -1.0, 20.0, -50.0, -87.0, -88.0, -88.5, -89.0, -90.0, -100.0, -110.0, -200.0, -1000.0, -60000.0, 60000.0, 100.0,
         float("inf"), float("-inf"), float("nan"), -1e10, 1e10, -1e30, 1e30]


# the general path; up to 16 rows; clusters, units and turns of the kernel for 17 to 128 rows, a width that is no
# multiple of four; pairs of SMs
@pytest.mark.parametrize("n,m,path", [(256, 24, 1), (5000, 8, 1), (256, 8, 0), (40000, 16, 0), (256, 24, 0), (9000, 100, 0),
                                      (12006, 32, 0), (40000, 64, 0), (60002, 100, 0), (512, 200, 0), (20002, 300, 0)])
@pytest.mark.parametrize("kind", ["float16", "bfloat16"])
def test_gates_at_the_limits(ctx, n, m, path, kind):
    """Rows of weights that are 1 in the first place: gate and up are the x in that place.  The unit is the float
    expression g / (1 + exp(-g)) * g within four roundings; what lies below the smallest normal float may be zero."""
    import aotx_b200
    torch = torch_mod()
    kind = getattr(torch, kind)
    k = 256
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
