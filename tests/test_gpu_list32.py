"""The mixed-precision list kernels (csrc/list32.cuh) at the edges of their
shapes: every particles-per-panel count they take, odd counts, trees on both
sides of the warps-per-panel rule, both source fields, against the same sums
in plain torch float64.

Tolerance, per target: the rounding of the kernels' float32 arithmetic.
Packed offsets lie below 2, three roundings each (delta = 6 * 2^-24) move a
pair's g d by at most 3 g delta; its strength, reciprocal and products add
8 * 2^-24 relative, its panel's running sum at most 13 additions and the sum
of the two halves another 2^-24 each."""
import numpy as np
import pytest

from test_gpu_list64 import points

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
U = 2.0 ** -24


def sums(lst, tgt, src, w, eps):
    """(sum g d, its rounding bound) over the interaction list: [panel][q][3], [panel][q]."""
    P, q = w.shape
    out = torch.zeros((P, q, 3), dtype=torch.float64, device="cuda")
    bound = torch.zeros((P, q), dtype=torch.float64, device="cuda")
    for k in range(0, len(lst), 1 << 14):
        t, s = lst[k:k + (1 << 14), 0], lst[k:k + (1 << 14), 1]
        d = src[s][:, None] - tgt[t][:, :, None]
        r2 = (d * d).sum(-1)
        g = w[s][:, None] / (0.5 * r2 + eps)
        out.index_add_(0, t, (g[..., None] * d).sum(2))
        bound.index_add_(0, t, (18 * U * g.abs() + 22 * U * g.abs() * r2.sqrt()).sum(2))
    return out, bound


@pytest.mark.parametrize("levels,degree,theta", [(1, 3, 0.7), (2, 0, 0.7), (3, 1, 0.7), (4, 2, 0.6), (5, 3, 0.8),
                                                 (6, 2, 0.8), (6, 3, 0.9), (3, 4, 0.7), (6, 4, 0.9), (3, 5, 0.7)])
def test_mixed_list_sums(sb, levels, degree, theta):
    eps = 1e-4
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, fmm_theta=theta, kernel_eps=eps,
                                       exact_cc=1, precision=sb.MIXED))
    x = points(sb, levels, degree)
    g = torch.Generator("cuda").manual_seed(levels * 10 + degree)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    shape = x.shape[:2]
    disp, w, w2 = 1e-3 * rnd(*x.shape), rnd(*shape), rnd(*shape)
    y = x + disp
    y = y / y.norm(dim=-1, keepdim=True)
    d = [disp[..., c].contiguous() for c in range(3)]
    lst = torch.from_numpy(ctx.interactions()).long().cuda()
    a, bound = sums(lst, x, y, w, eps)
    want = -torch.linalg.cross(x, a) / (4 * np.pi)
    got = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    ctx.bve_vel_interactions(*d, w, *got)
    assert bool(((torch.stack(got, -1) - want).norm(dim=-1) <= bound / (4 * np.pi)).all())
    if degree < 2:
        return
    b, more = sums(lst, x, x, w2, eps)
    want = want + (b - x * (x * b).sum(-1, keepdim=True)) / (4 * np.pi)
    got = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    ctx.swe_vel_interactions(*d, w, w2, *got)
    assert bool(((torch.stack(got, -1) - want).norm(dim=-1) <= (bound + more) / (4 * np.pi)).all())
