"""The Poisson list kernel at the edges of its shapes (every points-per-panel
class, trees on both sides of the warps-per-panel rule) against the same sums
in plain torch float64, target accumulated into.

Tolerance: 1e-12 of the largest value, the repository's float64 bound."""
import numpy as np
import pytest

from test_gpu_list64 import points

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("levels,degree,theta", [(1, 0, 0.7), (2, 1, 0.7), (4, 2, 0.6), (6, 2, 0.9), (5, 3, 0.7),
                                                 (6, 3, 0.9), (3, 4, 0.7), (3, 5, 0.8), (2, 6, 0.7), (3, 7, 0.9),
                                                 (2, 8, 0.7), (2, 9, 0.7), (2, 10, 0.7)])
def test_poisson_interactions(sb, levels, degree, theta):
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, fmm_theta=theta, exact_cc=1))
    if degree:
        x = points(sb, levels, degree)
    else:
        x = torch.from_numpy(np.concatenate([np.stack(sb.cube_sphere_spec_points(
            k, 0, sb.cubed_sphere_panels_init(k), sb.interp_init(0, True))[:3], -1) for k in range(1, levels + 1)])).cuda()
    g = torch.Generator("cuda").manual_seed(levels * 10 + degree)
    w = torch.randn(x.shape[:2], dtype=torch.float64, device="cuda", generator=g)
    t0 = torch.randn(x.shape[:2], dtype=torch.float64, device="cuda", generator=g)
    want, got = t0.clone(), t0.clone()
    lst = torch.from_numpy(ctx.interactions()).long().cuda()
    for k in range(0, len(lst), 1 << 13):
        t, s = lst[k:k + (1 << 13), 0], lst[k:k + (1 << 13), 1]
        dp = torch.einsum("eic,ejc->eij", x[t], x[s])
        v = torch.where(dp < 1 - 1e-15, torch.log(1 - dp), torch.zeros_like(dp)) * w[s][:, None]
        want.index_add_(0, t, -v.sum(2) / (4 * np.pi))
    ctx.poisson_fmm_interactions(w, got)
    assert float((got - want).abs().max() / want.abs().max()) <= 1e-12
