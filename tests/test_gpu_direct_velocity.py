"""The direct velocity of a grid (velocity=direct) on both sides of its dispatch
(sums over points in float64 and for panels of at most nine points, by panels in
source groups above), for trees whose leaves fill the groups unevenly, against
plain torch float64; and its shallow-water form.

Tolerance: 1e-12 of the largest value where the pairs are float64 (the
repository's float64 bound), 1e-6 where they are float32 (its mixed bound)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

K4 = 1 / (4 * np.pi)


def grid(sb, levels, degree):
    x, y, z, a = sb.cube_sphere_spec_points(levels, degree, sb.cubed_sphere_panels_init(levels),
                                            sb.interp_init(degree, True))
    return [torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (x, y, z, a)]


def sums(x, w, eps):
    """sum_j w_j (x_j - x_i) / (|x_j - x_i|^2 / 2 + eps), coincident pairs left out."""
    out = torch.empty_like(x)
    for k in range(0, len(x), 512):
        d = x[None] - x[k:k + 512, None]
        r2 = (d * d).sum(-1)
        g = torch.where(r2 > 0, w / (0.5 * r2 + eps), torch.zeros_like(r2))
        out[k:k + 512] = (g[..., None] * d).sum(1)
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("levels,degree", [(1, 0), (4, 0), (1, 1), (5, 1), (3, 2), (4, 2), (1, 3), (2, 3), (4, 3), (2, 4),
                                           (3, 4), (2, 5), (3, 6), (1, 10)])
def test_direct_velocity(sb, levels, degree, precision):
    f = grid(sb, levels, degree)
    vors = torch.sin(3 * f[0] + 0.2) * f[1] + f[2]
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, kernel_eps=1e-3, exact_cc=1, velocity=sb.VEL_DIRECT,
                                       precision=precision))
    vel = [torch.empty_like(vors) for _ in range(3)]
    ctx.bve_velocity(*f, vors, *vel)
    x = torch.stack([t.flatten() for t in f[:3]], 1)
    want = -K4 * torch.linalg.cross(x, sums(x, (f[3] * vors).flatten(), 1e-3))
    got = torch.stack([t.flatten() for t in vel], 1)
    tol = 1e-6 if precision and degree > 2 else 1e-12
    assert float((got - want).abs().max()) <= tol * float(want.abs().max())


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("levels,degree", [(1, 2), (4, 2), (3, 3), (4, 3), (2, 4), (3, 4), (2, 5)])
def test_direct_shallow_water_velocity(sb, levels, degree, precision):
    f = grid(sb, levels, degree)
    vors, divs = torch.sin(3 * f[0] + 0.2) * f[1] + f[2], torch.cos(2 * f[2]) * f[0]
    h = 2.9 + 0.1 * f[1]
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, kernel_eps=1e-3, exact_cc=1, velocity=sb.VEL_DIRECT,
                                       precision=precision, g_over_a=1.0))
    vel, base = ([torch.zeros_like(vors) for _ in range(3)] for _ in range(2))
    ctx.swe_init(*f, vors, divs, h, *vel, *base)
    x = torch.stack([t.flatten() for t in f[:3]], 1)
    b = sums(x, (f[3] * divs).flatten(), 1e-3)
    want = -K4 * torch.linalg.cross(x, sums(x, (f[3] * vors).flatten(), 1e-3)) + K4 * (b - x * (x * b).sum(1, keepdim=True))
    key = torch.round(x * 1e9).long()  # points that share a position take their mean
    where = torch.unique(key, dim=0, return_inverse=True)[1]
    total = torch.zeros((int(where.max()) + 1, 3), dtype=torch.float64, device="cuda").index_add_(0, where, want)
    count = torch.zeros(len(total), dtype=torch.float64, device="cuda").index_add_(0, where, torch.ones_like(want[:, 0]))
    want = (total / count[:, None])[where]
    got = torch.stack([t.flatten() for t in vel], 1)
    assert float((got - want).abs().max()) <= (1e-6 if precision else 1e-12) * float(want.abs().max())
