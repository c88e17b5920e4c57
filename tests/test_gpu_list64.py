"""The float64 list kernels (csrc/list64.cuh) at the edges of their shapes:
every particles-per-panel count they take, trees on both sides of the
warps-per-panel rule and both source fields, against the same sums in plain torch float64.

Tolerance: 1e-12 of the largest value, the repository's float64 parity bound
(the sums differ in the order of their additions only)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 1e-12


def pair_sums(ctx, tgt, src, w, eps):
    """sum_j w_j (y_j - x_i) / (|y_j - x_i|^2 / 2 + eps) over the interaction list, [panel][q][3]."""
    P, q = w.shape
    out = torch.zeros((P, q, 3), dtype=torch.float64, device="cuda")
    lst = torch.from_numpy(ctx.interactions()).long().cuda()
    for k in range(0, len(lst), 1 << 14):
        t, s = lst[k:k + (1 << 14), 0], lst[k:k + (1 << 14), 1]
        d = src[s][:, None] - tgt[t][:, :, None]
        r2 = (d * d).sum(-1)
        g = torch.where(r2 > 0, w[s][:, None] / (0.5 * r2 + eps), torch.zeros_like(r2))
        out.index_add_(0, t, (g[..., None] * d).sum(2))
    return out


def points(sb, levels, degree):
    interp, out = sb.interp_init(degree, True), []
    # the proxies of every tree level are the leaf points of that level's own grid
    for lev in range(1, levels + 1):
        x, y, z, _ = sb.cube_sphere_spec_points(lev, degree, sb.cubed_sphere_panels_init(lev), interp)
        out.append(np.stack([x, y, z], -1))
    return torch.from_numpy(np.concatenate(out)).cuda()


@pytest.mark.parametrize("levels,degree,theta,eps", [
    (1, 3, 0.7, 1e-4), (2, 0, 0.7, 1e-4), (3, 1, 0.7, 1e-4), (4, 2, 0.6, 1e-4), (5, 3, 0.8, 1e-4),
    (6, 2, 0.8, 1e-4), (6, 3, 0.9, 1e-6), (3, 4, 0.7, 1e-4), (6, 4, 0.9, 1e-4), (3, 5, 0.7, 1e-4)])
def test_list_sums(sb, levels, degree, theta, eps):
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, fmm_theta=theta, kernel_eps=eps,
                                       exact_cc=1))
    x = points(sb, levels, degree)
    g = torch.Generator("cuda").manual_seed(levels * 10 + degree)
    rnd = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    shape = x.shape[:2]
    disp, w, w2 = 1e-3 * rnd(*x.shape), rnd(*shape), rnd(*shape)
    y = x + disp
    y = y / y.norm(dim=-1, keepdim=True)
    d = [disp[..., c].contiguous() for c in range(3)]
    a = pair_sums(ctx, x, y, w, eps)
    want = -torch.linalg.cross(x, a) / (4 * np.pi)
    got = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    ctx.bve_vel_interactions(*d, w, *got)
    err = (torch.stack(got, -1) - want).abs().max() / want.abs().max()
    assert float(err) <= TOL, float(err)
    if degree < 2:
        return
    b = pair_sums(ctx, x, x, w2, eps)
    want = want + (b - x * (x * b).sum(-1, keepdim=True)) / (4 * np.pi)
    got = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    ctx.swe_vel_interactions(*d, w, w2, *got)
    err = (torch.stack(got, -1) - want).abs().max() / want.abs().max()
    assert float(err) <= TOL, float(err)
