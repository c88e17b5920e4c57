"""The float64 treecode adjoint's kernels at the edges of their shapes: tree
leaves of 9 to 400 particles, every proxy degree, trees of one to three levels
(clusters of eight blocks per leaf down to one).

The reverse step is linear in its cotangent, and on a mixed-precision context
of the same tree it runs the separate float32 pair kernels: the two agree to
float32 rounding (1e-6 of the largest value, the repository's mixed bound)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("levels,degree,proxy,leaf", [(2, 3, 5, 16), (3, 2, 6, 9), (3, 2, 7, 40), (4, 2, 9, 150),
                                                      (3, 3, 8, 64), (4, 3, 10, 256), (4, 4, 6, 512), (5, 3, 8, 256),
                                                      (5, 2, 4, 144), (3, 3, 2, 64), (3, 3, 1, 16)])
def test_adjoint_against_mixed_kernels(sb, levels, degree, proxy, leaf):
    g = sb.build_grid(levels, degree, exact_cc=True)
    f = [torch.from_numpy(a).cuda() for a in (g.x, g.y, g.z, g.area)]
    v = torch.from_numpy(np.exp(-((g.x - 0.8) ** 2 + g.y ** 2 + (g.z - 0.6) ** 2) / 0.1)).cuda()
    bar = torch.from_numpy(g.area * (g.x * g.y + g.z + 0.3 * g.y * g.z)).cuda()
    out = []
    for precision in (sb.FP64, sb.MIXED):
        ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, kernel_eps=1e-3, omega=1.0, dt=0.01,
                                           exact_cc=1, fmm_theta=0.7, proxy_degree=proxy, leaf_size=leaf,
                                           precision=precision))
        a, b = torch.empty_like(v), torch.empty_like(v)
        ctx.bve_adjoint_step(*f, v, bar, a)
        ctx.bve_adjoint_step(*f, v, -2.0 * bar, b)
        assert float((b + 2.0 * a).abs().max()) <= 1e-12 * float(a.abs().max())
        out.append(a)
    assert float((out[0] - out[1]).abs().max()) <= 1e-6 * float(out[0].abs().max())
