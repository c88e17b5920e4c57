"""The float64 treecode adjoint at the edges of its kernels' shapes (leaves of 9
to 400 particles, proxy degrees 2 to 10, trees of one to three levels) against
differences of the float64 forward step, <bar, J d> = <adjoint, d>.

Tolerance: the four-point difference's truncation is of order h^4 = 1e-16 of
the step's fifth derivative, its rounding of order 2^-53 / h = 1e-12, both
relative to |bar| |d| / sqrt(n), the size of such a product; 1e-8 of that size
leaves four orders for their factors and is a sixth of float32's rounding.
Proxy degree 1 on one-panel leaves is not among the cases: its velocity jumps by
some 1e-2 across panel edges, and a particle whose departure point crosses an
edge between the two sides makes the step itself discontinuous there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

H = 1e-4


@pytest.mark.parametrize("levels,degree,proxy,leaf", [(2, 3, 5, 16), (3, 2, 6, 9), (3, 2, 7, 40), (4, 2, 9, 150),
                                                      (3, 3, 8, 64), (4, 3, 10, 256), (4, 4, 6, 512), (5, 3, 8, 256),
                                                      (5, 2, 4, 144), (3, 3, 2, 64)])
def test_adjoint_against_differences(sb, levels, degree, proxy, leaf):
    g = sb.build_grid(levels, degree, exact_cc=True)
    f = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.x, g.y, g.z, g.area)]
    rng = np.random.default_rng(levels * 100 + degree * 10 + proxy)
    rnd = lambda: torch.from_numpy(rng.standard_normal(g.x.shape)).cuda()  # noqa: E731
    v = torch.from_numpy(np.exp(-((g.x - 0.8) ** 2 + (g.y - 0.1) ** 2 + (g.z - 0.6) ** 2) / 0.1) + 0.3 * g.x * g.y).cuda()
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, kernel_eps=1e-3, omega=1.0, dt=0.01,
                                       exact_cc=1, fmm_theta=0.7, proxy_degree=proxy, leaf_size=leaf))

    def step(w):
        w = w.clone()
        ctx.bve_back_rk4_step(*f, w, *[torch.empty_like(w) for _ in range(3)])
        return w

    for _ in range(2):
        bar, d = rnd(), rnd()
        adjoint = torch.empty_like(v)
        ctx.bve_adjoint_step(*f, v, bar, adjoint)
        first = ((step(v + H * d) - step(v - H * d)) * bar).sum()
        second = ((step(v + 2 * H * d) - step(v - 2 * H * d)) * bar).sum()
        fd = float(8 * first - second) / (12 * H)
        size = float(bar.norm() * d.norm()) / v.numel() ** 0.5
        assert abs(fd - float((adjoint * d).sum())) <= 1e-8 * size
