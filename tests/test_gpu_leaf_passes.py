"""The treecode's leaf passes (particles -> proxies, proxies -> particles) at
the edges of their tiles: proxy degrees 1..4 run without the degree as a
constant, 1..10 take register tiles of 1 x 1 to 4 x 4 moments, leaves of one
grid panel and of 4 to 484 particles leave the warps' rounds of 24 particles
unfilled, and even and odd grid degrees make leaf grids of 2 to 22 columns.

Float64 steps and two-field velocities against the oracle's treecode of the
same proxies and lists, whose operations differ only in their order: a sum of
at most 512 products per moment, two contractions per pass and up to five
levels leave below 1e-13 of the largest velocity; the bound is the 1e-12 of
the other treecode tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DT, OMEGA, EPS, TOL = 0.005, 2 * np.pi, 1e-4, 1e-12

# (levels, grid degree, leaf size, proxy degree)
CASES = [(3, 3, 64, 1), (3, 3, 16, 2), (3, 2, 36, 3), (3, 4, 100, 4), (4, 1, 64, 4), (4, 1, 4, 5), (3, 5, 144, 6),
         (3, 2, 9, 7), (3, 6, 196, 8), (4, 2, 144, 9), (3, 10, 484, 10)]


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def rel(a, b):
    a = torch.stack(a).cpu().numpy().reshape(3, -1) if isinstance(a, list) else a.cpu().numpy().ravel()
    b = np.asarray(b).reshape(a.shape)
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.fixture(params=CASES, ids=lambda c: "L%d-d%d-leaf%d-n%d" % c)
def case(request, sb, port):
    levels, deg, leaf, n = request.param
    cfg = sb.config_default(levels=levels, interp_degree=deg, kernel_eps=EPS, omega=OMEGA, dt=DT, fmm_theta=0.7,
                            proxy_degree=n, leaf_size=leaf, precision=sb.FP64, g_over_a=1.0)
    return request.param, cfg, sb.build_grid(levels, deg, exact_cc=True)


def test_step(sb, port, case):
    (levels, deg, leaf, n), cfg, g = case
    og = port.build(levels, deg, None, exact_cc=True)
    vor = np.sin(3 * g.x) * g.y + g.z
    want, wvel, _ = port.bve_step(og, vor, None, dt=DT, omega=OMEGA, eps=EPS, mode=2, tree=(n, leaf, 0.7, 0))
    v = cuda(vor)
    vel = [torch.zeros_like(v) for _ in range(3)]
    sb.Context(cfg).bve_back_rk4_step(cuda(g.x), cuda(g.y), cuda(g.z), cuda(g.area), v, *vel)
    assert rel(vel, np.stack(wvel)) <= TOL
    assert rel(v, want) <= TOL


def test_two_field_velocity(sb, port, case):
    (levels, deg, leaf, n), cfg, g = case
    if deg < 2 or leaf > 256:
        pytest.skip("the two-field treecode takes grid degrees from 2 and leaves of at most 256 particles")
    d = [2e-3 * np.random.default_rng(7).standard_normal(g.x.shape) for _ in range(3)]
    wv, wd = g.area * (g.z + np.cos(3 * g.x)), g.area * 0.3 * np.cos(2 * g.x - g.z)
    s = np.stack([g.x + d[0], g.y + d[1], g.z + d[2]])
    s /= np.linalg.norm(s, axis=0)
    p = (g.x, g.y, g.z)
    want = port.bltc_velocity_swe(levels, deg, leaf, n, 0.7, EPS, 0, p, (s[0], s[1], s[2]), wv, p, wd)
    u = [torch.zeros(g.x.shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    sb.Context(cfg).swe_tree_velocity(*[cuda(a) for a in d], cuda(wv), cuda(wd), *u)
    assert rel(u, want) <= TOL
