"""A non-finite point is reported by every kind of call (eager steps, replayed
graphs, host arrays, batches), by that call alone, and the context goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def config(sb, **kw):
    return sb.config_default(**{**dict(levels=3, interp_degree=3, kernel_eps=1e-4, omega=2 * np.pi, dt=0.005, exact_cc=1,
                                       fmm_theta=0.7), **kw})


def fields(sb):
    g = sb.build_grid(3, 3, exact_cc=True)
    return g, [torch.from_numpy(np.ascontiguousarray(a)) for a in (g.x, g.y, g.z, g.area, np.sin(2 * g.x) + g.z)]


@pytest.mark.parametrize("method", ["spectral", "tree", "direct"])
@pytest.mark.parametrize("call", ["step", "run", "host", "pinned"])
def test_reported_once_and_cleared(sb, method, call):
    more = dict(spectral={}, tree=dict(proxy_degree=6, leaf_size=64), direct=dict(velocity=sb.VEL_DIRECT))[method]
    ctx = sb.Context(config(sb, **more))
    _, f = fields(sb)
    put = {"host": lambda t: t.clone(), "pinned": lambda t: t.clone().pin_memory()}.get(call, lambda t: t.cuda())
    f = [put(t) for t in f]
    vel = [put(torch.zeros_like(f[0])) for _ in range(3)]
    good = f[4].clone()
    go = {"step": ctx.bve_back_rk4_step, "run": lambda *a: ctx.bve_run(*a, nsteps=2)}.get(call, ctx.bve_back_rk4_step_host)
    results = []
    for attempt in range(3):  # the first captures or times, the second replays
        f[4].copy_(good)
        go(*f, *vel)
        results.append(f[4].clone())
        f[4].copy_(good)
        f[4][2, 3] = float("nan")
        with pytest.raises(sb.SbslpmError) as e:
            go(*f, *vel)
        assert "non-finite" in str(e.value)
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])


@pytest.mark.parametrize("precision", [0, 1])
def test_batch(sb, precision):
    batch = sb.Batch(config(sb, precision=precision, leaf_size=64, proxy_degree=6), [0.6, 0.7, 0.8], [6, 8, 6])
    _, f = fields(sb)
    f = [t.cuda() for t in f]
    v0 = torch.stack([f[4], 0.5 * f[4], f[4] ** 2])
    vel = torch.zeros((3, 3) + tuple(f[4].shape), dtype=torch.float64, device="cuda")
    v = v0.clone()
    for go in (batch.step, lambda *a: batch.run(*a, nsteps=2), lambda *a: batch.run(*a, nsteps=2)):
        v.copy_(v0)
        go(*f[:4], v, vel)
        assert torch.isfinite(v).all()
        v.copy_(v0)
        v[1, 4, 5] = float("nan")
        with pytest.raises(sb.SbslpmError) as e:
            go(*f[:4], v, vel)
        assert "non-finite" in str(e.value)
        assert torch.isfinite(v[0]).all() and torch.isfinite(v[2]).all()  # the other members' own
