"""Coincident pairs of the float64 direct sum add nothing, whatever eps and the
strengths are: eps negative, NaN, subnormal or so small that a coincident
pair's weight overflows; infinite and NaN strengths.  Against the documented
formula in torch float64, both entry points.

Tolerance, per target, from the roundings (u = 2^-53): a pair's denominator
|d|^2 + 2 eps moves by at most 4 u (|d|^2 + 2 |eps|), its reciprocal, strength
and products by 8 u relative, a running sum of n pairs by n u; twice that for
the two evaluations, and 2 for the three components."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def inputs(nt, ns, scale=1.0):
    rng = np.random.default_rng(nt + ns)
    p = rng.standard_normal((nt + ns, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    t, s = (torch.from_numpy(a).cuda() for a in (p[:nt], p[nt:]))
    return t, s, torch.from_numpy(scale * rng.standard_normal(ns)).cuda()


def call(sb, name, t, s, w, eps):
    col = [[a[:, c].contiguous() for c in range(3)] for a in (t, s)]
    return torch.stack(getattr(sb, name)(*col[0], *col[1], w, eps), 1)


def reference(t, s, w, eps):
    d = s[None] - t[:, None]
    r2 = (d * d).sum(-1)
    g = torch.where(r2 > 0, w / (0.5 * r2 + eps), torch.zeros_like(r2))
    want = -torch.linalg.cross(t, (g[..., None] * d).sum(1)) / (4 * np.pi)
    spread = (r2 + 2 * abs(eps)) / (r2 + 2 * eps).abs()
    size = torch.where(r2 > 0, g.abs() * r2.sqrt() * (4 * spread + 8 + len(w)), torch.zeros_like(r2))
    return want, 4 * 2.0 ** -53 / (4 * np.pi) * size.sum(1)


@pytest.mark.parametrize("name", ["direct_sum_bve", "direct_sum_bve_noalloc"])
@pytest.mark.parametrize("eps", [1e-101, 1e-306, 1e-310, 0.0, -1e-3, -0.3])
def test_any_eps(sb, name, eps):
    t, s, w = inputs(70, 300, 1e4)
    s[::7] = t[:43]
    want, bound = reference(t, s, w, eps)
    got = call(sb, name, t, s, w, eps)
    assert torch.isfinite(want).all() and torch.isfinite(got).all()
    assert bool(((got - want).norm(dim=1) <= bound).all())


@pytest.mark.parametrize("name", ["direct_sum_bve", "direct_sum_bve_noalloc"])
def test_nan_eps(sb, name):
    t, s, w = inputs(5, 40)
    assert torch.isnan(call(sb, name, t, s, w, float("nan"))).all()
    assert not call(sb, name, t, t[:1].expand(5, 3), w[:5], float("nan"))[0].any()  # its own point alone


@pytest.mark.parametrize("name", ["direct_sum_bve", "direct_sum_bve_noalloc"])
@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan"), 1e308])
@pytest.mark.parametrize("eps", [1e-4, 1e-30])
def test_any_strength(sb, name, bad, eps):
    t, s, w = inputs(66, 200)
    s[150] = t[65]
    rest = w.clone()
    rest[150] = 0
    w[150] = bad
    want, bound = reference(t, s, rest, eps)
    got = call(sb, name, t, s, w, eps)
    assert float((got[65] - want[65]).norm()) <= float(bound[65])
    if not np.isfinite(bad):
        assert not torch.isfinite(got[:65]).all(dim=1).any()
