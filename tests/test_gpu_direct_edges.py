"""The stand-alone direct sum at the edges of its tiles: single points, counts
around 32, 64, 128 and the source shares, coincident points, a coincidence with
eps = 0, against plain torch float64.

Tolerance: float64 1e-12 of the largest value (the repository's float64
bound).  Mixed precision, per target, the rounding of its float32 arithmetic:
offsets below 2 in magnitude, three roundings each (delta = 6 * 2^-24), move a
pair's g d by at most 3 g delta; its strength, reciprocal and products add
8 * 2^-24 relative, its running sum over a tile 128 * 2^-24."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("eps", [1e-4, 0.0])
@pytest.mark.parametrize("nt,ns", [(1, 1), (31, 33), (64, 2047), (65, 2049), (127, 1024), (129, 1025), (700, 24577),
                                   (5001, 130)])
def test_direct_sum(sb, nt, ns, eps):
    rng = np.random.default_rng(nt * 7 + ns)
    p = rng.standard_normal((nt + ns, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    t, s = (torch.from_numpy(a).cuda() for a in (p[:nt], p[nt:]))
    s[0] = t[-1]  # the same bits: adds nothing
    w = torch.from_numpy(rng.standard_normal(ns)).cuda()
    d = s[None] - t[:, None]
    r2 = (d * d).sum(-1)
    g = torch.where(r2 > 0, w / (0.5 * r2 + eps), torch.zeros_like(r2))
    want = -torch.linalg.cross(t, (g[..., None] * d).sum(1)) / (4 * np.pi)
    points = [[a[:, c].contiguous() for c in range(3)] for a in (t, s)]
    got = torch.stack(sb.direct_sum_bve(*points[0], *points[1], w, eps), 1)
    scale = max(float(want.abs().max()), 1e-3 * float(g.abs().max()))  # one pair's |g d| at the least
    assert float((got - want).abs().max()) <= 1e-12 * scale
    if eps > 0:
        got = torch.stack(sb.direct_sum_bve(*points[0], *points[1], w, eps, sb.MIXED), 1)
        u = 2.0 ** -24
        bound = (18 * u * g.abs().sum(1) + 136 * u * (g.abs() * r2.sqrt()).sum(1)) / (4 * np.pi)
        assert bool(((got - want).norm(dim=1) <= bound).all())
