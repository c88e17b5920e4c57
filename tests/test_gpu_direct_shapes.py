"""The direct sum's launch shapes: target counts and source counts on both
sides of the lines at which a tile of targets takes one to eight blocks of one
to eight parts, against plain torch float64 at a sample of the targets.

Tolerance: as tests/test_gpu_direct_edges.py derives it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nt", [3, 20000, 151553, 303105, 606209, 700001, 2424900])
@pytest.mark.parametrize("ns", [1, 32, 33, 129, 257, 1025, 4097])
def test_direct_sum_shapes(sb, nt, ns):
    gen = torch.Generator("cuda").manual_seed(nt + ns)
    p = torch.randn(3, nt + ns, dtype=torch.float64, device="cuda", generator=gen)
    p /= p.norm(dim=0)
    t, s = [[a.contiguous() for a in c] for c in (p[:, :nt], p[:, nt:])]
    w = torch.randn(ns, dtype=torch.float64, device="cuda", generator=gen)
    at = torch.unique(torch.cat([torch.randint(nt, (150,), device="cuda", generator=gen),
                                 torch.tensor([0, nt - 1], device="cuda")]))
    x, y = torch.stack(t, 1)[at], torch.stack(s, 1)
    d = y[None] - x[:, None]
    r2 = (d * d).sum(-1)
    g = w / (0.5 * r2 + 1e-4)
    want = -torch.linalg.cross(x, (g[..., None] * d).sum(1)) / (4 * np.pi)
    got = torch.stack(sb.direct_sum_bve(*t, *s, w, 1e-4), 1)[at]
    scale = max(float(want.abs().max()), 1e-3 * float(g.abs().max()))
    assert float((got - want).abs().max()) <= 1e-12 * scale
    got = torch.stack(sb.direct_sum_bve(*t, *s, w, 1e-4, sb.MIXED), 1)[at]
    u = 2.0 ** -24
    bound = (18 * u * g.abs().sum(1) + 136 * u * (g.abs() * r2.sqrt()).sum(1)) / (4 * np.pi)
    assert bool(((got - want).norm(dim=1) <= bound).all())
