"""The piecewise departure search and remap on arrays that are not on 16-byte
boundaries (one value per load) against the same calls on aligned ones (two
where the panel size is even).

Tolerance: an interpolated value is a sum of q <= 64 products of magnitude at
most max|field| times a basis whose absolute sum stays below 4 (Chebyshev
nodes, degree <= 7), in either form: 2 * 64 * 4 * 2^-53 of the largest field
value, below 6e-14; a departure point moves by at most dt * 1.5 times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def off(t):
    """The same values in memory that starts 8 bytes after a 16-byte boundary."""
    b = torch.empty(t.numel() + 2, dtype=t.dtype, device=t.device)
    k = 1 if b.data_ptr() % 16 == 0 else 2
    v = b[k:k + t.numel()].view(t.shape)
    assert v.data_ptr() % 16 == 8
    return v.copy_(t)


@pytest.mark.parametrize("levels,degree", [(3, 1), (4, 2), (4, 3), (3, 5), (2, 7)])
def test_unaligned_arrays(sb, levels, degree):
    g = sb.build_grid(levels, degree, exact_cc=True)
    rng = np.random.default_rng(degree)
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, omega=2 * np.pi, dt=0.01, exact_cc=1,
                                       tracer_count=1))
    x = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.x, g.y, g.z)]
    p = torch.stack(x)
    v = []
    for _ in range(4):  # tangential velocities below 1 in magnitude
        w = torch.from_numpy(rng.uniform(-0.5, 0.5, 3)).cuda().view(3, 1, 1).expand_as(p)
        v.append(torch.linalg.cross(w, p, dim=0).contiguous())
    vors = torch.from_numpy(np.sin(3 * g.x) * g.y + g.z).cuda()
    tracer = (vors ** 2).unsqueeze(-1).contiguous()

    def run(place):
        a, u = [place(t) for t in x], [place(t) for t in v]
        dep = [place(torch.zeros_like(x[0])) for _ in range(3)]
        ctx.bve_departure(*a, *u, 0.01, *dep)
        new, newt = place(torch.zeros_like(vors)), place(torch.zeros_like(tracer))
        ctx.bve_remap(a[2], *dep, place(vors), place(tracer), new, newt)
        return torch.stack(dep), new, newt

    (d0, n0, t0), (d1, n1, t1) = run(lambda t: t.clone()), run(off)
    tol = 2 * 64 * 4 * 2.0 ** -53
    assert float((d0 - d1).abs().max()) <= 0.01 * 1.5 * tol + 4 * 2.0 ** -53
    # the fields' slopes (below 10) carry the points' difference into the values
    slope = 10 * 3 * (0.01 * 1.5 * tol + 4 * 2.0 ** -53)
    assert float((n0 - n1).abs().max()) <= tol * float(vors.abs().max()) + slope + 4 * np.pi * slope
    assert float((t0 - t1).abs().max()) <= tol * float(tracer.abs().max()) + 2 * slope
