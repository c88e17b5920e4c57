"""A context's first Poisson calls find its tables complete: fresh contexts,
on the default stream, a side stream and the context's own, give the same bits
on the first call as on the second."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("stream", ["default", "side", "own"])
@pytest.mark.parametrize("levels,degree", [(2, 2), (4, 3), (3, 5)])
def test_first_solve_equals_second(sb, levels, degree, stream):
    g = sb.build_grid(levels, degree, exact_cc=True)
    area, f = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.area, g.x * g.y + g.z))
    side = torch.cuda.Stream()
    cfg = sb.config_default(levels=levels, interp_degree=degree, fmm_theta=0.7, exact_cc=1)
    for _ in range(3):
        first, second = torch.zeros_like(f), torch.zeros_like(f)
        torch.cuda.synchronize()
        with torch.cuda.stream(side if stream == "side" else torch.cuda.current_stream()):
            if stream == "own":  # a context of the C interface that was given no stream
                h = sb._VP()
                assert sb.lib().sbslpm_create(sb.ctypes.byref(cfg), sb.ctypes.byref(h)) == 0
                for out in (first, second):
                    assert sb.lib().sbslpm_poisson_fmm(h, area.data_ptr(), f.data_ptr(), out.data_ptr()) == 0
                sb.lib().sbslpm_destroy(h)
            else:
                ctx = sb.Context(cfg)
                ctx.poisson_fmm(area, f, first)
                ctx.poisson_fmm(area, f, second)
        torch.cuda.synchronize()
        assert float(second.abs().max()) > 0
        assert torch.equal(first, second)
