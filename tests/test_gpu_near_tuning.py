"""Every near-field launch shape that the first step's timing can choose can be
read back and set again: on trees of few leaves it tries more than four
source-list splits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def context(sb, levels, degree, leaf, precision):
    ctx = sb.Context(sb.config_default(levels=levels, interp_degree=degree, kernel_eps=1e-4, omega=2 * np.pi, dt=0.005,
                                       fmm_theta=0.7, exact_cc=1, proxy_degree=8, leaf_size=leaf, precision=precision))
    ctx.set_cc_tuning(0, 0)
    return ctx


def step(sb, ctx, levels, degree):
    g = sb.build_grid(levels, degree, exact_cc=True)
    f = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.x, g.y, g.z, g.area, np.sin(3 * g.x) + g.z)]
    vel = [torch.zeros_like(f[0]) for _ in range(3)]
    ctx.bve_back_rk4_step(*f, *vel)
    return torch.stack([f[4], *vel])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("levels,degree,leaf,leaves", [(3, 3, 256, 6), (4, 3, 256, 24), (5, 3, 256, 96),
                                                       (5, 2, 36, 384), (6, 3, 64, 1536)])
def test_shape_read_back_and_set_again(sb, levels, degree, leaf, leaves, precision):
    first = context(sb, levels, degree, leaf, precision)
    first.set_near_mutual(False)
    step(sb, first, levels, degree)  # times the shapes
    first.set_near_mutual(False)
    want = step(sb, first, levels, degree)
    again = context(sb, levels, degree, leaf, precision)
    again.set_near_tuning(*first.near_tuning()[:3])
    again.set_near_mutual(False)
    assert again.near_tuning()[:3] == first.near_tuning()[:3]
    assert torch.equal(step(sb, again, levels, degree), want)


@pytest.mark.parametrize("levels,leaves", [(4, 24), (5, 96), (6, 384), (7, 1536)])
def test_splits_up_to_the_largest_one_timed(sb, levels, leaves):
    """16 blocks per SM's worth of splits, between 4 and 16; one more is refused."""
    top = min(16, max(4, 148 * 16 // leaves))
    ctx = context(sb, levels, 3, 256, 0)
    want = None
    for splits in sorted({1, 4, top}):
        ctx.set_near_tuning(128, 2, splits)
        assert ctx.near_tuning()[2] == splits
        got = step(sb, ctx, levels, 3)
        want = got if want is None else want
        assert float((got - want).abs().max() / want.abs().max()) <= 1e-12
    with pytest.raises(sb.SbslpmError):
        ctx.set_near_tuning(128, 2, top + 1)
