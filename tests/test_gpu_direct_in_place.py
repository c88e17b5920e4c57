"""Direct sums whose results overlay their inputs (positions, strengths, parts
of one buffer) give the bits of the same sum into arrays of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", ["direct_sum_bve", "direct_sum_bve_noalloc"])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 65, 5001, 40000])
def test_results_over_inputs(sb, name, precision, n):
    rng = np.random.default_rng(n)
    p = rng.standard_normal((3, n))
    p /= np.linalg.norm(p, axis=0)
    base = torch.from_numpy(np.concatenate([p, rng.standard_normal((1, n))])).cuda()
    f = getattr(sb, name)
    want = [a.clone() for a in f(*base[:3], *base[:3], base[3], 1e-4, precision)]

    def run(choose):
        b = torch.cat([base.flatten(), torch.zeros(3 * n, dtype=torch.float64, device="cuda")])
        rows = [b[k * n:(k + 1) * n] for k in range(7)]
        out = choose(b, rows)
        f(*rows[:3], *rows[:3], rows[3], 1e-4, precision, out)
        return out

    for choose in (lambda b, r: r[:3],  # over the positions
                   lambda b, r: (r[3], r[4], r[5]),  # over the strengths
                   lambda b, r: [b[k * n + n // 2:(k + 1) * n + n // 2] for k in (1, 2, 3)]):  # across two inputs
        assert all(torch.equal(a, w) for a, w in zip(run(choose), want))
    one = run(lambda b, r: (r[4], r[4], r[4]))[0]  # one array for all: the last component
    assert torch.equal(one, want[2])
