"""A trajectory that has become NaN (a post-selected outcome of probability 0, a
gate beyond float32's range in the float modes) spoils itself alone: the
launch ends, its neighbours' results keep their bits, and the library goes on.
At bonds of the shared-memory path, of the block Jacobi and of the cluster."""
import numpy as np
import pytest

from test_gpu_small_bonds import _random

pytestmark = pytest.mark.gpu
NONE = np.zeros(0)


def _state(pkg, ref, n, chi, prec):
    m = ref.from_vector(_random(np.random.default_rng(5), n), ref.Trunc.both(chi, 1e-10))
    return m.data, m.svals, pkg.Trunc.both(chi, 1e-10)


@pytest.mark.parametrize("prec", ["f64", "df", "mixed"])
@pytest.mark.parametrize("n,chi", [(2, 2), (7, 8), (10, 32), (13, 40), (14, 100)])
def test_impossible_outcome_spoils_one_trajectory(pkg, ref, prec, n, chi):
    parts = _state(pkg, ref, n, chi, prec)
    layer = pkg.gen_layer(3, 0, 0, n, 0.3)

    def run(bad):
        b = pkg.Batch([n] * 3, [parts[2]] * 3, prec)
        for i in (0, 2):
            b.import_state(i, *parts)
        # trajectory 1 is |0...0>: outcome 1 has probability 0
        b.step([1], [(NONE, np.zeros((0, 4, 4)), [n // 2], [0.5])], posts=[[1 if bad else 0]])
        out = []
        for _ in range(2):
            recs, ents = b.step([0, 1, 2], [layer] * 3)
            out += [recs[0], recs[2], ents[0], ents[2]]
        out += [b.svals(i, k).tolist() for i in (0, 2) for k in range(n - 1)]
        mid = b.svals(1, n // 2 - 1)
        b.close()
        return out, mid

    good, s = run(False)
    assert np.all(np.isfinite(s))
    spoilt, _ = run(True)
    assert spoilt == good


@pytest.mark.parametrize("prec", ["f64", "df", "mixed"])
@pytest.mark.parametrize("n,chi", [(7, 8), (10, 32), (13, 40), (14, 100)])
def test_single_state_that_is_not_a_number(pkg, ref, prec, n, chi):
    data, svals, tr = _state(pkg, ref, n, chi, prec)
    data = [d.copy() for d in data]
    data[n // 2][:, 1, :] = 0.0  # outcome 1 of that site is impossible
    g = pkg.MPS.from_parts(data, svals, tr, prec)
    g.measure_postsel_prob(n // 2, 1)
    assert not np.all(np.isfinite(g.probs(n // 2)))
    g.apply_unitary2(n // 2 - 1, np.eye(4))
    if prec != "f64":  # finite in float64, not in float32
        h = pkg.MPS.from_parts(*_state(pkg, ref, n, chi, prec), prec)
        h.apply_unitary2(n // 2 - 1, 1e39 * np.eye(4))
        h.entropy_vn(n // 2 - 1)
    ok = pkg.MPS.new_qubits(6, None, prec)
    ok.apply_unitary2(2, np.eye(4))
    assert abs(ok.entropy_vn(2)) < 1e-6 and ok.device_status() == 0
