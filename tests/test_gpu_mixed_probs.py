"""Outcome probabilities of mixed-precision states: the float rounding of the
Gammas does not show in p_0 + p_1, reads and records agree, and an outcome whose
probability is exactly 0 is never drawn.

Tolerances: p_0 + p_1 is divided out, so it is 1 to float64's rounding; read and
record sum the same double-float terms in two orders (2^-46 each, below 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NONE = np.zeros(0)
LAST = np.nextafter(1.0, 0.0)


def test_certain_outcomes(pkg):
    n, B = 8, 256
    b = pkg.Batch([n] * B, [pkg.Trunc.both(16, 1e-10)] * B, "mixed")
    ids = list(range(B))
    for t in range(3):
        b.step(ids, [pkg.gen_layer(5, i, t, n, 0.2) for i in ids])
    none = np.zeros((0, 4, 4))
    rng = np.random.default_rng(1)
    first, _ = b.step(ids, [(NONE, none, np.arange(n), rng.random(n)) for _ in ids])
    for u in (0.0, LAST):  # measured again: certain, whatever the uniform is
        again, ents = b.step(ids, [(NONE, none, np.arange(n), np.full(n, u)) for _ in ids])
        assert [[r[1] for r in x] for x in again] == [[r[1] for r in x] for x in first]
        assert all(r[2] == 1.0 for x in again for r in x)
        assert np.all(np.abs(ents) < 1e-6)
    assert b.device_status() == 0


@pytest.mark.parametrize("n,chi", [(6, 8), (12, 40)])
def test_reads_and_records_agree(pkg, n, chi):
    m = pkg.MPS.new_qubits(n, pkg.Trunc.both(chi, 1e-10), "mixed")
    for t in range(8):
        m.apply_bilayer(*pkg.gen_layer(7, 1, t, n, 0.1))
    for k in range(n):
        p = m.probs(k)
        assert abs(p.sum() - 1.0) < 1e-15
        c = m.clone()
        o, pr = c.measure_prob(k, 0.5)
        assert abs(pr - p[o]) < 1e-12
    assert m.device_status() == 0


def test_sum_far_from_one_is_reported_as_it_is(pkg):
    """An imported state that is not normalised: its own values, and the status bit."""
    g = [np.zeros((1, 2, 1), complex) for _ in range(3)]
    for x in g:
        x[0, 0, 0], x[0, 1, 0] = 0.6, 0.9
    m = pkg.MPS.from_parts(g, [np.ones(1)] * 2, None, "mixed")
    np.testing.assert_allclose(m.probs(1), [0.36, 0.81], atol=1e-7)
    m.measure_prob(1, 0.1)
    assert m.device_status() != 0


@pytest.mark.parametrize("prec,tol", [("f64", 1e-13), ("df", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("dims", [(1, 1), (1, 2), (2, 3), (3, 1), (5, 17), (33, 16), (31, 32), (16, 33), (70, 65),
                                  (128, 200), (300, 1)])
def test_sums_over_every_shape_of_a_site(pkg, prec, dims, tol):
    """Rows of 1 to 200 entries on groups of 1 to 32 lanes, in the read and in the
    measurement, against numpy; the tolerance is the mode's rounding of a sum of
    squares."""
    cl, cr = dims
    rng = np.random.default_rng(cl * 1000 + cr)
    g = [rng.standard_normal((a, 2, b)) + 1j * rng.standard_normal((a, 2, b)) for a, b in ((1, cl), (cl, cr), (cr, 1))]
    lam = [rng.random(cl) + 0.1, rng.random(cr) + 0.1]
    w = np.abs(g[1]) ** 2 * (lam[0] ** 2)[:, None, None] * (lam[1] ** 2)[None, None, :]
    g[1] /= np.sqrt(w.sum())
    p = w.sum((0, 2)) / w.sum()
    g += [np.eye(1, 2).reshape(1, 2, 1).astype(complex)] * 15  # (a chain long enough for such bonds)
    lam += [np.ones(1)] * 15
    m = pkg.MPS.from_parts(g, lam, None, prec, chi_cap=max(dims))
    np.testing.assert_allclose(m.probs(1), p, atol=tol)
    o, pr = m.clone().measure_prob(1, 0.3)
    assert o == (0 if 0.3 < p[0] else 1) and abs(pr - p[o]) < tol
