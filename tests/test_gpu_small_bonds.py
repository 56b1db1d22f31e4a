"""Bond operations held in shared memory (tn_local.cuh) at the edges of their
range: vector counts around the limits of the small path and of its SVD
scratch, odd and one-dimensional bonds, rank-deficient, graded and degenerate
spectra, refactors with and without the LQ reduction; and the observables that
run outside the executor.  Against the oracle on the same states.

Tolerances: a bond operation's backward error is a small multiple of
sqrt(c) eps (eps = 2^-53, 2^-47, 2^-24 for f64, df, mixed; c <= 70), i.e. below
1e-14 / 1e-12 / 1e-5; the state vector and everything read from it is held to
100 times that for f64 and df, and to 1e-4 for mixed, whose noise floor also
drops Schmidt values below 5e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "df": 1e-10, "mixed": 1e-4}


def _random(rng, n, decay=0.0):
    v = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    m = v.reshape(1 << (n // 2), -1)
    if decay:  # graded spectrum at the middle bond
        u, s, vh = np.linalg.svd(m, full_matrices=False)
        v = (u * 10.0 ** (-decay * np.arange(s.size) / max(1, s.size - 1))) @ vh
    return (v / np.linalg.norm(v)).reshape(-1)


def _low_rank(rng, n, r):
    h = n // 2
    a = np.linalg.qr(rng.standard_normal((1 << h, r)) + 1j * rng.standard_normal((1 << h, r)))[0]
    b = np.linalg.qr(rng.standard_normal((1 << (n - h), r)) + 1j * rng.standard_normal((1 << (n - h), r)))[0]
    s = np.linspace(1.0, 0.3, r)
    return ((a * s) @ b.T / np.linalg.norm(s)).reshape(-1)


def _equal(n):
    """Maximally entangled halves: every Schmidt value of the middle bond equal."""
    h = n // 2
    return np.eye(1 << h, dtype=complex).reshape(-1) / np.sqrt(1 << h)


def _haar4(rng):
    q, r = np.linalg.qr(rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


CASES = [("product", 4, 8), ("random", 2, 8), ("random", 3, 8), ("random", 7, 5), ("random", 8, 16), ("random", 9, 15),
         ("random", 10, 31), ("random", 10, 32), ("random", 12, 33), ("random", 12, 64), ("random", 13, 35),
         ("graded", 8, 16), ("graded", 10, 32), ("low", 8, 3), ("low", 10, 16), ("equal", 8, 16), ("equal", 10, 32)]


def _pair(pkg, ref, kind, n, chi, prec, seed):
    rng = np.random.default_rng(seed)
    psi = {"product": lambda: np.eye(1, 1 << n, 3, dtype=complex).reshape(-1), "random": lambda: _random(rng, n),
           "graded": lambda: _random(rng, n, 6.0), "low": lambda: _low_rank(rng, n, chi), "equal": lambda: _equal(n)}[kind]()
    m = ref.from_vector(psi, ref.Trunc.both(chi, 1e-10))
    g = pkg.MPS.from_parts(m.data, m.svals, pkg.Trunc.both(chi, 1e-10), prec)
    return rng, m, g


def _compare(g, m, n, tol):
    floor = 1e-4 if tol > 1e-6 else 1e-8  # values that the mode keeps to their own accuracy
    for b in range(n - 1):
        a, r = g.svals(b), m.svals[b]
        k = int(np.sum(r > floor))
        assert a.size >= k and np.max(np.abs(a[:k] - r[:k])) < tol, (b, a.size, r.size)
        assert abs(g.entropy_vn(b) - m.entropy_vn(b)) < tol
        assert abs(g.entropy_ry_schmidt(2.0, b) - m.entropy_ry_schmidt(2.0, b)) < tol
    for k in range(n):
        assert np.max(np.abs(g.probs(k) - m.probs(k))) < tol
    assert np.max(np.abs(g.contract() - m.contract())) < tol
    assert g.device_status() == 0


@pytest.mark.parametrize("prec", ["f64", "df", "mixed"])
@pytest.mark.parametrize("kind,n,chi", CASES)
def test_gate_on_small_bond(pkg, ref, kind, n, chi, prec):
    rng, m, g = _pair(pkg, ref, kind, n, chi, prec, 11)
    for k in sorted({0, n // 2 - 1, n - 2}):
        u = _haar4(rng)
        m.apply_unitary2(k, u)
        g.apply_unitary2(k, u)
    u1 = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0]
    m.apply_unitary1(n // 2, u1)
    g.apply_unitary1(n // 2, u1)
    # truncation amplifies: compare states at the scale of the kept weight
    _compare(g, m, n, TOL[prec])


@pytest.mark.parametrize("prec", ["f64", "df", "mixed"])
@pytest.mark.parametrize("kind,n,chi", [c for c in CASES if c[1] > 2])
def test_measurement_sweep_on_small_bonds(pkg, ref, kind, n, chi, prec):
    _, m, g = _pair(pkg, ref, kind, n, chi, prec, 12)
    # the likelier outcome: a projection onto a tiny one would amplify rounding
    p = int(np.argmax(m.local_probs(n // 2)))
    a, b = g.measure_postsel_prob(n // 2, p), m.measure_postsel_prob(n // 2, p)
    assert abs(a - b) < TOL[prec]
    _compare(g, m, n, TOL[prec])


@pytest.mark.parametrize("kind,n,chi", [("random", 2, 2), ("random", 12, 64), ("random", 13, 64), ("random", 14, 128),
                                        ("graded", 12, 64), ("low", 12, 5), ("equal", 10, 32)])
def test_from_vector_sites_on_one_cta(pkg, ref, kind, n, chi):
    """k_fv_local up to its limit (n = 13) and around it: sites that it leaves to
    the rounds (the middle of n = 14), rank-deficient and degenerate spectra."""
    rng = np.random.default_rng(13)
    psi = {"random": lambda: _random(rng, n), "graded": lambda: _random(rng, n, 6.0),
           "low": lambda: _low_rank(rng, n, chi), "equal": lambda: _equal(n)}[kind]()
    g, m = pkg.MPS.from_vector(psi), ref.from_vector(psi)
    for b in range(n - 1):
        a, r = g.svals(b), m.svals[b]
        k = int(np.sum(r > 1e-12))
        assert a.size >= k and np.max(np.abs(a[:k] - r[:k])) < 1e-12, b
    assert np.max(np.abs(g.contract() - psi)) < 1e-12
