"""float64 bond operations on a theta far from norm 1: operators of any finite size
are accepted, and what they do to the state's norm is divided out again, so the
result is that of the operator at its own size.  Against the oracle with the
unscaled operator; the scale is a rounding of every entry, so the tolerance is
that of test_gpu_small_bonds.py."""
import numpy as np
import pytest

from test_gpu_small_bonds import TOL, _compare, _haar4, _pair

pytestmark = pytest.mark.gpu
CASES = [("random", 8, 16), ("random", 10, 31), ("graded", 10, 32), ("low", 10, 16), ("equal", 10, 32),
         ("random", 13, 40)]


@pytest.mark.parametrize("scale", [1e-70, 1e-20, 1e-12, 1e-4, 1e6, 1e12, 1e25, 1e70])
@pytest.mark.parametrize("kind,n,chi", CASES)
def test_scaled_gate(pkg, ref, kind, n, chi, scale):
    rng, m, g = _pair(pkg, ref, kind, n, chi, "f64", 31)
    for k in sorted({0, n // 2 - 1, n - 2}):
        u = _haar4(rng)
        m.apply_unitary2(k, u)
        g.apply_unitary2(k, scale * u)
    _compare(g, m, n, TOL["f64"])


@pytest.mark.parametrize("scale", [1e-20, 1e-12, 1e-4, 1e12, 1e25])
@pytest.mark.parametrize("kind,n,chi", CASES)
def test_refactor_sweep_over_a_scaled_site(pkg, ref, kind, n, chi, scale):
    rng, m, g = _pair(pkg, ref, kind, n, chi, "f64", 32)
    u = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0]
    m.apply_unitary1(n // 2, u)
    g.apply_unitary1(n // 2, scale * u)
    p = int(np.argmax(m.local_probs(1)))
    a, b = g.measure_postsel_prob(1, p), m.measure_postsel_prob(1, p)
    assert abs(a - b) < TOL["f64"]
    _compare(g, m, n, TOL["f64"])
