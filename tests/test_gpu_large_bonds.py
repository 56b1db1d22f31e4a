"""Bond operations wider than the shared-memory path (tn_team.cuh, tn_oz.cuh):
vector counts just above svd_local's limit, odd numbers of 16-column blocks,
products with ragged tiles, graded, rank-deficient and degenerate spectra; on
the cluster of the single-state API and on the one CTA of a batch.  Against
the oracle on the same states.

Tolerances as in test_gpu_small_bonds.py: a bond operation's backward error is
a small multiple of sqrt(c) eps (c <= 256; eps = 2^-47, 2^-24), below 1e-12 and
1e-5, and what is read from the state is held to 100 times that (df) and to
1e-4 (mixed, whose noise floor also drops Schmidt values below 1e-5)."""
import numpy as np
import pytest

from test_gpu_small_bonds import _compare, _equal, _haar4, _low_rank, _random

pytestmark = pytest.mark.gpu
TOL = {"df": 1e-10, "mixed": 1e-4}
CASES = [("random", 13, 33), ("random", 14, 47), ("random", 14, 100),
         ("graded", 13, 64), ("low", 13, 40), ("equal", 14, 128)]


def _state(kind, n, chi, seed):
    rng = np.random.default_rng(seed)
    psi = {"random": lambda: _random(rng, n), "graded": lambda: _random(rng, n, 5.0),
           "low": lambda: _low_rank(rng, n, chi), "equal": lambda: _equal(n)}[kind]()
    return rng, psi


@pytest.mark.parametrize("prec", ["df", "mixed"])
@pytest.mark.parametrize("kind,n,chi", CASES)
def test_gate_and_measurement_on_large_bond(pkg, ref, kind, n, chi, prec):
    rng, psi = _state(kind, n, chi, 21)
    m = ref.from_vector(psi, ref.Trunc.both(chi, 1e-10))
    tr = pkg.Trunc.both(chi, 1e-10)
    g = pkg.MPS.from_parts(m.data, m.svals, tr, prec)
    b = pkg.Batch([n], [tr], prec)
    b.import_state(0, m.data, m.svals, tr)
    k, u, none = n // 2 - 1, _haar4(rng), np.zeros(0)
    m.apply_unitary2(k, u)
    g.apply_unitary2(k, u)
    b.step([0], [([k], u[None], none, none)])
    _compare(g, m, n, TOL[prec])
    s = b.svals(0, k)
    w = min(s.size, m.svals[k].size)
    assert np.max(np.abs(s[:w] - m.svals[k][:w])) < TOL[prec] and b.device_status() == 0
    # the likelier outcome, then the refactor sweep
    p = int(np.argmax(m.local_probs(k)))
    m.apply_meas_prob_layer([k], posts=[p])
    g.apply_meas_prob_layer([k], [0.0], [p])
    b.step([0], [(none, np.zeros((0, 4, 4)), [k], [0.0])], posts=[[p]])
    _compare(g, m, n, TOL[prec])
    for bd in range(n - 1):
        s, r = b.svals(0, bd), m.svals[bd]
        w = int(np.sum(r > (1e-4 if prec == "mixed" else 1e-8)))
        assert s.size >= w and np.max(np.abs(s[:w] - r[:w])) < TOL[prec], bd
    assert b.device_status() == 0


def test_same_bits_on_teams_of_every_size(pkg):
    """A double-float layer on clusters of eight (2 trajectories), of four (24)
    and on single CTAs (160, more than there are SMs): outcomes, probabilities,
    entropies and Schmidt values with the same bits."""
    n, chi = 14, 100
    _, psi = _state("random", n, 128, 22)
    tr = pkg.Trunc.both(chi, 1e-10)
    m = pkg.MPS.from_vector(psi, tr, "df")
    parts = m.export_parts()
    layers = [pkg.gen_layer(31, 0, t, n, 0.2) for t in range(2)]
    got = []
    for count in (2, 24, 160):
        b = pkg.Batch([n] * count, [tr] * count, "df")
        for i in (0, count - 1):
            b.import_state(i, *parts, tr)
        out = []
        for la in layers:
            recs, ent = b.step(list(range(count)), [la] * count)
            out += [recs[0], recs[-1], ent[0], ent[-1]]
        out += [b.svals(i, k).tolist() for i in (0, count - 1) for k in range(n - 1)]
        assert b.device_status() == 0
        b.close()
        got.append(out)
    assert got[0] == got[1] == got[2]
