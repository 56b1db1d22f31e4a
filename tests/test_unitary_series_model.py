"""The series that makes V unitary to the working precision (unit_entry in
tn_local.cuh, team_correction in tn_team.cuh) and the one of a refinement step
(unitary_step), restated in numpy at the limits that the kernels accept (read
from their source): what the truncated series leaves has to be below the
precision they work in, whatever the entries' pattern is.  Limits on single
entries do not give that: 64 x 64 of them at 2e-5 leave 1e-11.

Tolerances: the terms left out, as the comments derive them (1e-15 in the
shared-memory path, 2^-47 on the team), plus float64's own rounding of the
check, 4 c 2^-53."""
import pathlib
import re

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "tensor-net_gb300" / "csrc"


def _limit(name):
    text = (CSRC / "tn_local.cuh").read_text() + (CSRC / "tn_team.cuh").read_text()
    return float(re.search(rf"{name} = ([0-9.e-]+)f", text).group(1))


def _pattern(kind, c, rng):
    """Hermitian, zero diagonal."""
    if kind == "random":
        o = rng.standard_normal((c, c)) + 1j * rng.standard_normal((c, c))
    elif kind == "phases":  # entries of one size
        o = np.exp(2j * np.pi * rng.random((c, c)))
    else:  # one direction: spectral, Frobenius and row-sum norms alike
        v = np.exp(2j * np.pi * rng.random(c))
        o = np.outer(v, v.conj())
    o = np.triu(o, 1)
    return o + o.conj().T


def _left(s, w):
    i = np.eye(len(s))
    return np.linalg.norm((i + w).conj().T @ (i + s) @ (i + w) - i, 2)


@pytest.mark.parametrize("c", [2, 8, 31, 64])
@pytest.mark.parametrize("kind", ["random", "phases", "one"])
def test_shared_memory_path(kind, c):
    o = _pattern(kind, c, np.random.default_rng(c))
    tol = 1e-15 + 4 * c * 2.0 ** -53
    for name in ("kOffSquare", "kOffMax"):
        s = o * (_limit(name) / np.linalg.norm(o))
        q = s.astype(np.complex64)
        sq = q @ q
        hi = np.float32(0.375) * sq
        if name == "kOffMax":
            hi = hi - np.float32(0.3125) * (q @ sq)
        assert _left(s, -s / 2 + hi) < tol, name


@pytest.mark.parametrize("c", [65, 200, 512])
@pytest.mark.parametrize("kind", ["random", "phases", "one"])
def test_team(kind, c):
    o = _pattern(kind, c, np.random.default_rng(c))
    tol = 2.0 ** -47 + 4 * c * 2.0 ** -53
    for name in ("kTeamSquare", "kTeamMax"):
        s = o * (_limit(name) / np.sqrt(np.abs(o @ o).sum(1).max()))
        sq = s @ s
        hi = 0.375 * sq
        if name == "kTeamMax":
            hi = hi + sq @ (-0.3125 * s + 35 / 128 * sq)
        assert _left(s, -s / 2 + hi) < tol, name


@pytest.mark.parametrize("c", [2, 16, 64])
@pytest.mark.parametrize("kind", ["random", "phases", "one"])
def test_refinement_step(kind, c):
    k = 1j * _pattern(kind, c, np.random.default_rng(c))  # anti-Hermitian
    k *= _limit("kStepMax") / np.linalg.norm(k)
    y = k @ k
    z = y.astype(np.complex64) @ (np.float32(0.5) * k + np.float32(0.375) * y).astype(np.complex64)
    q = np.eye(c) + k + y / 2 + z
    assert np.linalg.norm(q.conj().T @ q - np.eye(c), 2) < 1e-15 + 4 * c * 2.0 ** -53


def test_first_order_corrections():
    """A + A K: K's square, left out, stays below the working precision."""
    src = (CSRC / "tn_local.cuh").read_text()
    f64, df = map(float, re.search(r"kFloatApply = .*\? ([0-9.e-]+)f : ([0-9.e-]+)f", src).groups())
    assert f64 ** 2 < 2.0 ** -53 and df ** 2 < 2.0 ** -47
    assert _limit("kSlight") ** 2 / 2 <= 2.0 ** -47
