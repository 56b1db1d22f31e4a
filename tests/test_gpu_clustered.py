"""Mixed precision on clustered spectra (groups of Schmidt values with relative
gaps of 1e-3 to 1e-6) wider than the double-float small-bond path: the vectors
that the float sweeps leave are orthogonal to their threshold, 4 sqrt(ell)
2^-23, not just to the size at which a separated spectrum would converge.  On
the cluster of the single-state API, in svd_local on one CTA (up to 128 vectors)
and in the block Jacobi (beyond).

Tolerance on an off-diagonal entry of B B^H, B the new right tensor with its
Lambda: the threshold, and a quarter of it for the rounding of a Gram entry and
of the stored Gamma."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clustered(n, group, gap, seed):
    rng = np.random.default_rng(seed)
    d = 1 << (n // 2)
    u, v = (np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))[0] for _ in range(2))
    level = np.repeat(np.linspace(1.0, 0.4, d // group), group)  # groups of nearly equal values
    s = level * (1.0 + gap * np.arange(d))
    s /= np.linalg.norm(s)
    return ((u * s) @ v).reshape(-1)


def _off(gamma, lam):
    b = (gamma * lam[None, None, :]).reshape(gamma.shape[0], -1)
    g = b @ b.conj().T
    return np.abs(g - np.diag(np.diag(g))).max()


@pytest.mark.parametrize("group,gap", [(16, 1e-3), (16, 1e-5), (128, 1e-4), (128, 1e-5), (128, 1e-6)])
@pytest.mark.parametrize("n,how", [(14, "cluster"), (14, "batch"), (16, "cluster"), (16, "batch")])
def test_vectors_of_a_clustered_spectrum_are_orthogonal(pkg, n, how, group, gap):
    psi, tr, k = _clustered(n, group, gap, 17), pkg.Trunc.both(1 << (n // 2), 1e-10), n // 2 - 1
    parts = pkg.MPS.from_vector(psi, tr, "f64").export_parts()
    rng = np.random.default_rng(18)
    local = [np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0] for _ in range(2)]
    gate = np.kron(*local)  # mixes the vectors, keeps the spectrum
    if how == "cluster":
        g = pkg.MPS.from_parts(*parts, tr, "mixed")
        g.apply_unitary2(k, gate)
        gammas, lams, status = *g.export_parts(), g.device_status()
    else:
        b = pkg.Batch([n], [tr], "mixed")
        b.import_state(0, *parts, tr)
        b.step([0], [([k], gate[None], np.zeros(0), np.zeros(0))])
        gammas, lams, status = *b.export_parts(0), b.device_status()
    assert status == 0 and len(lams[k]) == 1 << (n // 2)
    assert np.max(np.abs(np.sort(lams[k])[::-1] - parts[1][k])) < 1e-5
    tol = 4 * np.sqrt(2 * len(lams[k + 1])) * 2.0 ** -23
    assert _off(gammas[k + 1], lams[k + 1]) < 1.25 * tol
