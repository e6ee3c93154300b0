"""The reorthogonalized Lanczos basis: one Gram-Schmidt pass, and a second
where the first took away half of the norm's square or more, keeps it
orthogonal to rounding long after extreme eigenvalues have converged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _copies(a, b, ev):
    """Pairs of eigenvalues of the tridiagonal matrix at one eigenvalue in ev."""
    t = np.sort(np.linalg.eigvalsh(np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1)))
    at = [int(np.argmin(np.abs(ev - x))) for x in t if np.min(np.abs(ev - x)) < 1e-8]
    return len(at) - len(set(at))


@pytest.mark.parametrize("L,nup,ndn", [(6, 3, 3), (7, 3, 4)])
@pytest.mark.parametrize("tol", [1e-6, 1e-9, 1e-12])
def test_no_copies_and_unit_vector(L, nup, ndn, tol):
    """A site at energy 60 splits the spectrum: the upper end converges in a
    few steps, and a basis that loses its orthogonality then finds it again
    and again."""
    import pyqcm_gb300 as pg
    rng = np.random.default_rng(L)
    els = [(i, i + 1, float(rng.uniform(0.5, 1.5))) for i in range(L - 1)]
    els += [(i, i, float(rng.uniform(-1, 1)) + (60.0 if i == 2 else 0.0)) for i in range(L)]
    m = pg.ClusterModel(L)
    m.new_operator("h", "one-body", els + [(i + L, j + L, v) for i, j, v in els])
    m.new_operator("U", "interaction", [(i, i + L, float(rng.uniform(1, 4))) for i in range(L)])
    H = pg.Hamiltonian(m, {"h": 1.0, "U": 1.0}, f"R0:N{nup + ndn}:S{nup - ndn}")
    H.set_path(False)
    x0 = rng.normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    e0, psi, a, b = H.lanczos(x0=x0, tol=tol, max_iter=350, reorth=350)
    A = np.array([H.matvec(v) for v in np.eye(H.dim)])
    ev = np.linalg.eigvalsh(A)
    assert np.min(np.diff(ev)) > 1e-7  # a copy is one of the basis, not of the spectrum
    assert _copies(a, b, ev) == 0
    # |psi|^2 - 1 = z^T (V^T V - 1) z: every pass leaves a few roundings per vector
    assert abs(psi @ psi - 1) < 4 * len(a) * np.finfo(float).eps
    # the energy's error is the square of the residual over the gap, and rounding of |H| < 200
    assert abs(e0 - ev[0]) < tol ** 2 / (ev[1] - ev[0]) + 1e-12


def test_a_plain_run_finds_copies():
    """The same matrix without reorthogonalization does find copies: the test
    above would see a basis that is not orthogonal."""
    rng = np.random.default_rng(0)
    ev = np.concatenate([np.linspace(0, 12, 300), [60.0, 121.0]])
    x = rng.normal(size=len(ev))
    r, q, a, b = x / np.linalg.norm(x), np.zeros(len(ev)), [], []
    for j in range(90):
        if j:
            r, q = q / b[-1], -b[-1] * r
        q = q + ev * r
        a.append(r @ q)
        q = q - a[-1] * r
        b.append(np.linalg.norm(q))
    assert _copies(np.array(a), np.array(b), ev) > 0
