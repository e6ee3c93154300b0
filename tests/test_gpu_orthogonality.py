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


def test_vectors_one_by_one_when_memory_is_short():
    """The kept vectors are allocated 512 MB at a time; where the device has no
    room for that the run goes on with single ones (3,312,400 states, 19 vectors
    a time, 22 steps: the limit ends the run, not the memory)."""
    import models
    import pyqcm_gb300 as pg
    import torch
    ns, _, ops = models.hubbard_cluster(4, 4)
    params = {"t": 1.0, "U": 8.0, "mu": 4.0}
    m = pg.ClusterModel(ns)
    for name, (typ, els) in ops.items():
        if name in params:
            m.new_operator(name, typ, els)
    H = pg.Hamiltonian(m, params, "R0:N8:S0")
    x0 = np.random.default_rng(1).normal(size=H.dim)
    x0 /= np.linalg.norm(x0)

    def steps():
        with pytest.raises(pg.QcmgError) as err:
            H.lanczos(x0=x0, tol=1e-300, max_iter=22, reorth=100)
        return err.value.code

    assert steps() == -4  # also allocates the product's buffers
    torch.cuda.empty_cache()
    vector = 8 * H.dim
    span = (512 << 20) // vector * vector
    fill = torch.empty(torch.cuda.mem_get_info()[0] - span - 8 * vector, dtype=torch.uint8, device="cuda")
    try:
        assert span < torch.cuda.mem_get_info()[0] < 2 * span
        assert steps() == -4
    finally:
        del fill
        torch.cuda.empty_cache()
