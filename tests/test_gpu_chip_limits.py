"""On-chip Lanczos and band Lanczos (qcmg_chip.cu, qcmg_chip_band.cu) at the
limits of their ranges: the largest step counts and sectors around a tile of
32 states."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(L, nup, ndn, U):
    """The sector of an open chain with t = 1, on the FP64 path."""
    import pyqcm_gb300 as pg
    els = [(i, i + 1, -1.0) for i in range(L - 1)]
    m = pg.ClusterModel(L)
    m.new_operator("t", "one-body", els + [(i + L, j + L, v) for i, j, v in els])
    m.new_operator("U", "interaction", [(i, i + L, 1.0) for i in range(L)])
    H = pg.Hamiltonian(m, {"t": 1.0, "U": U}, f"R0:N{nup + ndn}:S{nup - ndn}")
    H.set_path(False)
    return H


@pytest.mark.parametrize("max_iter", [1000, 2**31 - 1])
def test_vector_of_a_long_run(max_iter):
    """A run of more than 320 steps (its vectors are then recomputed) with its
    vector, however many steps the caller allows: an attractive pair and one
    electron more on 31 sites, 14,415 states."""
    import pyqcm_gb300 as pg
    from pyqcm_gb300 import _lib
    H = _chain(31, 1, 2, -12.0)
    x0 = np.random.default_rng(3).normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    e0, psi, steps = _lib.c_double(), np.zeros(H.dim), _lib.c_int()
    tol = 1e-11
    _lib.check(pg.lib().qcmg_lanczos_ground_state(H._h, _lib.ptr(x0), 0, tol, max_iter, 0, e0, _lib.ptr(psi), steps,
                                                  None, None, 0))
    assert steps.value > 320
    # the Ritz residual and the rounding of the recomputed run: a few hundred
    # steps of products with |H| < 30, 30 x 1e3 x 2.2e-16 = 7e-12
    assert np.linalg.norm(H.matvec(psi) - e0.value * psi) < tol + 1e-10
@pytest.mark.parametrize("L,nup,ndn", [(31, 1, 0), (32, 1, 0), (7, 3, 0), (31, 1, 1), (32, 1, 1)])
def test_sectors_around_a_tile(L, nup, ndn):
    """31, 32, 35, 961 and 1,024 states: the last tile of 32 full, one short
    and nearly empty, fewer tiles than CTAs; the energy and the Green function
    of three start vectors against dense diagonalization."""
    H = _chain(L, nup, ndn, 4.0)
    A = np.array([H.matvec(v) for v in np.eye(H.dim)])
    e, W = np.linalg.eigh(A)
    rng = np.random.default_rng(L)
    x0 = rng.normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    e0, psi, _, _ = H.lanczos(x0=x0, tol=1e-10, reorth=0)
    # the energy's error is the square of the residual over the gap (> 1e-3)
    assert abs(e0 - e[0]) < 1e-12 * H.dim
    assert np.linalg.norm(A @ psi - e0 * psi) < 1e-8
    # start vectors in the span of six eigenvectors: the band ends by itself
    # (deflation) and its Green function is exact
    phi = rng.normal(size=(3, 6)) @ W[:, ::max(1, H.dim // 6)][:, :6].T
    phi /= np.linalg.norm(phi, axis=1)[:, None]
    zs = np.array([0.5j, 2.0j, 10.0j])
    eb, Q = H.build_Q_matrix(phi)
    G = np.einsum("am,zm,bm->zab", Q, 1.0 / (zs[:, None] - eb), Q)
    P = phi @ W
    ref = np.einsum("am,zm,bm->zab", P, 1.0 / (zs[:, None] - e), P)
    assert np.max(np.abs(G - ref)) < 1e-8


@pytest.mark.parametrize("p", [1, 2, 4, 9])
@pytest.mark.parametrize("nup,ndn", [(4, 3), (4, 4)])
def test_bands_of_large_sectors(p, nup, ndn):
    """10,584 and 15,876 states (9-site chain): the vector and the band's
    parts fill the shared memory of sixteen CTAs. Start vectors in the span of
    a Krylov space of few steps are not to be had here, so the moments
    <phi_i| H^k |phi_j> up to k = 3 are compared: they are those of the band
    after four steps of each vector."""
    H = _chain(9, nup, ndn, 4.0)
    rng = np.random.default_rng(p)
    phi = rng.normal(size=(p, H.dim))
    phi /= np.linalg.norm(phi, axis=1)[:, None]
    e, Q = H.build_Q_matrix(phi)
    v = phi.copy()
    for k in range(4):
        ref = phi @ v.T
        # |H| < 30: k products' rounding of 30^k, and the recurrence's of as many
        assert np.max(np.abs((Q * e ** k) @ Q.T - ref)) < 1e-12 * 30.0 ** k, k
        v = np.array([H.matvec(x) for x in v])
