"""On-chip Lanczos (qcmg_chip.cu) at the sizes where it can go wrong: one
state to the largest sector that fits, tiles of 64 states with remainders,
clusters larger than the number of tiles, vectors kept or recomputed, against
dense diagonalization or the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sector(L, nup, ndn, seed):
    """(engine Hamiltonian, oracle sector) of a random open chain."""
    import pyqcm_gb300 as pg
    import qcm_oracle as qo
    rng = np.random.default_rng(seed)
    t = [(i, i + 1, float(rng.uniform(-1, 1))) for i in range(L - 1)]
    e = [(i, i, float(rng.uniform(-1, 1))) for i in range(L)]
    ops = {"h": ("one-body", t + e + [(i + L, j + L, v) for i, j, v in t + e]),
           "U": ("interaction", [(i, i + L, float(rng.uniform(1, 4))) for i in range(L)])}
    m = pg.ClusterModel(L)
    for name, (typ, els) in ops.items():
        m.new_operator(name, typ, els)
    vals = {"h": 1.0, "U": 1.0}
    up, dn, pr = qo.combine_terms(ops, vals, L)
    return pg.Hamiltonian(m, vals, f"R0:N{nup + ndn}:S{nup - ndn}"), qo.Sector(L, nup, ndn, up, dn, pr)


# dims 1, 3, 9, 63 = 7 x 9, 64 = 8 x 8, 100, 1,225, 15,876, 16,170 = 210 x 77 is out of reach of a
# chain sector; 252 x 45 = 11,340 has unequal factors
@pytest.mark.parametrize("L,nup,ndn", [(3, 0, 3), (3, 1, 0), (3, 1, 2), (8, 1, 1), (5, 2, 3), (7, 3, 4), (9, 4, 4), (10, 5, 2)])
def test_ground_state(L, nup, ndn):
    H, S = _sector(L, nup, ndn, L + nup)
    x0 = np.random.default_rng(3).normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    e0, psi, alpha, beta = H.lanczos(x0=x0, tol=1e-10)
    assert abs(np.linalg.norm(psi) - 1) < 1e-6  # the replayed vector's norm, the recurrence's own accuracy
    r = S.matvec(psi) - e0 * psi
    # the Ritz residual is below tol at the last step; psi adds its rounding
    assert np.linalg.norm(r) < 1e-7
    if H.dim <= 1300:
        A = np.array([S.matvec(v) for v in np.eye(H.dim)])
        assert abs(e0 - np.linalg.eigvalsh(A)[0]) < 1e-10 * max(1.0, abs(e0))
    assert len(alpha) == len(beta)


def test_largest_sector_and_the_next():
    """16,384 states is the limit: 126 x 126 is on chip, 210 x 120 is not;
    both give the energy of the fully reorthogonalized recurrence."""
    for L, nup, ndn in ((9, 4, 5), (10, 4, 3)):
        H, _ = _sector(L, nup, ndn, 1)
        e0 = H.lanczos(tol=1e-11, want_psi=False)[0]
        e1 = H.lanczos(tol=1e-11, want_psi=False, reorth=200)[0]
        assert abs(e0 - e1) < 1e-10 * abs(e1)


def test_batch_equals_single_for_any_cluster_size():
    """Clusters of 16 (one sector), 8, 4, 2 and 1 CTAs give the same bits."""
    import pyqcm_gb300 as pg
    hs = [_sector(6, 3, 3, k)[0] for k in range(320)]
    one = [h.lanczos() for h in hs[:3]]
    for n in (2, 40, 80, 160, 320):
        got = pg.lanczos_batch(hs[:n], want_psi=True)
        for (e, psi, it), (e1, psi1, al, _) in zip(got, one):
            assert e == e1 and it == len(al) and np.array_equal(psi, psi1)


def test_no_convergence_is_reported():
    import pyqcm_gb300 as pg
    H, _ = _sector(8, 4, 4, 5)
    with pytest.raises(pg.QcmgError) as err:
        H.lanczos(max_iter=20)
    assert err.value.code == -4
    res = pg.lanczos_batch([H], max_iter=20, raise_errors=False)
    assert res[0][3] is not None and res[0][3].code == -4


def _green(e, Q, zs):
    return np.einsum("am,zm,bm->zab", Q, 1.0 / (zs[:, None] - e), Q)


def _oracle_green(S, phi, zs):
    """The oracle's run of the same recurrence with the same stopping rule: a
    random start vector's Green function at the centre of the spectrum is not
    converged when the lowest eigenvalue is, so the exact resolvent is not
    what a correct run gives."""
    import qcm_oracle as qo
    return _green(*qo.build_Q_matrix(S.mult_add, list(phi), S.dim), zs)


@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 8, 9, 12, 13])
@pytest.mark.parametrize("L,nup,ndn", [(6, 3, 3), (7, 3, 4)])
@pytest.mark.parametrize("start", ["free", "dependent"])
def test_band_lanczos(p, L, nup, ndn, start):
    """The Green function of p start vectors at imaginary frequencies: on chip
    for p <= 12, on the general path above and where a vector deflates."""
    H, S = _sector(L, nup, ndn, 11)
    rng = np.random.default_rng(p)
    phi = rng.normal(size=(p, S.dim))
    if start == "dependent" and p > 1:
        phi[-1] = phi[0]
    phi /= np.linalg.norm(phi, axis=1)[:, None]
    zs = np.array([1.0j, 4.0j, 20.0j])
    e, Q = H.build_Q_matrix(phi)
    G = _green(e, Q, zs)
    ref = _oracle_green(S, phi, zs)
    # the two runs stop at the same step; their rounding stays below 1e-8 in G
    assert np.max(np.abs(G - ref)) < 1e-8 * max(1.0, np.max(np.abs(ref)))


@pytest.mark.parametrize("L,nup,ndn,p", [(2, 1, 1, 2), (3, 1, 1, 3), (4, 2, 2, 4), (5, 2, 2, 4)])
def test_band_lanczos_exhausts_small_sectors(L, nup, ndn, p):
    """Krylov spaces that end (a vector deflates)."""
    H, S = _sector(L, nup, ndn, 4)
    phi = np.random.default_rng(2).normal(size=(p, S.dim))
    zs = np.array([0.7j, 3.0j])
    e, Q = H.build_Q_matrix(phi)
    G = _green(e, Q, zs)
    ref = _oracle_green(S, phi, zs)
    assert np.max(np.abs(G - ref)) < 1e-8 * np.max(np.abs(ref))


@pytest.mark.parametrize("cap", [2, 4, 5, 8, 9, 12, 13, 16, 17, 40, 64, 65, 90])
@pytest.mark.parametrize("L,nup,ndn", [(6, 3, 3), (7, 3, 4)])
def test_reorthogonalized_lists(cap, L, nup, ndn):
    """The projection kernels at every list size they are built for and past
    64 vectors, on 400 (pairs of elements) and 1,225 states (odd): the energy
    of dense diagonalization, restarting at the cap."""
    H, S = _sector(L, nup, ndn, 21)
    e0 = H.lanczos(tol=1e-6, max_iter=4000, reorth=cap, want_psi=False)[0]
    A = np.array([S.matvec(v) for v in np.eye(S.dim)])
    # the energy's error is the square of the residual over the gap (> 1e-3)
    assert abs(e0 - np.linalg.eigvalsh(A)[0]) < 1e-8
