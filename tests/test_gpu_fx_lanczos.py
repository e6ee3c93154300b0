"""The fixed-point path on sectors that reach it: Lanczos runs above 16,384
states with their vector (kept, recomputed, and recomputed after the room for
the kept vectors ran out), a long run without convergence, and products of
FP64 vectors from 2^21 states on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PARAMS = {"t": 1.0, "U": 8.0, "mu": 4.0}


def _hubbard(nx, ny, nup, ndn):
    import models
    import pyqcm_gb300 as pg
    ns, nb, ops = models.hubbard_cluster(nx, ny)
    m = pg.ClusterModel(ns, nb)
    for name, (typ, els) in ops.items():
        if name in PARAMS:
            m.new_operator(name, typ, els)
    H = pg.Hamiltonian(m, PARAMS, f"R0:N{nup + ndn}:S{nup - ndn}")
    assert H.fx_available()
    return H


def _residual(H, e0, psi):
    """|H psi - e0 psi| with the product on FP64 vectors, on the device."""
    import torch
    x = torch.from_numpy(psi).cuda()
    y = torch.empty_like(x)
    H.matvec_device(x.data_ptr(), y.data_ptr())
    return float(torch.linalg.vector_norm(y - e0 * x))


@pytest.mark.parametrize("shape,nup,ndn", [((10, 1), 5, 5), ((15, 1), 3, 2), ((4, 3), 5, 6)])
def test_ground_state_and_vector(shape, nup, ndn):
    """63,504, 47,775 (odd) and 731,808 states against the FP64 path."""
    H = _hubbard(*shape, nup, ndn)
    assert H.dim > 16384
    x0 = np.random.default_rng(1).normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    tol = 1e-11
    e0, psi, _, _ = H.lanczos(x0=x0, tol=tol, reorth=0)
    # the Ritz residual; a few hundred steps' rounding of |H| < 100 is below 1e-11
    assert _residual(H, e0, psi) < 2 * tol + 1e-11
    assert abs(np.linalg.norm(psi) - 1) < 1e-10
    H.set_path(False)
    e1, psi1, _, _ = H.lanczos(x0=x0, tol=tol, reorth=0)
    assert abs(e0 - e1) < 1e-11 * abs(e1)
    # the vectors' error is the residual over the gap (> 1e-2)
    assert abs(abs(psi @ psi1) / np.linalg.norm(psi1) - 1) < 1e-8


def test_vector_recomputed_where_the_basis_is_too_large():
    """64,128,064 states: 300 vectors are more than a quarter of the memory."""
    import torch
    H = _hubbard(4, 4, 6, 6)
    assert 300 * 8 * H.dim > torch.cuda.mem_get_info()[0] / 4
    tol = 1e-9
    e0, psi, al, _ = H.lanczos(tol=tol, reorth=0)
    assert _residual(H, e0, psi) < 2 * tol
    # seeded start vector of norm one: the recurrence keeps it
    assert abs(np.linalg.norm(psi) - 1) < 1e-7


def test_vector_recomputed_when_the_room_runs_out():
    """Vectors are kept in spans of 64 while they fit in a quarter of the free
    memory. With room for a few more than the steps of the run, the last span
    does not fit: the vector is recomputed, to the same bits."""
    import torch
    H = _hubbard(4, 3, 6, 6)
    x0 = np.random.default_rng(2).normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    e0, psi, al, be = H.lanczos(x0=x0, tol=1e-12, reorth=0)
    n = len(al)
    assert 140 < n < 290
    spans = (n + 2 + 63) // 64  # the last of them must not fit
    slots = (n + 2 + 64 * spans - 1) / 2
    if not n + 2 < slots < 64 * spans - 1:
        pytest.skip("the run's steps fill their last span")
    torch.cuda.empty_cache()
    leave = int(4 * slots * 8 * ((H.dim + 31) // 32 * 32))
    fill = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        room = torch.cuda.mem_get_info()[0] / 4 / (8 * ((H.dim + 31) // 32 * 32))
        assert n + 2 < room < 64 * spans
        e1, psi1, al1, be1 = H.lanczos(x0=x0, tol=1e-12, max_iter=n, reorth=0)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert e1 == e0 and np.array_equal(al, al1) and np.array_equal(be, be1)
    assert np.array_equal(psi, psi1)


def test_long_run_stays_finite():
    """700 steps without convergence: the lazy vector scale must not drift out
    of double range; the run ends with NOCONV, not a numerical breakdown."""
    import pyqcm_gb300 as pg
    H = _hubbard(10, 1, 5, 5)
    with pytest.raises(pg.QcmgError) as err:
        H.lanczos(tol=1e-300, max_iter=700, reorth=0, want_psi=False)
    assert err.value.code == -4, err.value


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("pinned", [True, False])
def test_large_products_on_host_vectors(offset, pinned):
    """2,944,656 states (13-site chain): y in page-locked memory (written in
    place, the old y prefetched on a second stream) and in pageable memory
    (staged), on a 16-byte-aligned y and on one 8 bytes further, accumulating
    and not."""
    import qcm_oracle as qo
    import models
    import torch
    from pyqcm_gb300 import _lib
    H = _hubbard(13, 1, 6, 6)
    assert H.dim >= 2**21
    ns, _, ops = models.hubbard_cluster(13, 1)
    up, dn, pr = qo.combine_terms({k: v for k, v in ops.items() if k in PARAMS}, PARAMS, ns)
    x = qo.seeded_start(H.dim, 7)
    ref = qo.Sector(ns, 6, 6, up, dn, pr).matvec(x, nthreads=8)
    # the fixed-point format's bound: 1e-13 of the largest component, of H x and y
    tol = 1e-13 * (np.max(np.abs(ref)) + 3.0)
    y = torch.empty(H.dim + 1, dtype=torch.float64, pin_memory=pinned).numpy()[offset:offset + H.dim]
    for _ in range(2):
        y[:] = 0.75
        H.mult_add(x, y)
        assert np.max(np.abs(y - 0.75 - ref)) <= tol
        y[:] = 3.0
        _lib.check(_lib.lib().qcmg_matvec(H._h, _lib.ptr(x), _lib.ptr(y), 0))
        assert np.max(np.abs(y - ref)) <= tol
    xd, yd = torch.from_numpy(x).cuda(), torch.full((H.dim,), 0.75, dtype=torch.float64, device="cuda")
    H.matvec_device(xd.data_ptr(), yd.data_ptr(), accumulate=True)
    assert np.max(np.abs(yd.cpu().numpy() - 0.75 - ref)) <= tol


@pytest.mark.parametrize("scale", [1e8, 3e10])
@pytest.mark.parametrize("nup,ndn", [(0, 1), (1, 1), (2, 1)])
def test_small_sectors_beyond_fp64(scale, nup, ndn):
    """A dimer with energies of 1e8 to 3e10 at a tolerance of 1e-12, below the
    rounding of an FP64 step: the on-chip run does not meet it, the fixed-point
    run that then decides does (its exact sums end the Krylov space); on the
    FP64 path the run ends with NOCONV."""
    import pyqcm_gb300 as pg
    m = pg.ClusterModel(2)
    m.new_operator("t", "one-body", [(0, 1, -1.0), (2, 3, -1.0)])
    m.new_operator("U", "interaction", [(0, 2, 1.0), (1, 3, 1.0)])
    m.new_operator("e", "one-body", [(0, 0, 1.0), (2, 2, 1.0)])
    H = pg.Hamiltonian(m, {"t": 0.921 * scale, "U": 3.0 * scale, "e": 0.37 * scale}, f"R0:N{nup + ndn}:S{nup - ndn}")
    assert H.fx_available()
    A = np.array([H.matvec(v) for v in np.eye(H.dim)])
    x0 = np.random.default_rng(5).normal(size=H.dim)
    x0 /= np.linalg.norm(x0)
    e0, psi, _, _ = H.lanczos(x0=x0, tol=1e-12, max_iter=300, reorth=0)
    e = np.linalg.eigvalsh(A)
    assert abs(e0 - e[0]) < 1e-13 * np.max(np.abs(e))
    assert np.linalg.norm(A @ psi - e0 * psi) < 1e-13 * np.max(np.abs(e))
