"""The fixed-point product on its own vectors (qcmg_matvec_fx) over the forms
of its passes, on sectors whose FP64-vector products take the FP64 kernel:
slabs staged by threads (du < 64), two small slabs per block (du <= 1006), two
large slabs, one per block; even and odd half bases, unequal spins; narrow
(integer) and wide diagonals; bands of pass D down to one sweep."""
import numpy as np
import pytest

import qcm_oracle as qo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mu", [4.0, 3.7])
@pytest.mark.parametrize("slabs", ["1", "2", ""])
@pytest.mark.parametrize("shape,nup,ndn", [((5, 1), 2, 3), ((7, 1), 3, 4), ((8, 1), 4, 4), ((3, 3), 4, 5), ((11, 1), 2, 5),
                                           ((4, 3), 6, 6), ((13, 1), 5, 5), ((12, 1), 2, 1)])
def test_fixed_point_product(monkeypatch, shape, nup, ndn, slabs, mu):
    import models
    import pyqcm_gb300 as pg
    import torch
    if slabs:
        monkeypatch.setenv("QCMG_FX_SLABS", slabs)
    ns, nb, ops = models.hubbard_cluster(*shape)
    params = {"t": 1.0, "U": 8.0, "mu": mu}
    ops = {k: v for k, v in ops.items() if k in params}
    m = pg.ClusterModel(ns, nb)
    for name, (typ, els) in ops.items():
        m.new_operator(name, typ, els)
    H = pg.Hamiltonian(m, params, f"R0:N{nup + ndn}:S{nup - ndn}")
    assert H.fx_available()
    up, dn, pr = qo.combine_terms(ops, params, ns)
    S = qo.Sector(ns, nup, ndn, up, dn, pr)
    x = qo.seeded_start(H.dim, 5)
    ref = S.matvec(x, nthreads=8)
    xd = torch.from_numpy(x).cuda()
    qx, qy = torch.empty(H.dim, dtype=torch.int64, device="cuda"), torch.empty(H.dim, dtype=torch.int64, device="cuda")
    y = torch.empty(H.dim, dtype=torch.float64, device="cuda")
    E, mb = pg._lib.c_int(), pg._lib.c_int()
    pg._lib.check(pg.lib().qcmg_fx_from_f64(H.dim, xd.data_ptr(), qx.data_ptr(), E, mb, None))
    for acc in (False, True):
        qy.copy_(qx)
        torch.cuda.synchronize()
        Ey = H.matvec_fx_device(qx.data_ptr(), E.value, mb.value, qy.data_ptr(), Ey_in=E.value if acc else None)
        pg._lib.check(pg.lib().qcmg_fx_to_f64(H.dim, qy.data_ptr(), Ey, y.data_ptr(), None))
        want = ref + x if acc else ref
        # the fixed-point format's bound: 1e-13 of the largest component
        assert np.max(np.abs(y.cpu().numpy() - want)) <= 1e-13 * np.max(np.abs(want))


@pytest.mark.parametrize("n", [(1, 1), (4, 4), (5, 5)])
def test_small_host_products_are_staged(n):
    """mult_add and matvec on host vectors below and above the staging limit,
    from unaligned and read-only arrays, with y elsewhere in memory."""
    import models
    import pyqcm_gb300 as pg
    ns, nb, ops = models.hubbard_cluster(10, 1)
    params = {"t": 1.0, "U": 8.0, "mu": 4.0}
    ops = {k: v for k, v in ops.items() if k in params}
    m = pg.ClusterModel(ns, nb)
    for name, (typ, els) in ops.items():
        m.new_operator(name, typ, els)
    H = pg.Hamiltonian(m, params, f"R0:N{sum(n)}:S0")
    up, dn, pr = qo.combine_terms(ops, params, ns)
    S = qo.Sector(ns, *n, up, dn, pr)
    rng = np.random.default_rng(1)
    x = rng.normal(size=H.dim + 1)[1:]
    x.flags.writeable = False
    ref = S.matvec(np.array(x))
    for _ in range(3):
        y0 = rng.normal(size=H.dim)
        y = y0.copy()
        H.mult_add(x, y)
        assert np.max(np.abs(y - y0 - ref)) <= 1e-13 * np.max(np.abs(ref))
        assert np.max(np.abs(H.matvec(x) - ref)) <= 1e-13 * np.max(np.abs(ref))


@pytest.mark.parametrize("shape,nup,ndn", [((10, 1), 5, 5), ((15, 1), 3, 2)])
@pytest.mark.parametrize("mu", [1.0, 4.0, 1e3, 1e6, -1e6])
def test_fixed_point_lanczos_with_a_shifted_diagonal(shape, nup, ndn, mu):
    """The update's usual shifts and, as a large multiple of the identity makes
    alpha outweigh beta, its general form; an even and an odd number of states."""
    import models
    import pyqcm_gb300 as pg
    ns, nb, ops = models.hubbard_cluster(*shape)
    E = []
    for value in (0.0, mu):
        params = {"t": 1.0, "U": 8.0, "mu": value}
        m = pg.ClusterModel(ns, nb)
        for name, (typ, els) in ops.items():
            if name in params:
                m.new_operator(name, typ, els)
        H = pg.Hamiltonian(m, params, f"R0:N{nup + ndn}:S{nup - ndn}")
        assert H.dim > 16384 and H.fx_available()
        E.append(H.lanczos(tol=1e-5, want_psi=False)[0])
    shift = mu * (nup + ndn)
    # each run: the residual squared over the gap (> 1e-2); and the format's
    # rounding of |H| times the ~100 steps
    bound = 2e-8 + 100 * 2.0 ** -53 * abs(shift)
    assert abs(E[0] - shift - E[1]) < bound
