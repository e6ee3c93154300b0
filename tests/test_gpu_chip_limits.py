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
