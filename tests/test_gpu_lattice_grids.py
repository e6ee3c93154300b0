"""Lattice integrals on grids of unusual size: more points than one launch
holds."""
import numpy as np
import pytest

from test_gpu_lattice_points import TOL, Problem, grid

pytestmark = pytest.mark.gpu


class OneWay(Problem):
    """One site with one hop v along x: V(K) = v e^{2 pi i K.R}."""

    def __init__(self):
        super().__init__(1, "onesided", 5)
        self.els = [(0, 0, 1, 0.25 + 0.0j)]


@pytest.mark.parametrize("nk,nw", [(64, 3), (2048, 300), (4096, 4100)])
def test_functional_of_many_points(nk, nw):
    """Up to 6.9e10 points (more warps than a grid has blocks). The K mean of
    log|a - v e^{i x}| is log max(|a|, |v|), to (|v| / |a|)^nk."""
    from pyqcm_gb300 import _lib
    p = OneWay()
    w, wt = np.linspace(0.5, 40.0, nw), np.full(nw, 1.0 / nw)
    A, G = p.matrices(1j * w, np.zeros((1, 3)))
    a, v = np.abs(A[:, 0, 0, 0] + 0.25), 0.25
    assert np.min(np.maximum(a, v) / np.minimum(a, v)) > 1.5  # 1.5^-64 < 1e-11
    out = _lib.c_double()
    blk = p.block()
    _lib.check(_lib.lib().qcmg_sef_grid(blk._h, nw, _lib.ptr(w), _lib.ptr(wt), nk, nk, 1, out))
    assert abs(out.value - np.sum(wt * (np.log(np.maximum(a, v)) + np.log(np.abs(G[:, 0, 0]))))) < TOL
