"""Lattice integrals on grids of unusual shape: one long row, rows shorter
than a warp, cubes (the means with translations' phases take one of two ways
by the rows' length), and more points than one launch holds."""
import numpy as np
import pytest

from test_gpu_lattice_points import TOL, Problem, grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [2, 8, 12, 16])
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("g", [(1024, 1, 1, 0.0), (997, 1, 1, 0.25), (1, 70, 1, 0.5), (2, 65, 1, 0.0), (8, 8, 8, 0.5),
                               (16, 5, 3, 0.0), (100, 9, 1, 0.5)])
def test_means_with_phases(L, kind, g):
    from pyqcm_gb300 import _lib
    p = Problem(L, kind, 4)
    z = np.array([0.3 + 0.3j, 2.0j])
    blk = p.block()
    out = np.zeros(2 * len(z) * len(p.R) * L * L)
    _lib.check(_lib.lib().qcmg_lattice_kmoments(blk._h, len(z), _lib.ptr(z.view(np.float64)), *g[:3], g[3], len(p.R),
                                                _lib.ptr(np.ascontiguousarray(p.R)), _lib.ptr(out)))
    K = grid(*g)
    X = np.linalg.inv(p.matrices(z, K)[0])
    ref = np.einsum("km,zkab->zmab", np.exp(2j * np.pi * (K @ p.R.T)), X) / len(K)
    got = out.view(np.complex128).reshape(ref.shape)
    assert np.max(np.abs(got - ref)) < TOL * max(1.0, np.max(np.abs(X)))


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
