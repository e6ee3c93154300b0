"""The lattice point kernels against numpy at the sizes where they can go
wrong: matrix dimensions at the ends of the register kernels' range and past
it, ragged wavevector counts, grids whose points pair up as (K, -K) in every
way (odd and even axes), and elements that do not pair (complex or one-sided)
and so take every point."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# The largest condition number of these matrices is ~1e3 and a point does
# O(L^2) roundings per result: L^2 eps kappa = 256 x 2.2e-16 x 1e3 = 6e-11.
TOL = 1e-10


class Problem:
    def __init__(self, L, kind, seed, nb=2, M=40):
        rng = np.random.default_rng([seed, L])
        self.L = L
        self.R = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [1, -1, 0], [-1, 1, 0]], float)
        minus = [0, 2, 1, 4, 3, 6, 5]
        self.els = []
        for _ in range(2 * L):
            r, c, n = rng.integers(L), rng.integers(L), rng.integers(1, 7)
            v = rng.normal() + (1j * rng.normal() if kind == "complex" else 0.0)
            self.els.append((r, c, n, v))
            if kind != "onesided":
                self.els.append((c, r, minus[n], np.conj(v)))
        h = rng.normal(size=(L, L))
        self.hdiff = (h + h.T) * 0.3 + 0j
        self.gpos = rng.uniform(0, 1, (L, 3))
        Q, _ = np.linalg.qr(rng.normal(size=(M + L, M + L)) + (1j * rng.normal(size=(M + L, M + L)) if kind == "complex" else 0.0))
        self.v = np.ascontiguousarray(Q[:L])
        self.e = rng.uniform(-5, 5, M + L)
        self.tcb, self.eb = rng.normal(size=(L, nb)) * 0.3 + 0j, rng.uniform(-2, 2, nb)

    def block(self):
        from pyqcm_gb300.lattice import _LatticeBlock

        class Model:
            cluster = type("C", (), {"n_sites": self.L})
            fourier = staticmethod(lambda sd: (self.R, self.els, self.hdiff, self.gpos))
        blk = _LatticeBlock(Model, False)
        blk.set_green(self.e, self.v, self.tcb, np.diag(self.eb))
        return blk

    def matrices(self, z, K):
        """M = G^-1 + Gamma - hdiff - V(K), G: (nz, nK, L, L), (nz, L, L)."""
        G = np.einsum("ai,zi,bi->zba", self.v, 1.0 / (z[:, None] - self.e), self.v.conj())
        gam = np.einsum("ik,zk,jk->zij", self.tcb, 1.0 / (z[:, None] - self.eb), self.tcb.conj())
        V = np.zeros((len(K), self.L, self.L), complex)
        for r, c, n, v in self.els:
            V[:, r, c] += v * np.exp(2j * np.pi * (K @ self.R[n]))
        return (np.linalg.inv(G) + gam - self.hdiff)[:, None] - V[None], G


def grid(gx, gy, gz, off=0.0):
    ax = [(np.arange(g) + off) / g if (g > 1 or a == 0) else np.zeros(1) for a, g in enumerate((gx, gy, gz))]
    l, j, i = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return np.stack([i.ravel(), j.ravel(), l.ravel()], 1)


@pytest.mark.parametrize("L", [1, 2, 3, 7, 12, 15, 16, 17])
@pytest.mark.parametrize("kind", ["real", "complex", "onesided"])
@pytest.mark.parametrize("g", [(1, 1, 1), (7, 5, 1), (8, 6, 2), (33, 1, 1)])
def test_functional_points(L, kind, g):
    from pyqcm_gb300 import _lib
    p = Problem(L, kind, 1)
    w, wt = np.array([0.4, 1.7, 30.0, 4e3]), np.array([0.3, 0.5, 0.2, 0.1])
    blk = p.block()
    out = _lib.c_double()
    _lib.check(_lib.lib().qcmg_sef_grid(blk._h, len(w), _lib.ptr(w), _lib.ptr(wt), *g, out))
    A, G = p.matrices(1j * w, grid(*g))
    ref = np.sum(wt[:, None] * (np.linalg.slogdet(A)[1] + np.linalg.slogdet(G)[1][:, None])) / A.shape[1]
    assert abs(out.value - ref) < TOL * L


@pytest.mark.parametrize("L", [1, 2, 3, 7, 12, 15, 16, 17])
@pytest.mark.parametrize("kind", ["real", "complex", "onesided"])
@pytest.mark.parametrize("nk", [1, 31, 32, 33, 70])
def test_periodized_points(L, kind, nk):
    from pyqcm_gb300 import _lib
    p = Problem(L, kind, 2)
    z = np.array([0.3 + 0.3j, -1.2 + 0.5j, 2.0j])
    K = np.ascontiguousarray(np.random.default_rng(5).uniform(-1, 1, (nk, 3)))
    blk = p.block()
    g = np.zeros(2 * len(z) * nk)
    _lib.check(_lib.lib().qcmg_cpt_periodized(blk._h, len(z), _lib.ptr(z.view(np.float64)), nk, _lib.ptr(K), _lib.ptr(g)))
    A, _ = p.matrices(z, K)
    u = np.exp(2j * np.pi * (K @ p.gpos.T))
    ref = np.einsum("ka,zkab,kb->zk", u.conj(), np.linalg.inv(A), u) / L
    assert np.max(np.abs(g.view(np.complex128).reshape(len(z), nk) - ref)) < TOL * max(1.0, np.max(np.abs(ref)))


@pytest.mark.parametrize("L", [1, 2, 4, 7, 8, 13, 16, 17])
@pytest.mark.parametrize("kind", ["real", "complex", "onesided"])
@pytest.mark.parametrize("g", [(1, 1, 1, 0.0), (7, 5, 1, 0.0), (8, 6, 2, 0.5), (33, 1, 1, 0.5), (40, 3, 1, 0.25)])
@pytest.mark.parametrize("moments", ["none", "few", "many"])
def test_inverse_means(L, kind, g, moments):
    """Plain means and means with translations' phases: few translations, and
    16 with more distinct x components than one pass takes."""
    from pyqcm_gb300 import _lib
    p = Problem(L, kind, 3)
    z = np.array([0.3 + 0.3j, -1.2 + 0.5j, 2.0j])
    R = {"none": np.zeros((0, 3)), "few": p.R.copy(),
         "many": np.array([[(-1) ** m * m, m % 3 - 1, m % 2] for m in range(16)], float)}[moments]
    if moments == "few" and g[0] == 33:
        R[3] = [0.5, 0.0, 0.0]  # not a lattice translation: no pairing
    blk = p.block()
    nm = max(1, len(R))
    out = np.zeros(2 * len(z) * nm * L * L)
    if len(R):
        _lib.check(_lib.lib().qcmg_lattice_kmoments(blk._h, len(z), _lib.ptr(z.view(np.float64)), *g[:3], g[3], nm,
                                                    _lib.ptr(np.ascontiguousarray(R)), _lib.ptr(out)))
    else:
        _lib.check(_lib.lib().qcmg_lattice_kmean(blk._h, len(z), _lib.ptr(z.view(np.float64)), *g[:3], g[3], _lib.ptr(out)))
    K = grid(*g)
    A, _ = p.matrices(z, K)
    X = np.linalg.inv(A)
    ph = np.exp(2j * np.pi * (K @ R.T)) if len(R) else np.ones((len(K), 1))
    ref = np.einsum("km,zkab->zmab", ph, X) / len(K)
    got = out.view(np.complex128).reshape(len(z), nm, L, L)
    assert np.max(np.abs(got - ref)) < TOL * max(1.0, np.max(np.abs(X)))


@pytest.mark.parametrize("L", [1, 2, 5, 12, 32])
@pytest.mark.parametrize("M", [1, 31, 32, 33, 500])
@pytest.mark.parametrize("nz", [1, 3, 4, 37])
@pytest.mark.parametrize("real", [True, False])
def test_green_function_sums(L, M, nz, real):
    """G(z) at the tile edges of the pole sum, real (symmetric) and complex."""
    import pyqcm_gb300 as pg
    rng = np.random.default_rng([L, M, nz])
    v = rng.normal(size=(L, M)) + (0 if real else 1j * rng.normal(size=(L, M)))
    e, z = rng.normal(size=M), rng.normal(size=nz) + 1j * rng.uniform(0.2, 1, nz)
    ref = np.einsum("ai,zi,bi->zba", v, 1.0 / (z[:, None] - e), v.conj())
    # M products of size |v|^2 / Im z, each with a few roundings
    bound = 8 * np.finfo(float).eps * M * np.max(np.abs(v)) ** 2 / np.min(z.imag)
    assert np.max(np.abs(pg.green_function(e, v, z) - ref)) < bound
