"""Performance cases of the exact-diagonalization and lattice-integral paths.

A case names a path ("kind") and its sizes.  The kinds follow the stages of a
cluster calculation:

  product    y += H x on the device's fixed-point vectors (the product inside Lanczos)
  product64  y += H x on FP64 device vectors, two hop magnitudes (t and t')
  mult_add   y += H x on host vectors (the call a host program's solver makes)
  ground     Lanczos ground state and its vector, optionally fully reorthogonalized
  batch      ground states of many impurity sectors in one call
  green      band Lanczos of the hole sector and its G(iw) (VCA cluster solve)
  impurity   one impurity problem from its parameters to G(iw) (a CDMFT step)
  sef        Potthoff functional on a (k, w) grid, from a saved impurity solution
  cpt        periodized Green function g(k, w) on the real axis
  host       CDMFT host function on a k grid
  averages   lattice averages of the one-body operators on a (k, w) grid

Clusters are nx x ny Hubbard clusters with open boundaries.  The lattice stages
read their cluster Green function from a file, as after an impurity stage that
was saved; its poles come from a seeded auxiliary one-body problem with a bath
and a self-energy, so the sum rule and the signs of a real solution hold.
`exact` restates each path in 64 bits with plain torch and numpy.
"""
import itertools
import math
import os
import tempfile

import numpy as np
import torch

import pyqcm_gb300 as pg
from pyqcm_gb300 import cdmft, ed
from pyqcm_gb300 import lattice as lat

BETA = 50.0  # inverse temperature of the Matsubara grids


def listed():
    return [
        # the 4x4 cluster at half filling: the largest sector that fits, one Lanczos product
        {"name": "product_4x4_half", "kind": "product", "nx": 4, "ny": 4, "nup": 8, "ndn": 8},
        # the 3x4 cluster with diagonal hopping: the product of a VCA cluster solve
        {"name": "product64_3x4_tp", "kind": "product64", "nx": 4, "ny": 3, "nup": 6, "ndn": 6},
        # the 8-site chain through the host call: latency, copies and launches
        {"name": "mult_add_chain8", "kind": "mult_add", "nx": 8, "ny": 1, "nup": 4, "ndn": 4, "tp": False},
        # ground state of the 3x4 cluster with its vector, the reference's recurrence
        {"name": "ground_3x4", "kind": "ground", "nx": 4, "ny": 3, "nup": 6, "ndn": 6, "reorth": 0},
        # ground state of a dilute 4x4 sector with every Krylov vector kept and projected out
        {"name": "ground_4x4_n8_reorth", "kind": "ground", "nx": 4, "ny": 4, "nup": 4, "ndn": 4, "reorth": 100},
        # 16 plaquette + 4 bath impurities in three sectors each: one lockstep CDMFT iteration
        {"name": "batch_2x2_b4", "kind": "batch", "instances": 16},
        # hole part of the VCA cluster's Green function: 731,808 states, 12 start vectors
        {"name": "green_3x4_tp", "kind": "green", "nx": 4, "ny": 3, "nup": 6, "ndn": 6, "nw": 64},
        # a 2x2 + 4 bath impurity from its parameters to G on 200 Matsubara frequencies
        {"name": "impurity_2x2_b4", "kind": "impurity", "nw": 200},
        # the VCA functional: 128x128 k x 256 frequencies x 2 spins, 12 x 12 blocks
        {"name": "sef_3x4", "kind": "sef", "nx": 4, "ny": 3, "nk": 128, "nw": 256, "poles": 1100},
        # the spectral map of the 8-site chain: 256 k x 512 real frequencies
        {"name": "cpt_chain8", "kind": "cpt", "nx": 8, "nk": 256, "nw": 512, "poles": 260},
        # the CDMFT host function of the plaquette with 8 baths: 64x64 k x 200 frequencies
        {"name": "host_2x2_b8", "kind": "host", "nbath": 8, "nk": 64, "nw": 200, "poles": 480},
        # averages of t, the Neel field and mu on the 2x4 cluster, both spins
        {"name": "averages_2x4", "kind": "averages", "nx": 4, "ny": 2, "nk": 64, "nw": 64, "poles": 500},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def filling(n):  # from a few electrons to half filling, the spins not always equal
        nup = rng.randint(max(1, n // 4), (n + 1) // 2)
        return nup, max(1, min(n // 2, nup + rng.choice((-1, 0, 0, 1))))

    def cluster(choices):
        nx, ny = rng.choice(choices)
        return nx, ny, *filling(nx * ny)

    kind = rng.choice(("product", "product64", "mult_add", "ground", "batch", "green", "impurity",
                       "sef", "cpt", "host", "averages"))
    if kind in ("product", "product64", "mult_add", "ground", "green"):
        small = [(7, 1), (8, 1), (3, 3), (4, 2), (5, 2), (11, 1), (4, 3)]
        choices = {"product": small + [(13, 1), (7, 2), (5, 3), (4, 4)],
                   "product64": [(3, 3), (4, 2), (5, 2), (4, 3), (7, 2)],
                   "mult_add": small, "ground": small + [(13, 1)],
                   "green": [(3, 3), (4, 2), (5, 2), (4, 3)]}[kind]
        nx, ny, nup, ndn = cluster(choices)
        case = {"kind": kind, "nx": nx, "ny": ny, "nup": nup, "ndn": ndn}
        if kind == "mult_add":
            case["tp"] = ny > 1 and rng.random() < 0.5
        if kind == "ground":
            case["reorth"] = rng.choice((0, 0, log(40, 120)))
        if kind == "green":
            case["nw"] = log(8, 256)
        return case
    if kind == "batch":
        return {"kind": kind, "instances": log(2, 16)}
    if kind == "impurity":
        return {"kind": kind, "nw": log(20, 400)}
    if kind == "sef":
        nx, ny = rng.choice(((2, 1), (2, 2), (3, 2), (4, 2), (5, 2), (4, 3)))
        return {"kind": kind, "nx": nx, "ny": ny, "nk": log(9, 128), "nw": log(16, 256), "poles": log(100, 1100)}
    if kind == "cpt":
        return {"kind": kind, "nx": rng.choice((2, 4, 5, 6, 8, 10, 12)), "nk": log(33, 400), "nw": log(50, 800),
                "poles": log(60, 600)}
    if kind == "host":
        return {"kind": kind, "nbath": rng.choice((0, 4, 8)), "nk": log(8, 64), "nw": log(30, 300),
                "poles": log(60, 700)}
    nx, ny = rng.choice(((2, 2), (3, 2), (4, 2)))
    return {"kind": kind, "nx": nx, "ny": ny, "nk": log(8, 64), "nw": log(14, 64), "poles": log(60, 500)}


# ---------------------------------------------------------------------------
# models


def _bonds(nx, ny):
    """Nearest-neighbour and diagonal bonds of the open nx x ny cluster, x fastest."""
    at = lambda x, y: x + nx * y
    near = [(at(x, y), at(x + 1, y)) for y in range(ny) for x in range(nx - 1)]
    near += [(at(x, y), at(x, y + 1)) for y in range(ny - 1) for x in range(nx)]
    diag = [(at(x, y), at(x + d, y + 1)) for y in range(ny - 1) for x in range(nx) for d in (-1, 1)
            if 0 <= x + d < nx]
    return near, diag


def _neel(nx, ny):
    return [1.0 if (x + y) % 2 == 0 else -1.0 for y in range(ny) for x in range(nx)]


def _cluster_model(nx, ny):
    n = nx * ny
    near, diag = _bonds(nx, ny)
    both = lambda els: els + [(i + n, j + n, v) for i, j, v in els]
    m = pg.ClusterModel(n)
    m.new_operator("t", "one-body", both([(i, j, -1.0) for i, j in near]))
    if diag:
        m.new_operator("tp", "one-body", both([(i, j, -1.0) for i, j in diag]))
    m.new_operator("U", "interaction", [(i, i + n, 1.0) for i in range(n)])
    m.new_operator("mu", "one-body", both([(i, i, -1.0) for i in range(n)]))
    m.new_operator("M", "one-body", [(i, i, s) for i, s in enumerate(_neel(nx, ny))]
                   + [(i + n, i + n, -s) for i, s in enumerate(_neel(nx, ny))])
    return m


def _sector(nup, ndn):
    return f"R0:N{nup + ndn}:S{nup - ndn}"


HUBBARD = {"t": 1.0, "U": 8.0, "mu": 4.0}


def _vca_values(seed):
    """t' = -0.3 and a Weiss field of the scan's range."""
    return dict(HUBBARD, tp=-0.3, M=float(np.random.default_rng([seed, 1]).uniform(0.05, 0.2)))


def _impurity_values(rng, nbath):
    U = rng.uniform(4, 12)
    v = {"t": 1.0, "U": U, "mu": U * rng.uniform(0.4, 0.5)}
    for k in range(nbath):
        v[f"eb{k + 1}"] = (1 if k % 2 else -1) * rng.uniform(0.3, 2.0)
        v[f"tb{k + 1}"] = rng.uniform(0.2, 0.8)
    return {k: float(x) for k, x in v.items()}


def _matsubara(n):
    return (2 * np.arange(n) + 1) * np.pi / BETA


def _lattice_grid(nw):
    """Gauss-Legendre frequencies and weights of the fixed-grid integrals."""
    return lat.legendre_frequency_grid(1.0, 10.0, nw - 2 * (nw // 3), nw // 3, nw // 3)


# geometry of the lattice cases: sites, superlattice vectors
def _lattice(case):
    if case["kind"] == "cpt":
        return [(i, 0, 0) for i in range(case["nx"])], [(case["nx"], 0, 0)]
    nx, ny = (2, 2) if case["kind"] == "host" else (case["nx"], case["ny"])
    # an odd height shifts the next row by one, so the Neel wavevector stays commensurate
    return [(x, y, 0) for y in range(ny) for x in range(nx)], [(nx, 0, 0), (ny % 2, ny, 0)]


def _lattice_params(case, seed):
    """(lattice values, cluster values) of the one-body operators and U."""
    rng = np.random.default_rng([seed, 2])
    U = 4.0 if case["kind"] == "cpt" else 8.0
    lv = {"t": 1.0, "U": U, "mu": U / 2}
    if case["kind"] in ("sef", "averages"):
        lv.update({"tp": -0.3, "M": 0.0})
    cv = dict(lv)
    if case["kind"] in ("sef", "averages"):
        cv["M"] = float(rng.uniform(0.05, 0.2))
    if case["kind"] == "host":
        cv.update({k: v for k, v in _impurity_values(rng, case["nbath"]).items() if k[:2] in ("eb", "tb")})
    return lv, cv


LINKS = {"t": [(1, 0, 0), (0, 1, 0)], "tp": [(1, 1, 0), (-1, 1, 0)]}


def _links(case, name):
    return [k for k in LINKS[name] if case["kind"] != "cpt" or k[1] == 0]


def _spins(case):
    return (False, True) if case["kind"] in ("sef", "averages") else (False,)


def _bath(case, cv):
    """(couplings L x nb, energies nb) of the host case's bath."""
    nb = case.get("nbath", 0)
    L = len(_lattice(case)[0])
    tcb = np.zeros((L, nb))
    for k in range(nb):
        tcb[k % L, k] = cv[f"tb{k + 1}"]
    return tcb, np.array([cv[f"eb{k + 1}"] for k in range(nb)])


def _cluster_matrix(case, cv, down):
    """One-body matrix of the cluster sites (hopping, mu and the Neel field)."""
    sites, _ = _lattice(case)
    idx = {s: i for i, s in enumerate(sites)}
    T = np.zeros((len(sites), len(sites)))
    for name in LINKS:
        for d in (_links(case, name) if name in cv else ()):
            for i, s in enumerate(sites):
                j = idx.get(tuple(a + b for a, b in zip(s, d)))
                if j is not None:
                    T[i, j] -= cv[name]
                    T[j, i] -= cv[name]
    for i, s in enumerate(sites):
        T[i, i] += -cv["mu"] + cv.get("M", 0.0) * (1 if (s[0] + s[1]) % 2 == 0 else -1) * (-1 if down else 1)
    return T


def _lehmann(case, seed, down):
    """Poles e (M) and residues v (L, M) of a cluster Green function: the
    cluster, its bath and seeded self-energy poles as one Hermitian matrix."""
    _, cv = _lattice_params(case, seed)
    rng = np.random.default_rng([seed, 3, int(down)])
    tcb, eb = _bath(case, cv)
    L, nb = tcb.shape
    n = max(case["poles"], L + nb + 2)
    A = np.zeros((n, n))
    A[:L, :L] = _cluster_matrix(case, cv, down) + cv["U"] / 2 * np.eye(L)
    A[:L, L:L + nb] = tcb
    A[L:L + nb, :L] = tcb.T
    A[range(L, L + nb), range(L, L + nb)] = eb
    na = n - L - nb
    g = rng.normal(size=(L, na)) * cv["U"] / 2 / math.sqrt(na)
    A[:L, L + nb:] = g
    A[L + nb:, :L] = g.T
    A[range(L + nb, n), range(L + nb, n)] = rng.choice((-1.0, 1.0), na) * rng.uniform(0.5, cv["U"], na)
    e, W = np.linalg.eigh(A)
    return e, np.ascontiguousarray(W[:L])


def _saved_solution(cluster, case, seed):
    """Hands the instance the saved impurity stage."""
    names = sorted(cluster.values)
    d = {"value_names": np.array(names), "values": np.array([cluster.values[n] for n in names]),
         "mixing": 4 if len(_spins(case)) > 1 else 0, "GS_energy": -10.0, "E0": -10.0, "n_states": 1,
         "s0_sector": np.array(cluster.target_sectors[0].name()), "s0_energy": -10.0, "s0_weight": 1.0}
    for down in _spins(case):
        e, v = _lehmann(case, seed, down)
        tag = "s0_down" if down else "s0_up"
        d.update({f"{tag}_L": v.shape[0], f"{tag}_M": len(e), f"{tag}_e": e, f"{tag}_v": v.astype(np.complex128)})
    with tempfile.TemporaryDirectory() as folder:
        path = os.path.join(folder, "solution.npz")
        np.savez(path, **d)
        cluster.read_qmatrix(path)


def _lattice_instance(case, seed):
    sites, sup = _lattice(case)
    lv, cv = _lattice_params(case, seed)
    n, nb = len(sites), case.get("nbath", 0)
    if case["kind"] == "host":
        lm = cdmft.plaquette_bath_model(nb, _sector((n + nb) // 2, (n + nb) // 2))
        lm.set_parameters({**{k: v for k, v in lv.items()}, "tp": 0.0,
                           **{k + "_1": v for k, v in cv.items() if k[:2] in ("eb", "tb")}})
    else:
        lm = lat.LatticeModel(pg.ClusterModel(n), sites, [s[:2] for s in sup] if len(sup) > 1 else sup)
        lm.interaction_operator("U", 1.0)
        for name in ("t", "tp"):
            for d in (_links(case, name) if name in lv else ()):
                lm.hopping_operator(name, d, -1.0)
        if "M" in lv:
            lm.density_wave("M", "Z", (1, 1, 0), 1.0, 0.0)
        lm.set_target_sectors(_sector((n + 1) // 2, n // 2))
        lm.set_parameters({**lv, **({"M_1": cv["M"]} if "M" in cv else {})})
    inst = lm.instance()
    _saved_solution(inst.cluster, case, seed)
    return inst


# ---------------------------------------------------------------------------
# preparation and the passes


def _unit(n, seed):
    x = np.random.default_rng([seed, 4]).standard_normal(n)
    return x / np.linalg.norm(x)


def _device_unit(n, seed):
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
    return x / torch.linalg.vector_norm(x)


def _batch_problems(case, seed):
    """(sector, values) of every impurity sector of the batch."""
    rng = np.random.default_rng([seed, 5])
    for _ in range(case["instances"]):
        values = _impurity_values(rng, 4)
        for sector in ("R0:N7:S1", "R0:N8:S0", "R0:N9:S1"):
            yield sector, values


def _plaquette_cluster(nbath):
    lm = cdmft.plaquette_bath_model(nbath, _sector((4 + nbath) // 2, (4 + nbath) // 2))
    lm.finalize()
    return lm.cluster


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("product", "product64", "mult_add", "ground"):
        tp = kind == "product64" or case.get("tp", False)
        H = pg.Hamiltonian(_cluster_model(case["nx"], case["ny"]), _vca_values(seed) if tp else HUBBARD,
                           _sector(case["nup"], case["ndn"]))
        s["H"] = H
        H.fx_available()  # the product's tables, built once per sector
        if kind == "product":
            x = _device_unit(H.dim, seed)
            E, mb = pg._lib.c_int(), pg._lib.c_int()
            s["x"] = torch.empty(H.dim, dtype=torch.int64, device="cuda")
            pg._lib.check(pg.lib().qcmg_fx_from_f64(H.dim, x.data_ptr(), s["x"].data_ptr(), E, mb, None))
            s["y"] = s["x"].clone()
            s["E"], s["mb"] = E.value, mb.value
        elif kind == "product64":
            s["x"] = _device_unit(H.dim, seed)
            s["y"] = _device_unit(H.dim, seed + 1000003)
        else:
            s["x"] = _unit(H.dim, seed)
            s["y"] = _unit(H.dim, seed + 1000003)
    elif kind == "batch":
        cm = _plaquette_cluster(4)
        s["H"] = [pg.Hamiltonian(cm, values, sector) for sector, values in _batch_problems(case, seed)]
        for H in s["H"]:
            H.set_path(False)
    elif kind == "green":
        n = case["nx"] * case["ny"]
        m, values = _cluster_model(case["nx"], case["ny"]), _vca_values(seed)
        H = pg.Hamiltonian(m, values, _sector(case["nup"], case["ndn"]))
        E0, psi, _, _ = H.lanczos(x0=_unit(H.dim, seed))
        s["E0"], s["z"] = E0, 1j * _matsubara(case["nw"])
        s["phi"] = ed.apply_c_device(n, list(range(n)), -1, case["nup"], case["ndn"], torch.from_numpy(psi).cuda())
        s["H"] = pg.Hamiltonian(m, values, _sector(case["nup"] - 1, case["ndn"]))
    elif kind == "impurity":
        s["cm"], s["values"] = _plaquette_cluster(4), _impurity_values(np.random.default_rng([seed, 6]), 4)
        s["z"] = 1j * _matsubara(case["nw"])
    else:
        s["inst"] = _lattice_instance(case, seed)
        if kind in ("sef", "averages"):
            s["w"], s["wt"] = _lattice_grid(case["nw"])
        elif kind == "cpt":
            s["z"] = np.linspace(-8.0, 8.0, case["nw"]) + 0.1j
            s["k"] = np.arange(case["nk"])[:, None] / case["nk"] * np.array([[1.0, 0.0, 0.0]])
        else:
            s["w"], s["wt"] = _matsubara(case["nw"]), np.ones(case["nw"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "product":
        # y's mantissas are taken at x's exponent on every pass, so that passes repeat
        E = s["H"].matvec_fx_device(s["x"].data_ptr(), s["E"], s["mb"], s["y"].data_ptr(), asynchronous=True,
                                    Ey_in=s["E"])
        return s["y"], E
    if kind == "product64":
        s["H"].matvec_device(s["x"].data_ptr(), s["y"].data_ptr(), accumulate=True, asynchronous=True)
        return s["y"]
    if kind == "mult_add":
        s["H"].mult_add(s["x"], s["y"])
        return s["y"]
    if kind == "ground":
        E0, psi, _, _ = s["H"].lanczos(x0=s["x"], reorth=case["reorth"])
        return np.array([E0]), psi
    if kind == "batch":
        res = pg.lanczos_batch(s["H"], want_psi=True)
        return np.array([r[0] for r in res]), np.concatenate([r[1] for r in res])
    if kind == "green":
        e, Q = s["H"].build_Q_matrix_device(s["phi"])
        return pg.green_function(s["E0"] - e, Q, s["z"])
    if kind == "impurity":
        return pg.ModelInstance(s["cm"], s["values"], "R0:N8:S0").Green_function(s["z"])
    if kind in ("sef", "averages"):
        lat.set_wavevector_grid(case["nk"], case["nk"])
        lat.discrete_integration_grid(s["w"], s["wt"])
        if kind == "sef":
            return np.array([s["inst"].Potthoff_functional()])
        a = s["inst"].averages()
        return np.array([a[n] for n in sorted(a)])
    if kind == "cpt":
        return s["inst"].periodized_Green_function(s["z"], s["k"])
    return s["inst"].CDMFT_host(s["w"], s["wt"], kside=case["nk"])


# ---------------------------------------------------------------------------
# the work of one pass


def _dim(L, nup, ndn):
    return math.comb(L, nup) * math.comb(L, ndn)


def _product_flops(L, nup, ndn, bonds):
    """Multiply-adds of one product: a hop needs one of its two ends filled."""
    hops = sum(2.0 * bonds * n * (L - n) / (L * (L - 1)) for n in (nup, ndn))
    return 2.0 * (hops + 1) * _dim(L, nup, ndn)


def work(case):
    kind = case["kind"]
    if kind in ("product", "product64", "mult_add", "ground", "green"):
        L, nup, ndn = case["nx"] * case["ny"], case["nup"], case["ndn"]
        near, diag = _bonds(case["nx"], case["ny"])
        bonds = len(near) + (len(diag) if kind in ("product64", "green") or case.get("tp") else 0)
        D, prod = _dim(L, nup, ndn), _product_flops(L, nup, ndn, bonds)
        if kind in ("product", "product64", "mult_add"):
            return {"bytes": 24.0 * D, "flops": prod}
        if kind == "ground":  # about 100 steps: product and update; the replay for the vector, or the projections
            m = 100
            if case["reorth"]:
                return {"bytes": 8.0 * D * (m * 5 + 2 * m * m), "flops": m * prod + 4.0 * m * m * D}
            return {"bytes": 2 * m * 40.0 * D, "flops": 2 * m * (prod + 10.0 * D)}
        # about 600 vectors: product, L dots, L + 1 band updates each way
        D, prod = _dim(L, nup - 1, ndn), _product_flops(L, nup - 1, ndn, bonds)
        return {"bytes": 600 * 8.0 * D * (3 * L + 5), "flops": 600 * (prod + 6.0 * (L + 1) * D)}
    if kind == "batch":  # about 100 steps and as many of the replay
        D = case["instances"] * (2 * 3920 + 4900)
        return {"bytes": 200 * 40.0 * D, "flops": 200 * 40.0 * D}
    if kind == "impurity":  # ground state (200 products), two band Lanczos runs of 110 steps
        return {"bytes": 200 * 40.0 * 4900 + 220 * 8.0 * 3920 * 17,
                "flops": 200 * 40.0 * 4900 + 220 * 60.0 * 3920 + 8.0 * 16 * 220 * case["nw"]}
    L, M = len(_lattice(case)[0]), case["poles"]
    spins, nw = len(_spins(case)), case["nw"]
    nk = case["nk"] if kind == "cpt" else case["nk"] ** 2
    pts = nw * nk * spins
    per = {"sef": 8.0 / 3.0 * L ** 3, "cpt": 8.0 / 3.0 * L ** 3 + 8.0 * L * L}.get(kind, 8.0 * L ** 3)
    out = {"sef": 8, "cpt": 16 * pts, "host": 16 * nw * L * L, "averages": 24}[kind]
    return {"bytes": 8.0 * spins * M * (1 + 2 * L) + out, "flops": pts * per + 8.0 * L * L * M * nw * spins}


# ---------------------------------------------------------------------------
# the same results from plain torch and numpy


def _popcount(x):
    c = torch.zeros_like(x)
    for b in range(32):
        c += (x >> b) & 1
    return c


def _half(L, n):
    """Basis states of n electrons on L orbitals, increasing."""
    x = torch.arange(1 << L, device="cuda")
    return x[_popcount(x) == n]


def _hops(L, n, terms):
    """(source index, coefficient) of every hop term on the half basis: y[i] += c[i] x[src[i]]."""
    states = _half(L, n)
    out = []
    for i, j, v in terms:
        ni, nj = (states >> i) & 1, (states >> j) & 1
        moves = ni != nj
        src = torch.where(moves, states ^ ((1 << i) | (1 << j)), states)
        between = ((1 << max(i, j)) - 1) & ~((1 << (min(i, j) + 1)) - 1)
        sign = 1.0 - 2.0 * (_popcount(states & between) & 1).double()
        out.append((torch.searchsorted(states, src), torch.where(moves, v * sign, torch.zeros_like(sign))))
    return out


class _Hubbard:
    """H of one sector on (dn, up) arrays: hop terms, site energies per spin, U on `sites`."""

    def __init__(self, L, nup, ndn, terms, eup, edn, U, sites):
        self.shape = (math.comb(L, ndn), math.comb(L, nup))
        self.up, self.dn = _hops(L, nup, terms), _hops(L, ndn, terms)
        bu, bd = _half(L, nup), _half(L, ndn)
        self.diag = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        for k in range(L):
            nu, nd = ((bu >> k) & 1).double()[None, :], ((bd >> k) & 1).double()[:, None]
            self.diag += eup[k] * nu + edn[k] * nd + (U * nu * nd if k < sites else 0.0)

    def __call__(self, x):
        X = x.reshape(self.shape)
        y = self.diag * X
        for src, c in self.up:
            y += X[:, src] * c[None, :]
        for src, c in self.dn:
            y += X[src] * c[:, None]
        return y.reshape(-1)


def _cluster_exact(case, values, nup, ndn):
    nx, ny = case["nx"], case["ny"]
    near, diag = _bonds(nx, ny)
    terms = [(i, j, -values["t"]) for i, j in near]
    terms += [(i, j, -values["tp"]) for i, j in diag] if "tp" in values else []
    s = np.array(_neel(nx, ny)) * values.get("M", 0.0)
    return _Hubbard(nx * ny, nup, ndn, terms, s - values["mu"], -s - values["mu"], values["U"], nx * ny)


def _impurity_exact(values, nup, ndn):
    near, _ = _bonds(2, 2)
    terms = [(i, j, -values["t"]) for i, j in near] + [(k % 4, 4 + k, values[f"tb{k + 1}"]) for k in range(4)]
    e = np.array([-values["mu"]] * 4 + [values[f"eb{k + 1}"] for k in range(4)])
    return _Hubbard(8, nup, ndn, terms, e, e, values["U"], 4)


def _krylov(H, x0, steps, tol):
    """Lanczos with every vector projected out twice: (V, T) with V H V^T = T; stops
    when the lowest Ritz pair's residual is below tol (tol = 0: after `steps`)."""
    n = x0.numel()
    V = torch.empty((min(steps, n), n), dtype=torch.float64, device="cuda")
    V[0] = x0 / torch.linalg.vector_norm(x0)
    a, b = [], []
    for j in range(len(V)):
        w = H(V[j])
        a.append(float(V[j] @ w))
        for _ in range(2):
            w = w - (V[:j + 1] @ w) @ V[:j + 1]
        b.append(float(torch.linalg.vector_norm(w)))
        T = np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1)
        if b[-1] < 1e-12 or (tol and j % 5 == 4 and abs(np.linalg.eigh(T)[1][-1, 0]) * b[-1] < tol):
            break
        if j + 1 < len(V):
            V[j + 1] = w / b[-1]
    return V[:j + 1], T


def _lowest(H, x0):
    """Ground state (E0, psi) from the start vector x0."""
    V, T = _krylov(H, x0, 300, 1e-13)
    e, W = np.linalg.eigh(T)
    return float(e[0]), torch.from_numpy(W[:, 0]).cuda() @ V


def _removed(L, nup, ndn, psi, orb, pm):
    """c_orb (pm = -1) or its adjoint on the up electrons of psi."""
    src, dst = _half(L, nup), _half(L, nup + pm)
    ok = ((dst >> orb) & 1) == (1 if pm > 0 else 0)
    at = torch.searchsorted(src, torch.where(ok, dst ^ (1 << orb), src[0]))
    sign = torch.where(ok, 1.0 - 2.0 * (_popcount(dst & ((1 << orb) - 1)) & 1).double(), torch.zeros_like(dst).double())
    return (psi.reshape(math.comb(L, ndn), -1)[:, at] * sign[None, :]).reshape(-1)


def _dense(H):
    n = H.shape[0] * H.shape[1]
    A = torch.empty((n, n), dtype=torch.float64, device="cuda")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(n):
        x[k] = 1.0
        A[k] = H(x)
        x[k] = 0.0
    return A


def _cluster_green(case, seed, down, z):
    """G(z) (nz, L, L) of the saved solution."""
    e, v = (torch.from_numpy(a).cuda().to(torch.complex128) for a in _lehmann(case, seed, down))
    u = 1.0 / (z[:, None] - e[None, :])
    return (v[None] * u[:, None, :]) @ v.T


def _gamma(case, seed, z):
    tcb, eb = _bath(case, _lattice_params(case, seed)[1])
    t, e = torch.from_numpy(tcb).cuda().to(torch.complex128), torch.from_numpy(eb).cuda()
    return (t[None] / (z[:, None] - e[None, :])[:, None, :]) @ t.T


def _inter(case):
    """[(name, i, j, translation, amplitude)] of the lattice hops, each with its
    conjugate; translation (0, 0, 0) stays in the cluster."""
    sites, sup = _lattice(case)
    idx = {s: i for i, s in enumerate(sites)}
    lv, _ = _lattice_params(case, 0)
    out = []
    for name in LINKS:
        for d in (_links(case, name) if name in lv else ()):
            for i, s in enumerate(sites):
                r = tuple(a + b for a, b in zip(s, d))
                for n in itertools.product(range(-3, 4), repeat=len(sup)):
                    base = tuple(r[c] - sum(n[k] * sup[k][c] for k in range(len(sup))) for c in range(3))
                    if base in idx:
                        break
                n = tuple(n) + (0,) * (3 - len(n))
                out.append((name, i, idx[base], n, -1.0))
                out.append((name, idx[base], i, tuple(-c for c in n), -1.0))
    return out


def _hopping(case, seed, down, K):
    """t(K) - t_cluster (nK, L, L) for K in the superlattice's dual basis."""
    sites, _ = _lattice(case)
    lv, cv = _lattice_params(case, seed)
    h = torch.zeros((len(sites), len(sites)), dtype=torch.complex128, device="cuda")
    for i, s in enumerate(sites):
        sign = (1 if (s[0] + s[1]) % 2 == 0 else -1) * (-1 if down else 1)
        h[i, i] += (lv.get("M", 0.0) - cv.get("M", 0.0)) * sign
    V = h[None].repeat(len(K), 1, 1)
    for name, i, j, n, a in _inter(case):
        if any(n):
            V[:, i, j] += lv[name] * a * torch.exp(2j * math.pi * (K @ torch.tensor(n, dtype=torch.float64, device="cuda")))
    return V, h


def _grid(nk, off):
    k = (torch.arange(nk, dtype=torch.float64, device="cuda") + off) / nk
    K = torch.zeros((nk * nk, 3), dtype=torch.float64, device="cuda")
    K[:, 0], K[:, 1] = k.repeat(nk), k.repeat_interleave(nk)
    return K


def _exact_lattice(case, seed):
    kind = case["kind"]
    sites, sup = _lattice(case)
    L = len(sites)
    eye = torch.eye(L, dtype=torch.complex128, device="cuda")
    if kind == "cpt":
        z = torch.from_numpy(np.linspace(-8.0, 8.0, case["nw"]) + 0.1j).cuda()
        k = torch.arange(case["nk"], dtype=torch.float64, device="cuda") / case["nk"]
        K = torch.zeros((case["nk"], 3), dtype=torch.float64, device="cuda")
        K[:, 0] = k * case["nx"]
        V, _ = _hopping(case, seed, False, K)
        u = torch.exp(2j * math.pi * k[:, None] * torch.arange(L, device="cuda")[None, :])
        Gi = torch.linalg.inv(_cluster_green(case, seed, False, z))
        return torch.stack([(u.conj() * torch.linalg.solve(g[None] - V, u[:, :, None])[:, :, 0]).sum(1) / L for g in Gi])
    if kind == "host":
        w = _matsubara(case["nw"])
        z = torch.from_numpy(1j * w).cuda()
        V, _ = _hopping(case, seed, False, _grid(case["nk"], 0.5))
        Gi, Gm = torch.linalg.inv(_cluster_green(case, seed, False, z)), _gamma(case, seed, z)
        P = torch.stack([torch.linalg.inv(g[None] - V).mean(0) for g in Gi + Gm])
        return {False: torch.linalg.inv(P) - Gm - Gi}
    w, wt = _lattice_grid(case["nw"])
    z = torch.from_numpy(1j * w).cuda()
    K = _grid(case["nk"], 0.0)
    lv, cv = _lattice_params(case, seed)
    if kind == "sef":
        total = -10.0
        for down in (False, True):
            V, h = _hopping(case, seed, down, K)
            G = _cluster_green(case, seed, down, z)
            for q in range(len(w)):
                total -= wt[q] * float(torch.linalg.slogdet(V @ G[q][None] - eye[None])[1].mean())
            total += 0.5 * float(h.diagonal().real.sum())
        return np.array([total / L])
    names = ("M", "mu", "t", "tp")
    got = dict.fromkeys(names, 0.0)
    phase = {n: torch.exp(2j * math.pi * (K @ torch.tensor(n, dtype=torch.float64, device="cuda")))
             for n in {t[3] for t in _inter(case)} | {(0, 0, 0)}}
    for down in (False, True):
        V, _ = _hopping(case, seed, down, K)
        Gi = torch.linalg.inv(_cluster_green(case, seed, down, z))
        sgn = [(1 if (s[0] + s[1]) % 2 == 0 else -1) * (-1 if down else 1) for s in sites]
        els = _inter(case) + [("M", i, i, (0, 0, 0), float(sgn[i])) for i in range(L)]
        els += [("mu", i, i, (0, 0, 0), -1.0) for i in range(L)]
        for q in range(len(w)):
            Gc = torch.linalg.inv(Gi[q][None] - V) - eye[None] / (z[q] - 2.0)
            mean = {n: (Gc * p[:, None, None]).mean(0).cpu().numpy() for n, p in phase.items()}
            for name, r, c, n, a in els:
                got[name] += wt[q] * (a * mean[n][c, r]).real
    return np.array([got[n] / (-L if n == "mu" else L) for n in names])


def exact(case, seed):
    kind = case["kind"]
    if kind == "product":
        return None  # whole numbers
    if kind in ("product64", "mult_add"):
        tp = kind == "product64" or case["tp"]
        H = _cluster_exact(case, _vca_values(seed) if tp else HUBBARD, case["nup"], case["ndn"])
        n = H.shape[0] * H.shape[1]
        if kind == "product64":
            return _device_unit(n, seed + 1000003) + H(_device_unit(n, seed))
        x, y = (torch.from_numpy(_unit(n, k)).cuda() for k in (seed, seed + 1000003))
        return (y + H(x)).cpu().numpy()
    if kind == "ground":  # the vector's sign is the solver's own
        H = _cluster_exact(case, HUBBARD, case["nup"], case["ndn"])
        return [np.array([_lowest(H, torch.from_numpy(_unit(H.shape[0] * H.shape[1], seed)).cuda())[0]]), None]
    if kind == "batch":
        E = []
        for sector, values in _batch_problems(case, seed):
            n, s = int(sector.split(":")[1][1:]), int(sector.split(":")[2][1:])
            H = _impurity_exact(values, (n + s) // 2, (n - s) // 2)
            E.append(_lowest(H, _device_unit(H.shape[0] * H.shape[1], 7))[0])
        return [np.array(E), None]
    if kind == "green":
        L, nup, ndn = case["nx"] * case["ny"], case["nup"], case["ndn"]
        values = _vca_values(seed)
        x0 = torch.from_numpy(_unit(_dim(L, nup, ndn), seed)).cuda()
        E0, psi = _lowest(_cluster_exact(case, values, nup, ndn), x0)
        H = _cluster_exact(case, values, nup - 1, ndn)
        phi = torch.stack([_removed(L, nup, ndn, psi, o, -1) for o in range(L)])
        z = 1j * _matsubara(case["nw"])
        G = np.zeros((len(z), L, L), np.complex128)
        for b in range(L):
            V, T = _krylov(H, phi[b], 160, 0.0)
            P = (phi @ V.T).cpu().numpy() * float(torch.linalg.vector_norm(phi[b]))
            e, W = np.linalg.eigh(T)
            G[:, :, b] = ((W[0][None, :] / (z[:, None] - (E0 - e)[None, :])) @ (P @ W).T)
        return G
    if kind == "impurity":
        values = _impurity_values(np.random.default_rng([seed, 6]), 4)
        E0, psi = _lowest(_impurity_exact(values, 4, 4), _device_unit(4900, 7))
        z = torch.from_numpy(1j * _matsubara(case["nw"])).cuda()
        G = torch.zeros((len(z), 4, 4), dtype=torch.complex128, device="cuda")
        for pm in (-1, 1):
            e, W = torch.linalg.eigh(_dense(_impurity_exact(values, 4 + pm, 4)))
            q = (torch.stack([_removed(8, 4, 4, psi, o, pm) for o in range(4)]) @ W).to(torch.complex128)
            G += (q[None] / (z[:, None] - pm * (e - E0)[None, :])[:, None, :]) @ q.T
        return G.cpu().numpy()
    return _exact_lattice(case, seed)
