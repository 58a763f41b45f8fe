"""The work that a program has this engine do, as cases that can be timed.

Every case goes through the public entry points: the builders' engine
(chem_gb300.fock.JKEngine), the molecule set-up and the MP2 driver.  The
molecules are the ones of the repository's own workloads (water, water
clusters, all-trans alkanes, cc-pVDZ with the jkfit or ri auxiliary basis)
and its seeded synthetic tensor; the sizes run from one water molecule to
C20H42.  A case names the molecule, the seed makes what changes between
calls: orbitals and densities, or the geometry where the set-up itself is
the work.
"""
from __future__ import annotations

import functools

import numpy as np
import torch

from chem_gb300 import geometry, ints, mp2
from chem_gb300.dfsystem import build_dfsystem
from chem_gb300.fock import JKEngine, host_array
from chem_gb300.layout import schwarz_layout
from chem_gb300.molecule import molecule_from_angstrom
from chem_gb300.synthetic import occupied, synthetic_layout

EPS = 1e-10  # Schwarz and block-filter threshold of the repository's workloads


def listed():
    return [
        # The smallest call: one water molecule on the FP64 path (the
        # reference's own example), where launches and latency are the time.
        {"name": "water_fp64", "kind": "fock", "mol": "water", "n": 1, "precision": "fp64",
         "kmethod": "dfmo", "jmode": "vinv"},
        # A small request of a serving loop: a water cluster, every call one
        # Fock build on the mixed path.
        {"name": "water5_split", "kind": "fock", "mol": "water", "n": 5, "precision": "split",
         "kmethod": "dfmo", "jmode": "cholesky"},
        # An ordinary Fock build: decane on the mixed path.
        {"name": "c10h22_split", "kind": "fock", "mol": "alkane", "n": 10, "precision": "split",
         "kmethod": "dfmo", "jmode": "cholesky"},
        # The repository's headline: one C20H42 Fock build on the mixed path,
        # host matrices in and out.
        {"name": "c20h42_split", "kind": "fock", "mol": "alkane", "n": 20, "precision": "split",
         "kmethod": "dfmo", "jmode": "cholesky"},
        # The last iterations of an SCF run on the FP64 path.
        {"name": "c8h18_fp64", "kind": "fock", "mol": "alkane", "n": 8, "precision": "fp64",
         "kmethod": "dflmo", "jmode": "cholesky"},
        # Exchange from a density alone (the DF-AO builder).
        {"name": "c12h26_dfao", "kind": "dfao", "mol": "alkane", "n": 12},
        # Exchange between different left and right orbitals, as the ADC
        # matrix-vector products request it; an odd number of vectors.
        {"name": "c14h30_asym", "kind": "asym", "mol": "alkane", "n": 14, "nocc": 37},
        # One SCF iteration on the device: Fock build, energy, DIIS error and
        # overlaps, then the extrapolated Fock matrix.
        {"name": "c10h22_scf", "kind": "scf", "mol": "alkane", "n": 10},
        # A molecule the engine has not seen, its integrals already on the
        # host: upload, fit with the metric, first Fock build.
        {"name": "c12h26_new", "kind": "newmol", "mol": "alkane", "n": 12, "ints": "host"},
        # A new geometry with the integrals computed on the device.
        {"name": "water6_geometry", "kind": "newmol", "mol": "water", "n": 6, "ints": "device"},
        # SOS-AO-MP2: the Laplace sum over eight quadrature points.
        {"name": "c8h18_mp2", "kind": "mp2", "mol": "alkane", "n": 8, "nlap": 8},
        # Exchange of a pre-fitted block-sparse tensor in auxiliary batches.
        {"name": "synthetic_k", "kind": "synthetic", "nbf": 1200, "naux": 3600, "nocc": 180,
         "batch": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["fock", "fock", "fock", "fp64", "dfao", "asym", "scf", "newmol", "newmol",
                       "mp2", "synthetic"])
    if kind == "fock":
        mol = rng.choice(["alkane", "water"])
        return {"kind": "fock", "mol": mol, "n": _log(rng, 2, 19) if mol == "alkane" else
                _log(rng, 1, 14), "precision": "split", "kmethod": rng.choice(["dfmo", "dflmo"]),
                "jmode": "cholesky"}
    if kind == "fp64":
        mol = rng.choice(["alkane", "water"])
        return {"kind": "fock", "mol": mol, "n": rng.randint(1, 9), "precision": "fp64",
                "kmethod": rng.choice(["dfmo", "dflmo"]),
                "jmode": rng.choice(["vinv", "cholesky"])}
    if kind == "dfao":
        return {"kind": "dfao", "mol": "alkane", "n": rng.randint(3, 13)}
    if kind == "asym":
        return {"kind": "asym", "mol": "alkane", "n": rng.randint(5, 16),
                "nocc": _log(rng, 3, 110)}
    if kind == "scf":
        return {"kind": "scf", "mol": rng.choice(["alkane", "water"]), "n": rng.randint(2, 13)}
    if kind == "newmol":
        mol = rng.choice(["alkane", "water"])
        ints_ = rng.choice(["host", "device"])
        return {"kind": "newmol", "mol": mol, "ints": ints_,
                "n": rng.randint(2, 11 if ints_ == "host" else 8)}
    if kind == "mp2":
        return {"kind": "mp2", "mol": "alkane", "n": rng.randint(2, 8), "nlap": rng.randint(3, 8)}
    return {"kind": "synthetic", "nbf": _log(rng, 300, 1190), "naux": _log(rng, 700, 3500),
            "nocc": _log(rng, 30, 175), "batch": rng.choice([256, 512, 800, 1024])}


# ---- molecules -------------------------------------------------------------

def _molecule(mol, n, dfbasis="cc-pvdz-jkfit", seed=None):
    if mol == "alkane":
        sym, xyz = geometry.alkane(n)
    elif n == 1:
        sym, xyz = geometry.water()
    else:
        sym, xyz = geometry.water_cluster(n, np.random.default_rng(1000 + n))
    if seed is not None:  # a step of a geometry optimisation or of dynamics
        xyz = xyz + np.random.default_rng(seed).normal(0.0, 0.01, xyz.shape)
    return molecule_from_angstrom(sym, xyz, "cc-pvdz", dfbasis)


@functools.lru_cache(maxsize=2)
def _system(mol, n, dfbasis="cc-pvdz-jkfit"):
    """Host set-up of a fixed molecule: a program makes it once and keeps it."""
    return build_dfsystem(_molecule(mol, n, dfbasis), eps=EPS)


def _orbitals(ds, nocc, seed):
    """Occupied orbitals of a Fock matrix near the core Hamiltonian's, as the
    iterations of an SCF run pass them: orthonormal in the overlap metric."""
    s, U = np.linalg.eigh(ds.S)
    X = (U * s ** -0.5) @ U.T
    F = X @ ds.Hcore @ X
    N = np.random.default_rng(seed).normal(0.0, 0.02, F.shape)
    _, C = np.linalg.eigh(F + 0.5 * (N + N.T))
    return np.ascontiguousarray(X @ C[:, :nocc])


def _pinned(a):
    out = host_array(a.shape)
    out[...] = a
    return out


def _new_case(case, seed):
    """(molecule, host system) of a set-up case: its geometry is the seed's."""
    m = _molecule(case["mol"], case["n"], seed=seed)
    return m, build_dfsystem(m, eps=EPS, device_ints=case["ints"] == "device")


# ---- inputs ----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "synthetic":
        layout, decay = synthetic_layout(case["nbf"], case["naux"])
        st["eng"] = JKEngine(layout, None, None, None, eps=0.0, precision="split", fitted=True,
                             synthetic=(seed, decay), aux_batch=case["batch"])
        st["C"] = _pinned(occupied(case["nbf"], case["nocc"], seed))
        st["K"] = host_array((case["nbf"], case["nbf"]))
        return st
    if kind == "newmol":
        m, ds = _new_case(case, seed)
        st["ds"] = ds
        C = _orbitals(ds, m.nocc, seed)
        st["C"], st["P"] = C, 2.0 * (C @ C.T)
        return st
    if kind == "mp2":
        ds = _system(case["mol"], case["n"], "cc-pvdz-ri")
        st["eng"] = JKEngine(ds.layout, ds.B, ds.Linv, ds.Vinv, eps=EPS, precision="split")
        Co, Cv, eo, ev = _mp2_orbitals(ds, case, seed)
        st["factors"] = mp2.laplace_factors(Co, Cv, eo, ev, ds.S, case["nlap"])
        return st
    ds = _system(case["mol"], case["n"])
    n = ds.nbf
    st["eng"] = eng = JKEngine(ds.layout, ds.B, ds.Linv, ds.Vinv, eps=EPS,
                               precision=case.get("precision", "split"))
    if kind == "fock":
        eng.set_jmode(case["jmode"])
        C = _orbitals(ds, ds.nocc, seed)
        st["C"], st["P"] = _pinned(C), _pinned(2.0 * (C @ C.T))
        st["out"] = (host_array((n, n)), host_array((n, n)))
        st["kmethod"] = case["kmethod"]
    elif kind == "dfao":
        C = _orbitals(ds, ds.nocc, seed)
        st["P"] = _pinned(C @ C.T)
    elif kind == "asym":
        st["U"], st["Vt"] = _pair(ds, case["nocc"], seed)
    elif kind == "scf":
        s, U = np.linalg.eigh(ds.S)
        eng.scf_begin(ds.Hcore, ds.S, (U * s ** -0.5) @ U.T, ds.nocc)
        for slot in (0, 1):  # the two iterations before this one
            eng.scf_build(_orbitals(ds, ds.nocc, 3 * seed + slot), slot)
        st["C"] = _orbitals(ds, ds.nocc, 3 * seed + 2)
        st["coef"] = _diis()
    return st


def _mp2_orbitals(ds, case, seed):
    """Random orthonormal orbitals of the seed; the orbital energies, and so
    the quadrature, are the molecule's."""
    Co, Cv, _, _ = mp2.random_orbitals(ds.S, ds.nocc, seed)
    _, _, eo, ev = mp2.random_orbitals(ds.S, ds.nocc, 77)
    return Co, Cv, eo, ev


def _pair(ds, nocc, seed):
    """Left (nbf x nocc) and right (nocc x nbf) vectors: orbitals and a
    response of them."""
    U = _orbitals(ds, nocc, seed)
    R = np.random.default_rng(seed + 1).normal(0.0, 0.05, (nocc, nocc))
    return U, np.ascontiguousarray((U + U @ R).T)


def _diis():
    c = np.zeros(8)
    c[:3] = 0.1, -0.3, 1.2
    return c


# ---- one pass ---------------------------------------------------------------

def run(st):
    kind = st["kind"]
    if kind == "fock":
        return st["eng"].compute_jk(st["P"], st["C"], st["kmethod"], out=st["out"])
    if kind == "dfao":
        return st["eng"].compute_k_ao(st["P"])
    if kind == "asym":
        return st["eng"].compute_k_lmo_asym(st["U"], st["Vt"])
    if kind == "scf":
        e, rms, ov = st["eng"].scf_build(st["C"], 2)
        return e, rms, ov, st["eng"].scf_extrapolate(st["coef"])
    if kind == "newmol":
        ds = st["ds"]
        eng = JKEngine(ds.layout, ds.B, ds.Linv, ds.Vinv, eps=EPS, precision="split")
        J, K = eng.compute_jk(st["P"], st["C"])
        eng.close()
        return J, K
    if kind == "mp2":
        return mp2.sos_mp2_laplace(st["eng"], st["factors"])
    return st["eng"].compute_jk(Cocc=st["C"], out=(None, st["K"]))[1]


# ---- what a pass cannot do without -------------------------------------------

def _pairs(layout):
    """Kept function pairs (mu, nu) in both orders, and with mu <= nu."""
    both = int(layout.panel_K @ layout.bsizes)
    return both, (both + layout.nbf) // 2


def work(case):
    kind = case["kind"]
    if kind == "synthetic":
        layout, _ = synthetic_layout(case["nbf"], case["naux"])
        n, x, o = case["nbf"], case["naux"], case["nocc"]
        both, up = _pairs(layout)
        return {"bytes": 8 * (x * up + n * o + n * n),
                "flops": 2 * x * both * o + x * o * n * (n + 1)}
    df = "cc-pvdz-ri" if kind == "mp2" else "cc-pvdz-jkfit"
    m = _molecule(case["mol"], case["n"], df)
    layout = schwarz_layout(m, *ints.schwarz(m), EPS)
    n, x, o = layout.nbf, layout.naux, case.get("nocc", m.nocc)
    both, up = _pairs(layout)
    tensor, metric = 8 * x * up, 8 * x * (x + 1) // 2
    build = 4 * x * up + 2 * x * x  # both passes of J and the metric between them
    build += 2 * x * both * o + x * o * n * (n + 1)  # half transform, exchange
    fit = x * x * min(up, n * o)  # the metric's factor on whichever side is smaller
    if kind == "fock":
        split = case["precision"] == "split"  # the fitted tensor is resident
        return {"bytes": tensor + metric + 8 * (3 * n * n + n * o),
                "flops": build + (0 if split else fit)}
    if kind == "newmol":
        given = tensor + metric if case["ints"] == "host" else metric
        return {"bytes": given + 8 * (3 * n * n + n * o), "flops": build + fit}
    if kind == "dfao":
        return {"bytes": tensor + 16 * n * n, "flops": 2 * x * both * n + x * n * n * (n + 1)}
    if kind == "asym":
        return {"bytes": tensor + 8 * (n * n + 2 * n * o),
                "flops": 4 * x * both * o + 2 * x * o * n * n}
    if kind == "scf":
        return {"bytes": tensor + metric + 8 * (6 * n * n + n * o), "flops": build + 10 * n ** 3}
    v = n - o  # mp2
    point = 2 * x * both * o + 2 * x * o * n * v + x * x * o * v + 2 * x * x
    return {"bytes": tensor + 8 * case["nlap"] * n * n, "flops": case["nlap"] * point}


# ---- the same in 64 bits -------------------------------------------------------

def _gpu(a):
    return torch.from_numpy(np.array(a)).cuda()


def _dense(layout, B):
    """The dense tensor (naux, nbf, nbf) of a panel array."""
    n, x = layout.nbf, layout.naux
    off = np.concatenate([[0], np.cumsum(layout.bsizes)]).astype(int)
    T = torch.zeros((x, n, n), dtype=torch.float64, device="cuda")
    for i in range(layout.nblk):
        b, k, o = int(layout.bsizes[i]), int(layout.panel_K[i]), int(layout.panel_off[i])
        cols = np.concatenate([np.arange(off[j], off[j + 1]) for j in layout.nbr[i]])
        P = _gpu(B[o:o + b * x * k].reshape(b, x, k))
        rows = T[:, off[i]:off[i + 1], :]
        rows[:, :, torch.from_numpy(cols).cuda()] = P.permute(1, 0, 2)
    return T


def _filter(M, layout):
    off = np.concatenate([[0], np.cumsum(layout.bsizes)]).astype(int)
    for i in range(layout.nblk):
        for j in range(layout.nblk):
            blk = M[off[i]:off[i + 1], off[j]:off[j + 1]]
            if np.linalg.norm(blk) < EPS:
                blk[...] = 0.0
    return M


def _half(T, Linv, C):
    """L^-1 (X|mu i) as a (naux, nbf * nocc) matrix."""
    x, n, _ = T.shape
    H = torch.matmul(T.reshape(x * n, n), C).reshape(x, -1)
    return Linv @ H


def _exchange(Hu, Hv, n):
    x = Hu.shape[0]
    a = Hu.reshape(x, n, -1).permute(1, 0, 2).reshape(n, -1)
    b = a if Hv is Hu else Hv.reshape(x, n, -1).permute(1, 0, 2).reshape(n, -1)
    return -(a @ b.T)


def _exact_jk(ds, B, C, P, vinv=False):
    T = _dense(ds.layout, B)
    Linv, Cg, Pg = _gpu(ds.Linv), _gpu(C), _gpu(P)
    g = torch.einsum("xmn,mn->x", T, Pg)
    h = _gpu(ds.Vinv) @ g if vinv else Linv.T @ (Linv @ g)
    J = torch.einsum("xmn,x->mn", T, h)
    H = _half(T, Linv, Cg)
    return J, _exchange(H, H, ds.nbf)


def exact(case, seed):
    kind = case["kind"]
    if kind == "synthetic":
        layout, decay = synthetic_layout(case["nbf"], case["naux"])
        eng = JKEngine(layout, None, None, None, fitted=True, synthetic=(seed, decay))
        B = eng.download_b()  # the seeded tensor is made on the device
        eng.close()
        n, x = case["nbf"], case["naux"]
        C = _gpu(occupied(n, case["nocc"], seed))
        off = np.concatenate([[0], np.cumsum(layout.bsizes)]).astype(int)
        H = torch.zeros((n, x, case["nocc"]), dtype=torch.float64, device="cuda")
        for i in range(layout.nblk):
            b, k, o = int(layout.bsizes[i]), int(layout.panel_K[i]), int(layout.panel_off[i])
            cols = np.concatenate([np.arange(off[j], off[j + 1]) for j in layout.nbr[i]])
            H[off[i]:off[i + 1]] = _gpu(B[o:o + b * x * k].reshape(b, x, k)) @ \
                C[torch.from_numpy(cols).cuda()]
        H = H.reshape(n, -1)
        return -(H @ H.T).cpu().numpy()
    if kind == "newmol":
        m, ds = _new_case(case, seed)
        B = ints.eri3c_panels(m, ds.layout) if case["ints"] == "device" else ds.B
        C = _orbitals(ds, m.nocc, seed)
        J, K = _exact_jk(ds, B, C, 2.0 * (C @ C.T))
        return tuple(_filter(M.cpu().numpy(), ds.layout) for M in (J, K))
    if kind == "mp2":
        ds = _system(case["mol"], case["n"], "cc-pvdz-ri")
        Co, Cv, eo, ev = _mp2_orbitals(ds, case, seed)
        f = mp2.laplace_factors(Co, Cv, eo, ev, ds.S, case["nlap"])
        x, n = ds.naux, ds.nbf
        T = (_gpu(ds.Linv) @ _dense(ds.layout, ds.B).reshape(x, n * n)).reshape(x, n, n)
        e = np.zeros(case["nlap"])
        for t in range(case["nlap"]):
            H = torch.einsum("xnm,mi->xin", T, _gpu(f.Lo[t]))
            W = torch.matmul(H, _gpu(f.Lv[t])).reshape(x, -1)
            e[t] = float((W @ W.T).square().sum())
        return {"points": e, "energy": float(e.sum()), "scaled": 1.3 * float(e.sum())}
    ds = _system(case["mol"], case["n"])
    n = ds.nbf
    if kind == "fock":
        C = _orbitals(ds, ds.nocc, seed)
        J, K = _exact_jk(ds, ds.B, C, 2.0 * (C @ C.T), vinv=case["jmode"] == "vinv")
        return tuple(_filter(M.cpu().numpy(), ds.layout) for M in (J, K))
    T, Linv = _dense(ds.layout, ds.B), _gpu(ds.Linv)
    if kind == "dfao":
        C = _orbitals(ds, ds.nocc, seed)
        Bf = (Linv @ T.reshape(ds.naux, n * n)).reshape(ds.naux, n, n)
        K = _exchange(torch.matmul(Bf, _gpu(C @ C.T)), Bf, n)
        return _filter(K.cpu().numpy(), ds.layout)
    if kind == "asym":
        U, Vt = _pair(ds, case["nocc"], seed)
        K = _exchange(_half(T, Linv, _gpu(U)), _half(T, Linv, _gpu(Vt.T)), n)
        return _filter(K.cpu().numpy(), ds.layout)
    s, U = np.linalg.eigh(ds.S)
    X = (U * s ** -0.5) @ U.T
    Fs, errs, e = [], [], 0.0
    del T
    for slot in range(3):
        C = _orbitals(ds, ds.nocc, 3 * seed + slot)
        P = C @ C.T
        J, K = (_filter(M.cpu().numpy(), ds.layout) for M in _exact_jk(ds, ds.B, C, 2.0 * P))
        F = ds.Hcore + J + K
        Fs.append(F)
        errs.append(F @ P @ ds.S - ds.S @ P @ F)
        e = float(np.sum(P * (ds.Hcore + F)))
    ov = np.zeros(8)
    ov[:3] = [float(np.sum(errs[2] * q)) for q in errs]
    Fo = X @ sum(c * F for c, F in zip(_diis(), Fs)) @ X
    return e, float(np.sqrt(np.mean(errs[2] ** 2))), ov, Fo
