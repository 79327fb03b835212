"""The work a user of this package has it do, as timed cases: two-site gates, canonical forms,
environment contractions, the batched engine and a whole TEBD run, each through the Python mirror
of the reference's API.

Outputs are gauge-invariant: singular vectors are fixed only up to a phase per column, so a case
that factorises a bond returns the bond's spectrum and the two sites contracted over it (the state
the call leaves on them) instead of the sites themselves.  QR factors have a fixed convention
(LAPACK's real diagonal) and are returned as they are.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "qrochet.jl_gb300"))
import qrochet as Q  # noqa: E402
from qrochet import random as R  # noqa: E402
from qrochet.batch import Batch  # noqa: E402
from qrochet.serve import random_request  # noqa: E402

D = 2  # qubits, the physical dimension of every workload here


def listed():
    return [
        # a gate on the bonds near the ends of a chain, or early in a circuit: latency only
        {"name": "gate fp64 chi16", "kind": "gate", "precision": "fp64", "cl": 16, "cb": 16, "cr": 16, "decades": 2.0},
        # a gate in the middle of a plain ComplexF64 simulation
        {"name": "gate fp64 chi128", "kind": "gate", "precision": "fp64", "cl": 128, "cb": 128, "cr": 128, "decades": 3.0},
        # mixed precision on the uneven bonds that a cutoff leaves behind
        {"name": "gate mixed ragged", "kind": "gate", "precision": "mixed", "cl": 93, "cb": 101, "cr": 77, "decades": 4.0},
        # a bond of a weakly entangled state: the Schmidt values decay over many decades
        {"name": "gate mixed chi384 decay", "kind": "gate", "precision": "mixed", "cl": 384, "cb": 384, "cr": 384, "decades": 7.0},
        # the headline: a TEBD step at chi = 1024 on both sides (theta 2048 x 2048)
        {"name": "gate mixed chi1024", "kind": "gate", "precision": "mixed", "cl": 1024, "cb": 1024, "cr": 1024, "decades": 0.5},
        # one step of a canonize! QR sweep at a large bond
        {"name": "canonize qr chi512", "kind": "canonize", "method": "qr", "direction": "right", "precision": "fp64",
         "cl": 512, "cb": 512, "cr": 512},
        # one step of the SVD sweep back, on uneven bonds
        {"name": "canonize svd fp64", "kind": "canonize", "method": "svd", "direction": "left", "precision": "fp64",
         "cl": 163, "cb": 190, "cr": 178},
        # canonize!, norm and every nearest-neighbour <ZZ> of a small chain
        {"name": "chain canonize n16", "kind": "chain", "precision": "fp64", "n": 16, "chi": 32},
        # Pauli strings on a mid-sized state in plain FP64
        {"name": "expect fp64 chi256", "kind": "env", "op": "expect", "precision": "fp64", "n": 32, "chi": 256, "strings": 4},
        # energy of a large state, contractions in split precision
        {"name": "mpo split chi704", "kind": "env", "op": "mpo", "precision": "split", "n": 40, "chi": 704, "strings": 1},
        # a batch of uneven circuits, simulate and measure
        {"name": "batch mixed", "kind": "batch", "precision": "mixed", "requests": 32, "n_max": 40, "depth_max": 9,
         "chi_log2": 6, "layout": 17},
        # a whole brick-wall TEBD run from |0...0> with its read-out
        {"name": "tebd mixed n32", "kind": "tebd", "precision": "mixed", "n": 32, "depth": 11, "chi": 64},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gate", "gate", "gate", "canonize", "canonize", "env", "env", "chain", "batch", "tebd"])
    if kind == "gate":
        prec = rng.choice(["fp64", "mixed", "mixed"])
        b = _logint(rng, 9, 150 if prec == "fp64" else 600)
        return {"kind": kind, "precision": prec, "cl": max(8, int(b * rng.uniform(0.75, 1.2))), "cb": b,
                "cr": max(8, int(b * rng.uniform(0.75, 1.2))), "decades": round(rng.uniform(0.5, 7.5), 2)}
    if kind == "canonize":
        method = rng.choice(["qr", "svd"])
        prec = rng.choice(["fp64", "mixed"])
        b = _logint(rng, 9, 800 if method == "qr" else 220 if prec == "fp64" else 500)
        return {"kind": kind, "method": method, "direction": rng.choice(["left", "right"]), "precision": prec,
                "cl": max(8, int(b * rng.uniform(0.7, 1.2))), "cb": b, "cr": max(8, int(b * rng.uniform(0.7, 1.2)))}
    if kind == "env":
        op = rng.choice(["expect", "mpo", "overlap", "norm"])
        prec = rng.choice(["fp64", "fp64", "split"])
        top = 560 if prec == "split" else 128 if op == "mpo" else 230
        return {"kind": kind, "op": op, "precision": prec, "n": rng.randint(6, 32), "chi": _logint(rng, 9, top),
                "strings": rng.randint(1, 4) if op == "expect" else 1}
    if kind == "chain":
        return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "n": rng.randint(6, 20), "chi": rng.randint(12, 40)}
    if kind == "batch":
        return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "requests": _logint(rng, 2, 30),
                "n_max": rng.randint(12, 40), "depth_max": rng.randint(5, 9), "chi_log2": rng.choice([5, 6]),
                "layout": rng.randint(1, 10 ** 6)}
    return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "n": rng.randint(8, 28), "depth": rng.randint(4, 10),
            "chi": rng.randint(14, 60)}


# ---- inputs ---------------------------------------------------------------------------------------
def _randc(gen, *shape):
    """Standard complex Gaussian entries on the GPU, as a Fortran-ordered host array."""
    t = torch.randn(tuple(reversed(shape)), dtype=torch.complex128, device="cuda", generator=gen)
    return t.cpu().numpy().T


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _pair(case, seed):
    """Two neighbouring sites (reference layout, dims (o, l, r)), the Lambda between them (norm 1,
    decaying over `decades`) and a Haar gate."""
    g = _gen(seed)
    cl, cb, cr = case["cl"], case["cb"], case["cr"]
    a = _randc(g, D, cl, cb) / math.sqrt(D * cl)
    b = _randc(g, D, cb, cr) / math.sqrt(D * cr)
    lam = 10.0 ** (-case.get("decades", 0.5) * np.arange(cb) / cb)
    lam /= np.linalg.norm(lam)
    return np.asfortranarray(a), np.asfortranarray(b), lam, R.haar_unitary(R.rng(seed), D * D)


def _sites(case, seed):
    """A uniform chain in reference layout with polarised qubits (so that <Z> does not vanish)."""
    g = _gen(seed)
    n, chi = case["n"], case["chi"]
    w = np.array([1.0, 0.6]) / math.sqrt(1.36)
    out = []
    for i in range(n):
        cl, cr = (1 if i == 0 else chi), (1 if i == n - 1 else chi)
        a = _randc(g, D, cl, cr) * (w / math.sqrt(cl))[:, None, None]
        out.append(np.asfortranarray(a[:, 0, :] if i == 0 else a[:, :, 0] if i == n - 1 else a))
    return out


def _strings(case, seed):
    """Pauli strings of weight 1-4 on random sites: [[(site, letter)]]."""
    g = R.rng(seed + 1)
    out = []
    for _ in range(case["strings"]):
        w = int(g.integers(1, 5))
        out.append([(int(s), "Z") for s in sorted(g.choice(case["n"], size=w, replace=False) + 1)])
    return out


def _requests(case, seed):
    """Uneven circuits and Pauli strings laid out by the case's `layout`; the Haar gates are the seed's."""
    g, h = R.rng(case["layout"]), R.rng(seed)
    out = [random_request(g, n_range=(8, case["n_max"]), depth_range=(3, case["depth_max"]),
                          chi_choices=tuple(2 ** k for k in range(4, case["chi_log2"] + 1)), nobs=2)
           for _ in range(case["requests"])]
    for r in out:
        r.gates = [(s, R.haar_unitary(h, D * D)) for s, _ in r.gates]
    return out


def _gate_on(m, *sites):
    return Q.gate_from_matrix(m, list(sites))


def _end_sites(cl, cr):
    """The outer sites of a four-site chain around a pair with these outer bonds."""
    return np.full((D, cl), 1.0 / cl, dtype=np.complex128), np.full((D, cr), 1.0 / cr, dtype=np.complex128)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("gate", "canonize"):
        a, b, lam, u = _pair(case, seed)
        left, right = _end_sites(case["cl"], case["cr"])
        s["psi"] = Q.MPS([left, a, b, right])
        s["psi"].set_precision(case["precision"])
        s["pinned"] = [Q.PinnedArray(a.shape), Q.PinnedArray(b.shape), Q.PinnedArray(a.shape), Q.PinnedArray(b.shape)]
        s["a"], s["b"], s["a_out"], s["b_out"] = (p.array for p in s["pinned"])
        s["a"][...], s["b"][...] = a, b
        s["lam"], s["gate"] = lam, _gate_on(u, 2, 3)
    elif kind == "env":
        s["psi"] = Q.MPS(_sites(case, seed))
        s["psi"].set_precision(case["precision"])
        if case["op"] == "overlap":
            arrays = _sites(case, seed)
            noise = _sites(case, seed + 7919)
            s["phi"] = Q.MPS([x + 0.1 * y for x, y in zip(arrays, noise)])
            s["phi"].set_precision(case["precision"])
        elif case["op"] == "mpo":
            s["mpo"] = Q.MPO(R.xxz_mpo_arrays(case["n"]))
        elif case["op"] == "expect":
            s["obs"] = [[_gate_on(R.PAULI[p], i) for i, p in o] for o in _strings(case, seed)]
    elif kind == "chain":
        s["psi"] = Q.MPS(_sites(case, seed))
        s["psi"].set_precision(case["precision"])
        zz = np.kron(R.PAULI["Z"], R.PAULI["Z"])
        s["obs"] = [_gate_on(zz, i, i + 1) for i in range(1, case["n"])]
    elif kind == "batch":
        s["requests"] = _requests(case, seed)
    else:
        s["layers"] = [[_gate_on(m, i, i + 1) for i, m in layer]
                       for layer in R.brickwall_layers(case["n"], case["depth"], seed)]
        s["obs"] = [_gate_on(R.PAULI["X"], i) for i in range(1, case["n"] + 1)]
    return s


# ---- the calls --------------------------------------------------------------------------------------
def _to_gpu(x):
    """A downloaded site (o, l, r), column-major, as the (r, l, o) GPU tensor of the same memory order."""
    return torch.from_numpy(x.T).cuda()


def _merged(a, lam, b):
    """The state on two sites, A diag(lam) B as a ((l, o) x (o, r)) matrix on the GPU."""
    a, b = _to_gpu(a), _to_gpu(b)
    cb, cl = a.shape[0], a.shape[1]
    at = a.reshape(cb, cl * D) * torch.from_numpy(lam).cuda()[:, None]
    bt = b.transpose(0, 1).reshape(cb, -1)
    return at.T @ bt


def _download(s, psi, site, key):
    cl, d, cr = psi.site_dims(site)
    out = s[key]
    return psi.download_site(site, out) if out.shape == (d, cl, cr) else psi.site_array(site)


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind in ("gate", "canonize"):
        # the host program owns the state: both sites go in, the call runs, both sites come back
        psi = s["psi"]
        psi.upload_site(2, s["a"])
        psi.upload_site(3, s["b"])
        psi.set_lambda(1, s["lam"])
        if kind == "gate":
            Q.evolve_(psi, s["gate"], threshold=1e-10, maxdim=case["cb"])
        else:
            Q.canonize_site_(psi, 2 if case["direction"] == "right" else 3, case["direction"], method=case["method"])
        a, b = _download(s, psi, 2, "a_out"), _download(s, psi, 3, "b_out")
        if case.get("method") == "qr":
            return {"left": _to_gpu(a), "right": _to_gpu(b)}
        lam = psi.lambda_between(2, 3)
        return {"spectrum": lam, "state": _merged(a, lam, b)}
    if kind == "env":
        psi = s["psi"]
        if case["op"] == "norm":
            v = [Q.norm(psi)]
        elif case["op"] == "overlap":
            v = [Q.overlap(psi, s["phi"])]
        elif case["op"] == "mpo":
            v = [Q.mpo_expect(psi, s["mpo"])]
        else:
            v = [Q.expect(psi, o) for o in s["obs"]]
        v = np.array(v, dtype=np.complex128)
        return v.astype(np.complex64) if case["precision"] == "split" else v
    if kind == "chain":
        psi = Q.canonize(s["psi"])
        return {"norm": Q.norm(psi), "zz": np.array([Q.expect(psi, [o]) for o in s["obs"]]),
                "spectra": [psi.lambda_between(i, i + 1) for i in range(1, case["n"])]}
    if kind == "batch":
        with Batch(precision=case["precision"]) as bt:
            ids = [bt.add(r) for r in s["requests"]]
            bt.run()
            lams = [bt.lambda_on(i, b) for i, r in zip(ids, s["requests"]) for b in range(r.n - 1)]
            return {"values": np.concatenate([bt.values(i) for i in ids]),
                    "bonds": np.concatenate([bt.bond_dims(i) for i in ids]),
                    "spectra": np.concatenate([x for x in lams if x is not None])}
    psi = Q.zeros_chain(case["n"])
    psi.set_precision(case["precision"])
    for layer in s["layers"]:
        Q.evolve_layer_(psi, layer, threshold=1e-10, maxdim=case["chi"])
    return {"x": np.array([Q.expect(psi, [o]) for o in s["obs"]]), "bonds": np.array(psi.bond_dims()),
            "spectra": np.concatenate([psi.lambda_between(i, i + 1) for i in range(1, case["n"])])}


# ---- what a pass cannot do without --------------------------------------------------------------
def _svd_flops(m, n):
    m, n = max(m, n), min(m, n)
    return 4.0 * (4.0 * m * m * n + 8.0 * m * n * n + 9.0 * n ** 3)


def _gate_work(cl, cb, cr, keep):
    m, n = D * cl, D * cr
    flops = 8.0 * m * n * cb + 8.0 * m * n * D * D + _svd_flops(m, n)
    return flops, 16.0 * (m * cb + cb * n + (m + n) * keep) + 8.0 * (cb + keep)


def _circuit_work(n, depth, chi, nobs):
    """A brick wall on |0...0>: every gate at the bond sizes a light cone from a product state allows."""
    bd, flops, byts = [1] * (n - 1), 0.0, 0.0
    for layer in range(depth):
        for i in range(0 if layer % 2 == 0 else 1, n - 1, 2):
            cl, cr = (1 if i == 0 else bd[i - 1]), (1 if i == n - 2 else bd[i + 1])
            keep = min(chi, D * cl, D * cr)
            f, b = _gate_work(cl, bd[i], cr, keep)
            bd[i], flops, byts = keep, flops + f, byts + b
    ends = [1] + bd + [1]
    sweep = sum(8.0 * D * ends[i] * ends[i + 1] * (ends[i] + ends[i + 1]) for i in range(n))
    return flops + nobs * sweep, byts + 16.0 * D * sum(ends[i] * ends[i + 1] for i in range(n))


def work(case):
    kind = case["kind"]
    if kind == "gate":
        f, b = _gate_work(case["cl"], case["cb"], case["cr"], case["cb"])
        return {"flops": f, "bytes": b}
    if kind == "canonize":
        cl, cb, cr = case["cl"], case["cb"], case["cr"]
        near, far = (cl, cr) if case["direction"] == "right" else (cr, cl)
        m = D * near
        f = 8.0 * cb * cb * D * far
        f += _svd_flops(m, cb) if case["method"] == "svd" else 8.0 * (2.0 * m * cb * cb - 2.0 * cb ** 3 / 3.0) * 2.0
        return {"flops": f, "bytes": 2 * 16.0 * D * cb * (cl + cr)}
    if kind == "env":
        n, chi = case["n"], case["chi"]
        w = 5 if case["op"] == "mpo" else 1
        reps = case["strings"] if case["op"] == "expect" else 1
        chains = 2 if case["op"] == "overlap" else 1
        return {"flops": reps * 8.0 * w * 2 * D * float(chi) ** 3 * (n - 2), "bytes": chains * 16.0 * D * chi * chi * (n - 2) + 64.0}
    if kind == "chain":
        n, chi = case["n"], case["chi"]
        f = (n - 1) * (8.0 * 4 * chi ** 3 + _svd_flops(D * chi, chi)) + n * 8.0 * 2 * D * chi ** 3 * (n - 1)
        return {"flops": f, "bytes": 2 * 16.0 * D * chi * chi * n}
    if kind == "batch":
        f = b = 0.0
        n, depth = (8 + case["n_max"]) // 2, (3 + case["depth_max"]) // 2
        for k in range(case["requests"]):
            chi = 2 ** (4 + k % (case["chi_log2"] - 3))
            x, y = _circuit_work(n, depth, chi, 2)
            f, b = f + x, b + y
        return {"flops": f, "bytes": b}
    f, b = _circuit_work(case["n"], case["depth"], case["chi"], case["n"])
    return {"flops": f, "bytes": b}


# ---- the same results in plain numpy and torch, 64 bits -------------------------------------------
def _theta(a, lam, b):
    """(o, l, r) arrays -> theta[(l, o1), (o2, r)] with l (and o2) running fastest in their groups."""
    cl, cb, cr = a.shape[1], a.shape[2], b.shape[2]
    x = np.transpose(a, (1, 0, 2)).reshape(cl * D, cb) * lam[None, :]
    return (x @ np.transpose(b, (1, 0, 2)).reshape(cb, D * cr)).reshape(cl, D, D, cr)


def _apply(u, t):
    """A two-site gate on theta[l, o1, o2, r]."""
    return np.einsum("abcd,lcdr->labr", u.reshape(D, D, D, D), t, optimize=True)


def _as_matrix(t):
    """theta[l, o1, o2, r] in the order of _merged: rows (l, o) o fastest, columns (r, o) o fastest."""
    return np.transpose(t, (0, 1, 3, 2)).reshape(t.shape[0] * D, t.shape[3] * D)


def _split(t, threshold, maxdim):
    cl, cr = t.shape[0], t.shape[3]
    u, sv, vh = np.linalg.svd(t.reshape(cl * D, D * cr), full_matrices=False)
    keep = [k for k in range(min(len(sv), maxdim)) if sv[k] > threshold]
    return u[:, keep].reshape(cl, D, -1), sv[keep], vh[keep].reshape(-1, D, cr)


def _circuit(n, gates, chi, threshold):
    """Gates [(left site, 4 x 4)] on |0...0> -> (sites (l, o, r), {bond: Lambda})."""
    a = [np.array([1.0, 0.0], dtype=np.complex128).reshape(1, D, 1) for _ in range(n)]
    lam = {}
    for i, m in gates:
        x, y = a[i - 1], a[i]
        if i - 1 in lam:
            x = x * lam[i - 1][None, None, :]
        t = _apply(m, np.einsum("lar,rbs->labs", x, y, optimize=True))
        a[i - 1], lam[i - 1], a[i] = _split(t, threshold, chi)
    return a, lam


def _sweep(a, lam, ops, b=None):
    """<b| prod ops |a> of two chains of (l, o, r) sites sharing their Lambdas."""
    b = a if b is None else b
    e = np.ones((1, 1), dtype=np.complex128)
    for i in range(len(a)):
        x, y = a[i], b[i]
        if i - 1 in lam:
            x, y = x * lam[i - 1][:, None, None], y * lam[i - 1][:, None, None]
        if i + 1 in ops:
            x = np.einsum("ab,lbr->lar", ops[i + 1], x)
        t = np.tensordot(e, x, ([0], [0]))
        e = np.tensordot(t, y.conj(), ([0, 1], [0, 1]))
    return complex(e[0, 0])


def _env_exact(case, seed):
    n = case["n"]

    def lor(arrays):
        t = [x[:, None, :] if i == 0 else x[:, :, None] if i == n - 1 else x for i, x in enumerate(arrays)]
        return [torch.from_numpy(np.ascontiguousarray(np.transpose(x, (1, 0, 2)))).cuda() for x in t]

    ket = lor(_sites(case, seed))
    bra = ket
    if case["op"] == "overlap":
        bra = lor([x + 0.1 * y for x, y in zip(_sites(case, seed), _sites(case, seed + 7919))])
    if case["op"] == "mpo":
        mpo = R.xxz_mpo_arrays(n)
        ws = [x[:, :, None, :] if i == 0 else x[:, :, :, None] if i == n - 1 else x for i, x in enumerate(mpo)]
        sweeps = [[torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in ws]]
    else:
        strings = _strings(case, seed) if case["op"] == "expect" else [[]]
        sweeps = [[torch.from_numpy(R.PAULI[dict(o).get(i + 1, "I")]).cuda()[:, :, None, None] for i in range(n)]
                  for o in strings]
    out = []
    for ops in sweeps:
        e = torch.ones((1, 1, 1), dtype=torch.complex128, device="cuda")  # [w, a, b]
        for x, w, y in zip(ket, ops, bra):
            t = torch.einsum("wab,air->wbir", e, x)
            t = torch.einsum("oiwv,wbir->vrbo", w, t)
            e = torch.einsum("vrbo,bos->vrs", t, y.conj())
        out.append(complex(e[0, 0, 0].cpu()))
    if case["op"] == "norm":
        out = [math.sqrt(abs(out[0]))]
    return np.array(out, dtype=np.complex128)


def _chain_exact(case, seed):
    n = case["n"]
    a = [x[:, None, :] if i == 0 else x[:, :, None] if i == n - 1 else x for i, x in enumerate(_sites(case, seed))]
    a = [np.transpose(x, (1, 0, 2)) for x in a]
    norm = math.sqrt(abs(_sweep(a, {}, {})))
    zz = np.array([_sweep(a, {}, {i: R.PAULI["Z"], i + 1: R.PAULI["Z"]}) for i in range(1, n)])
    for i in range(n - 1, 0, -1):
        cl, _, cr = a[i].shape
        q, r = np.linalg.qr(a[i].reshape(cl, D * cr).T)
        a[i] = q.T.reshape(-1, D, cr)
        a[i - 1] = np.tensordot(a[i - 1], r, ([2], [1]))
    spectra = []
    for i in range(n - 1):
        cl, _, cr = a[i].shape
        _, sv, vh = np.linalg.svd(a[i].reshape(cl * D, cr), full_matrices=False)
        a[i + 1] = np.tensordot(vh * sv[:, None], a[i + 1], ([1], [0]))
        spectra.append(sv)
    return {"norm": norm, "zz": zz, "spectra": spectra}


def exact(case, seed):
    kind = case["kind"]
    if kind == "gate":
        a, b, lam, u = _pair(case, seed)
        x, sv, y = _split(_apply(u, _theta(a, lam, b)), 1e-10, case["cb"])
        return {"spectrum": sv, "state": _as_matrix(np.tensordot(x * sv, y, ([2], [0])))}
    if kind == "canonize":
        a, b, lam, _ = _pair(case, seed)
        if case["method"] == "svd":
            t = _theta(a, lam, b)
            near = np.transpose(a, (1, 0, 2)).reshape(-1, case["cb"]) if case["direction"] == "right" \
                else np.transpose(b, (1, 0, 2)).reshape(case["cb"], -1)
            return {"spectrum": np.linalg.svd(near, compute_uv=False), "state": _as_matrix(t)}
        cl, cb, cr = case["cl"], case["cb"], case["cr"]
        if case["direction"] == "right":  # rows (l, o) with l fastest
            q, r = np.linalg.qr(a.reshape(D * cl, cb))
            nxt = np.tensordot(r * lam, b, ([1], [1]))
            return {"left": q.reshape(D, cl, -1).T, "right": np.transpose(nxt, (2, 0, 1))}
        q, r = np.linalg.qr(np.transpose(b, (2, 0, 1)).reshape(cr * D, cb))  # rows (o, r), o fastest
        prv = np.tensordot(a * lam, r, ([2], [1]))
        return {"left": prv.T, "right": np.transpose(q.reshape(cr, D, -1), (0, 2, 1))}
    if kind == "env":
        return _env_exact(case, seed)
    if kind == "chain":
        return _chain_exact(case, seed)
    if kind == "batch":
        reqs = _requests(case, seed)
        vals, bonds, spectra = [], [], []
        for q in reqs:
            a, lam = _circuit(q.n, q.gates, q.chi_max, q.threshold)
            vals += [_sweep(a, lam, {i: R.PAULI[p] for i, p in o}) for o in q.observables]
            bonds += [x.shape[2] for x in a[:-1]]
            spectra += [lam[b] for b in range(q.n - 1) if b in lam]
        return {"values": np.array(vals), "bonds": np.array(bonds), "spectra": np.concatenate(spectra)}
    gates = [g for layer in R.brickwall_layers(case["n"], case["depth"], seed) for g in layer]
    a, lam = _circuit(case["n"], gates, case["chi"], 1e-10)
    return {"x": np.array([_sweep(a, lam, {i: R.PAULI["X"]}) for i in range(1, case["n"] + 1)]),
            "bonds": np.array([x.shape[2] for x in a[:-1]]),
            "spectra": np.concatenate([lam[b] for b in range(case["n"] - 1)])}
