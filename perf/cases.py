"""Performance cases of the MPS trajectory engine: what its users run, through its public entry points.

A case is a dict of plain values.  ``kind`` says which call it is:

  read        entropies and site probabilities of a resident state (the per-step observables)
  gate        one two-qubit gate on a bond of a branched state (clone + apply_unitary2)
  measure     one projective measurement with its full refactor sweep on a branched state (clone + measure_prob)
  trajectory  a whole single-state trajectory: new_qubits, then gates + measurements + entropy per layer
  batch       the first layers of a batch of trajectories from |0...0> (reset, then one step per layer)
  steady      one even and one odd layer of a batch that is already entangled
  serve       requests submitted to a resident server and drained
  coev        the multi-chi coevolution replay
  from_vector factorisation of a dense state

Entangled starting states are those of a monitored Haar brickwork circuit, simulated densely and cut into Schmidt form
here, so that spectra and ranks are those a trajectory meets.  Results are returned in float64, except in the MIXED mode,
whose state and arithmetic are complex64: there they are returned in float32, the precision that the mode has.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import __graft_entry__  # noqa: E402

P_CYCLE = (0.05, 0.10, 0.15, 0.20, 0.30)  # measurement probabilities of the benchmark's batch
SEED_SPAN = 1 << 30


def listed():
    return [
        # the observables read after each layer of a single trajectory: launch latency is everything
        dict(name="read_df", kind="read", n=16, chi=64, prec="df"),
        # the plain complex128 method on the system size of the reference's own timings (N=12), from |0...0>
        dict(name="trajectory_f64", kind="trajectory", n=12, chi=64, cutoff=1e-12, depth=12, p=0.1, prec="f64"),
        # the plain workload's N=16, chi=64 in the FP64-class mode: small and growing bonds, one state at a time
        dict(name="trajectory_df", kind="trajectory", n=16, chi=64, cutoff=1e-12, depth=10, p=0.1, prec="df"),
        # a gate on a saturated bond of the benchmark's chi_max=256: the operation that its layers are made of
        dict(name="gate_df_chi256", kind="gate", n=18, chi=256, cutoff=1e-10, prec="df"),
        # the same in single precision, as the large and batching workloads run it
        dict(name="gate_mixed_chi256", kind="gate", n=18, chi=256, cutoff=1e-10, prec="mixed"),
        # one measurement of a mid-size ragged state: the serial refactor sweep (odd n, chi no multiple of a tile)
        dict(name="measure_df", kind="measure", n=13, chi=50, cutoff=1e-10, prec="df"),
        # the benchmark's batch (N=64, chi_max=256, 304 trajectories, p cycling) over its first, growing layers
        dict(name="batch_df_n64", kind="batch", ntraj=304, n=64, chi=256, cutoff=1e-10, depth=5, prec="df"),
        # saturated layers of one trajectory per SM: gates, measurements and refactors at the bond capacity
        dict(name="steady_df_chi128", kind="steady", ntraj=152, n=16, chi=128, cutoff=1e-10, prec="df"),
        # the batching workload: 512 trajectories of mixed n, chi_max and p in one launch per layer
        dict(name="batch_mixed_512", kind="batch", ntraj=512, n=0, chi=0, cutoff=1e-10, depth=6, prec="mixed"),
        # light requests of the serving workload, served together
        dict(name="serve_df", kind="serve", requests=24, n_lo=16, n_hi=32, chi=32, depth=10, prec="df"),
        # the coevolution replay over the reference's chi_max values
        dict(name="coev_f64", kind="coev", n=10, depth=10, p=0.1, runs=4, prec="f64"),
        # a prepared dense state brought into Schmidt form
        dict(name="from_vector_n13", kind="from_vector", n=13, prec="df"),
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["read", "gate", "gate", "measure", "trajectory", "batch", "batch", "steady", "steady", "serve",
                       "coev", "from_vector"])
    prec = rng.choice(["df", "df", "df", "mixed", "f64"])
    if kind == "read":
        return dict(kind=kind, n=rng.randint(8, 17), chi=log_int(4, 128), prec=prec)
    if kind == "gate":
        return dict(kind=kind, n=rng.randint(13, 18), chi=log_int(16, 128 if prec == "f64" else 256), cutoff=1e-10,
                    prec=prec)
    if kind == "measure":
        return dict(kind=kind, n=rng.randint(8, 15), chi=log_int(6, 40 if prec == "f64" else 64), cutoff=1e-10,
                    prec=prec)
    if kind == "trajectory":
        return dict(kind=kind, n=rng.randint(5, 14), chi=log_int(4, 64), cutoff=1e-12, depth=rng.randint(4, 10),
                    p=round(rng.uniform(0.05, 0.3), 3), prec=prec)
    if kind == "batch":
        return dict(kind=kind, ntraj=log_int(8, 400), n=rng.randint(9, 64), chi=log_int(8, 256), cutoff=1e-10,
                    depth=rng.randint(2, 5), prec="df" if prec == "f64" else prec)
    if kind == "steady":
        return dict(kind=kind, ntraj=log_int(4, 300), n=rng.randint(10, 15), chi=log_int(8, 90), cutoff=1e-10,
                    prec="df" if prec == "f64" else prec)
    if kind == "serve":
        return dict(kind=kind, requests=log_int(4, 24), n_lo=8, n_hi=rng.randint(12, 32), chi=log_int(8, 32),
                    depth=rng.randint(4, 9), prec="df")
    if kind == "coev":
        return dict(kind=kind, n=rng.randint(6, 10), depth=rng.randint(4, 9), p=round(rng.uniform(0.05, 0.25), 3),
                    runs=rng.randint(1, 6), prec=rng.choice(["f64", "df"]))
    return dict(kind=kind, n=rng.randint(7, 13), prec=rng.choice(["f64", "df"]))


# ---------------------------------------------------------------- inputs
def haar(rng, count):
    """``count`` Haar-random U(4) gates: QR of Ginibre matrices with the phases of R's diagonal divided out."""
    z = rng.standard_normal((count, 4, 4)) + 1j * rng.standard_normal((count, 4, 4))
    q, r = np.linalg.qr(z)
    d = np.diagonal(r, axis1=1, axis2=2)
    return q * (d / np.abs(d))[:, None, :]


def layer(rng, n, t, p):
    """One brickwork layer: (gate sites, gates, measured sites, outcome uniforms)."""
    ks = np.arange(t % 2, n - 1, 2).astype(np.uint32)
    mk = np.flatnonzero(rng.random(n) < p).astype(np.uint32)
    return ks, haar(rng, ks.size), mk, rng.random(mk.size)


def dense_state(rng, n, depth, p, calm=7):
    """2^n amplitudes of a monitored brickwork circuit after ``depth`` layers (on the GPU when there is one), the last
    ``calm`` of them unmeasured: a chain this short would otherwise stop at ranks that a long one passes."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=dev)
    psi[0] = 1.0
    for t in range(depth):
        ks, gates, mk, us = layer(rng, n, t, p if t < depth - calm else 0.0)
        g = torch.from_numpy(gates).to(dev)
        for k, u4 in zip(ks, g):
            k = int(k)
            psi = torch.einsum("ab,vbw->vaw", u4, psi.view(1 << k, 4, -1)).reshape(-1)
        for k, u in zip(mk, us):
            v = psi.view(1 << int(k), 2, -1)
            p0 = float((v[:, 0].abs() ** 2).sum())
            s = 0 if u < p0 else 1
            w = torch.zeros_like(v)
            w[:, s] = v[:, s]
            psi = (w / math.sqrt(p0 if s == 0 else 1.0 - p0)).reshape(-1)
    return psi.cpu().numpy()


def schmidt_form(psi, n, chi, cutoff):
    """(gammas, lambdas) of a dense state, left to right, ranks cut to chi and to values above cutoff."""
    gammas, lams = [], []
    q = psi.reshape(1, -1) / np.linalg.norm(psi)
    left = np.ones(1)
    for k in range(n - 1):
        u, s, vh = np.linalg.svd(q.reshape(2 * left.size, -1), full_matrices=False)
        s = s / np.linalg.norm(s)
        r = max(1, min(chi, int(np.sum(s > cutoff))))
        s = s[:r] / np.linalg.norm(s[:r])
        gammas.append(u[:, :r].reshape(left.size, 2, r) / left[:, None, None])
        lams.append(s)
        q = vh[:r] * s[:, None]
        left = s
    gammas.append(q.reshape(left.size, 2, 1) / left[:, None, None])
    return gammas, lams


def entangled(rng, n, chi, cutoff=1e-10):
    return schmidt_form(dense_state(rng, n, n + 2, 0.05), n, chi, cutoff)


def mix(case, rng):
    """(n, chi, p) of every trajectory of a batch: the case's own, p cycling, or (n = 0) the mixed workload's draw."""
    if case["n"]:
        return [(case["n"], case["chi"], P_CYCLE[i % len(P_CYCLE)]) for i in range(case["ntraj"])]
    return [(int(rng.choice([16, 32, 48, 64])), int(rng.choice([32, 64, 128, 256])), float(rng.uniform(0.05, 0.3)))
            for _ in range(case["ntraj"])]


def inputs(case, seed):
    """Everything random of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 0x6D7073])
    k = case["kind"]
    if k == "read":
        return dict(state=entangled(rng, case["n"], case["chi"]))
    if k == "gate":
        return dict(state=entangled(rng, case["n"], case["chi"], case["cutoff"]), gate=haar(rng, 1)[0])
    if k == "measure":
        return dict(state=entangled(rng, case["n"], case["chi"], case["cutoff"]), u=float(rng.random()))
    if k == "trajectory":
        return dict(layers=[layer(rng, case["n"], t, case["p"]) for t in range(case["depth"])])
    if k == "batch":
        specs = mix(case, rng)
        return dict(specs=specs, layers=[[layer(rng, n, t, p) for (n, _, p) in specs] for t in range(case["depth"])])
    if k == "steady":
        specs = mix(case, rng)
        return dict(specs=specs, states=[entangled(rng, case["n"], case["chi"], case["cutoff"]) for _ in range(2)],
                    layers=[[layer(rng, n, t, p) for (n, _, p) in specs] for t in range(2)])
    if k == "serve":
        return dict(seed=int(rng.integers(SEED_SPAN)),
                    reqs=[(int(rng.integers(case["n_lo"], case["n_hi"] + 1)), float(rng.uniform(0.02, 0.3)))
                          for _ in range(case["requests"])])
    if k == "coev":
        return dict(layers=[layer(rng, case["n"], t, case["p"])[:3] for t in range(case["depth"])],
                    seed=int(rng.integers(SEED_SPAN)))
    return dict(psi=dense_state(rng, case["n"], case["n"], 0.05))


# ---------------------------------------------------------------- the calls
class State:
    pass


def prepare(case, seed):
    pkg = __graft_entry__.load_package()
    s = State()
    s.case, s.pkg, s.x = case, pkg, inputs(case, seed)
    k, x, prec = case["kind"], s.x, case["prec"]
    if k in ("read", "gate", "measure"):
        s.trunc = pkg.Trunc.both(case["chi"], case.get("cutoff", 1e-10))
        s.mps = pkg.MPS.from_parts(*x["state"], s.trunc, prec)
    elif k == "batch" or k == "steady":
        s.truncs = [pkg.Trunc.both(c, case["cutoff"]) for (_, c, _) in x["specs"]]
        s.ns = [n for (n, _, _) in x["specs"]]
        s.batch = pkg.Batch(s.ns, s.truncs, prec)
        s.ids = list(range(len(s.ns)))
        s.packed = [pkg.Batch.pack(s.ids, la) for la in x["layers"]]
        if k == "steady":
            for i in s.ids:
                s.batch.import_state(i, *x["states"][i % len(x["states"])], s.truncs[i])
    elif k == "serve":
        s.server = pkg.Server(1 << 32, max_slots=64, precision=prec, max_chi=64, max_n=64)
    return s


def typed(case, x):
    """An array of results in the mode's own precision."""
    return np.asarray(x, np.float32 if case["prec"] == "mixed" else np.float64)


def padded(v, shape):
    """v in the corner of an array of zeros: ranks differ from state to state, the shape of the results does not."""
    out = np.zeros(shape)
    out[tuple(slice(0, d) for d in v.shape)] = v
    return out


def records(n, layers, rec):
    """Outcomes (-1 where a site is not measured) and probabilities of a trajectory as (layer, site) arrays."""
    at = np.concatenate([t * n + np.asarray(la[2], np.int64) for t, la in enumerate(layers)])
    oc, pr = np.full(len(layers) * n, -1, np.int32), np.zeros(len(layers) * n)
    oc[at], pr[at] = [r[0] for r in rec], [r[1] for r in rec]
    return oc.reshape(-1, n), pr.reshape(-1, n)


def spectra(m, n, width):
    """Schmidt values of every bond, zeros beyond each bond's rank."""
    out = np.zeros((n - 1, width))
    for b in range(n - 1):
        v = m.svals(b)
        out[b, :v.size] = v
    return out


def gate_output(case, lam_l, g0, lam_m, g1, lam_r):
    """The bond after a gate without the free phases of its Schmidt vectors: its Schmidt values and the squared
    moduli of both tensors weighted with the Lambdas beside them.  Single precision does not resolve the vectors of
    neighbouring Schmidt values, so MIXED returns their populations on the outer indices, which it does resolve."""
    w0 = np.abs(g0) ** 2 * (lam_l ** 2)[:, None, None] * lam_m ** 2
    w1 = np.abs(g1) ** 2 * (lam_m ** 2)[:, None, None] * lam_r ** 2
    x = case["chi"]
    out = [padded(lam_m, (x,)), padded(w0, (x, 2, x)), padded(w1, (x, 2, x))]
    if case["prec"] == "mixed":
        out[1:] = [out[1].sum(2), out[2].sum(0)]
    return out


def steps(case, x, recs):
    """Outputs of the steps of a batch, a row per layer: the first two trajectories by themselves (p = 0.05 and 0.10
    where p cycles), the others together.  recs: per step (outcomes, probs, entropies)."""
    width, nt = max(n for (n, _, _) in x["specs"]), len(x["specs"])
    oc = np.full((len(recs), nt * width), -1, np.int32)
    pr = np.zeros((len(recs), nt * width))
    for t, (la, rec) in enumerate(zip(x["layers"], recs)):
        at = np.concatenate([i * width + mk.astype(np.int64) for i, (_, _, mk, _) in enumerate(la)])
        oc[t, at], pr[t, at] = rec[0], rec[1]
    en = np.array([rec[2] for rec in recs])
    cuts = [0] + [i for i in (1, 2) if i < nt] + [nt]
    return dict(outcomes=[oc[:, a * width:b * width] for a, b in zip(cuts, cuts[1:])],
                probs=[typed(case, pr[:, a * width:b * width]) for a, b in zip(cuts, cuts[1:])],
                entropies=[typed(case, en[:, a:b]) for a, b in zip(cuts, cuts[1:])])


def run(s):
    case, pkg, x = s.case, s.pkg, s.x
    kind, n, prec = case["kind"], case.get("n", 0), case["prec"]
    if kind == "read":
        b = n // 2 - 1
        return typed(case, [s.mps.entropy_vn(b), s.mps.entropy_ry_schmidt(2.0, b), *s.mps.probs(n // 2)])
    if kind == "gate":
        m, k = s.mps.clone(), n // 2 - 1
        m.apply_unitary2(k, x["gate"])
        out = gate_output(case, m.svals(k - 1), m.gamma(k), m.svals(k), m.gamma(k + 1), m.svals(k + 1))
        m.close()
        return [typed(case, v) for v in out]
    if kind == "measure":
        m = s.mps.clone()
        oc, pr = m.measure_prob(n // 2, x["u"])
        out = [oc, typed(case, [pr]), typed(case, spectra(m, n, case["chi"])),
               typed(case, [m.probs(k) for k in range(n)])]
        m.close()
        return out
    if kind == "trajectory":
        m = pkg.MPS.new_qubits(n, pkg.Trunc.both(case["chi"], case["cutoff"]), prec)
        rec, ent = [], []
        for (gk, g, mk, us) in x["layers"]:
            rec += m.apply_bilayer(gk, g, mk, us)
            ent.append(m.entropy_vn(n // 2 - 1))
        oc, pr = records(n, x["layers"], [r[1:] for r in rec])
        out = [oc, typed(case, pr), typed(case, ent), typed(case, spectra(m, n, case["chi"])),
               typed(case, [m.probs(k) for k in range(n)])]
        m.close()
        return out
    if kind == "batch" or kind == "steady":
        if kind == "batch":
            for i in s.ids:
                s.batch.reset(i, s.ns[i], s.truncs[i])
        return steps(case, x, [s.batch.step_packed(pk) for pk in s.packed])
    if kind == "serve":
        ids = [s.server.submit(rn, pkg.Trunc.both(case["chi"], 1e-10), p, case["depth"], x["seed"], i)
               for i, (rn, p) in enumerate(x["reqs"])]
        got = {}
        while len(got) < len(ids):
            s.server.tick()
            for d in s.server.poll(history=True):
                got[d["id"]] = d["entropies"]
        return typed(case, [got[i] for i in ids])
    if kind == "coev":
        r = pkg.run_coevolution_layers(n, x["layers"], case["runs"], x["seed"], precision=prec)
        at = r["sites"][:, 0] * n + r["sites"][:, 1]
        oc = np.full((case["runs"], case["depth"] * n), -1, np.int32)
        pr = np.zeros((*r["probs"].shape[:2], case["depth"] * n))
        oc[:, at], pr[:, :, at] = r["outcomes"], r["probs"]
        return [oc, pr]
    m = pkg.MPS.from_vector(x["psi"], None, prec)
    out = [spectra(m, n, 1 << (n // 2)), np.array([m.probs(k) for k in range(n)])]
    m.close()
    return out


# ---------------------------------------------------------------- work
def op_work(cl, cm, cr, eb):
    """Flops of one bond operation (theta contraction + the Golub-Reinsch count of a complex SVD with both sides)
    and the bytes of its two tensors, read and written."""
    a, b = max(2 * cl, 2 * cr), min(2 * cl, 2 * cr)
    return (8.0 * 2 * cl * cm * 2 * cr + 4.0 * (4.0 * a * a * b + 8.0 * a * b * b + 9.0 * b ** 3),
            2.0 * eb * (2 * cl * cm + 2 * cm * cr))


def work(case):
    kind, eb = case["kind"], 8 if case["prec"] == "mixed" else 16
    n, chi = case.get("n", 0), case.get("chi", 0)

    def full(n, chi, t=None):
        """Bond dimensions, chain ends included, saturated or after t layers from |0...0>."""
        return [min(2 ** min(i, n - i, 40), chi, 2 ** (t if t is not None else 40)) for i in range(n + 1)]

    def layer_work(n, dims, p, t):
        flops = nbytes = 0.0
        ops = list(range(t % 2, n - 1, 2))
        if p * n >= 0.5:  # a measured layer refactors nearly every bond on the way right and on the way back
            ops += list(range(n - 1)) + list(range(n - 2))
        for k in ops:
            f, b = op_work(dims[k], dims[k + 1], dims[k + 2], eb)
            flops, nbytes = flops + f, nbytes + b
        return flops, nbytes

    if kind == "read":
        d = full(n, chi)
        return dict(bytes=8.0 * 4 * d[n // 2] + eb * 2.0 * d[n // 2] * d[n // 2 + 1], flops=16.0 * d[n // 2] ** 2)
    if kind == "gate":
        d, k = full(n, chi), n // 2 - 1
        f, b = op_work(d[k], d[k + 1], d[k + 2], eb)
        return dict(bytes=b, flops=f)
    if kind == "measure":
        f, b = layer_work(n, full(n, chi), 1.0, n)
        return dict(bytes=b, flops=f)
    if kind in ("trajectory", "batch"):
        specs = [(n, chi, case["p"])] if kind == "trajectory" else mix(case, np.random.default_rng(1))
        f = b = 0.0
        for (m, c, p) in specs:
            for t in range(case["depth"]):
                lf, lb = layer_work(m, full(m, c, t + 1), p, t)
                f, b = f + lf, b + lb
        return dict(bytes=b, flops=f)
    if kind == "steady":
        f = b = 0.0
        for t in range(2):
            lf, lb = layer_work(n, full(n, chi), 1.0, t)
            f, b = f + lf, b + lb
        return dict(bytes=b * case["ntraj"], flops=f * case["ntraj"])
    if kind == "serve":
        m = (case["n_lo"] + case["n_hi"]) // 2
        f = b = 0.0
        for t in range(case["depth"]):
            lf, lb = layer_work(m, full(m, chi, t + 1), 0.16, t)
            f, b = f + lf, b + lb
        return dict(bytes=b * case["requests"], flops=f * case["requests"])
    if kind == "coev":
        f = b = 0.0
        for c in (4, 8, 12, 16, 20, 24, 28, 32, 36, 40, 44, 48, 56, 64, 72, 1 << 20):
            for t in range(case["depth"]):
                lf, lb = layer_work(n, full(n, c, t + 1), case["p"], t)
                f, b = f + lf, b + lb
        return dict(bytes=b * case["runs"], flops=f * case["runs"])
    f = 0.0
    for k in range(n - 1):
        m, q = 2 ** min(k + 1, n - k), 2 ** (n - k - 1)
        a, c = max(m, q), min(m, q)
        f += 4.0 * (4.0 * a * c * c + 22.0 * c ** 3)
    return dict(bytes=16.0 * 2 ** n * 3, flops=f)


# ---------------------------------------------------------------- 64-bit values
class Plain:
    """Schmidt-form MPS in plain complex128 numpy: the textbook update of each call."""

    def __init__(self, n, chi, cutoff, state=None):
        self.n, self.chi, self.cutoff = n, chi, cutoff
        if state is None:
            self.g = [np.zeros((1, 2, 1), complex) for _ in range(n)]
            for g in self.g:
                g[0, 0, 0] = 1.0
            self.lam = [np.ones(1) for _ in range(n - 1)]
        else:
            self.g, self.lam = [g.copy() for g in state[0]], [x.copy() for x in state[1]]

    def left(self, k):
        return self.lam[k - 1] if k else np.ones(1)

    def right(self, k):
        return self.lam[k] if k < self.n - 1 else np.ones(1)

    def bond(self, k, gate=None):
        l, r = self.left(k), self.right(k + 1)
        a = (self.g[k] * l[:, None, None] * self.lam[k]).reshape(2 * l.size, -1)
        b = (self.g[k + 1] * r).reshape(-1, 2 * r.size)
        th = (a @ b).reshape(l.size, 4, r.size)
        if gate is not None:
            th = np.einsum("ab,vbw->vaw", gate, th)
        u, s, vh = np.linalg.svd(th.reshape(2 * l.size, 2 * r.size), full_matrices=False)
        s = s / np.linalg.norm(s)
        c = max(1, min(self.chi, int(np.sum(s > self.cutoff))))
        s = s[:c] / np.linalg.norm(s[:c])
        self.g[k] = u[:, :c].reshape(l.size, 2, c) / l[:, None, None]
        self.g[k + 1] = vh[:c].reshape(c, 2, r.size) / r
        self.lam[k] = s
        for i in (k, k + 1):
            self.g[i] = self.g[i] / math.sqrt(self.probs(i).sum())

    def probs(self, k):
        w = np.abs(self.g[k]) ** 2 * (self.left(k) ** 2)[:, None, None] * self.right(k) ** 2
        return w.sum(axis=(0, 2))

    def project(self, k, u):
        p = self.probs(k)
        s = 0 if u < p[0] else 1
        self.g[k][:, 1 - s] = 0.0
        self.g[k] = self.g[k] / math.sqrt(p[s])
        return s, float(p[s])

    def bilayer(self, gk, gates, mk, us):
        for k, g in zip(gk, gates):
            self.bond(int(k), g)
        rec, last = [], None
        for k, u in zip(mk, us):
            for b in range(last, int(k)) if last is not None else ():
                self.bond(b)
            rec.append(self.project(int(k), u))
            last = int(k)
        if last is not None:
            for b in [*range(last, self.n - 1), *range(self.n - 3, -1, -1)]:
                self.bond(b)
        return rec

    def entropy(self, b):
        s2 = self.lam[b] ** 2
        return float(-(s2 * np.log(s2)).sum())

    def spectra(self, width):
        out = np.zeros((self.n - 1, width))
        for b, v in enumerate(self.lam):
            out[b, :v.size] = v
        return out

    def all_probs(self):
        return np.array([self.probs(k) for k in range(self.n)])


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("serve", "coev"):
        return None
    x = inputs(case, seed)
    if kind == "read":
        m, b = Plain(n, case["chi"], 1e-10, x["state"]), n // 2 - 1
        return np.array([m.entropy(b), -math.log((m.lam[b] ** 4).sum()), *m.probs(n // 2)])
    if kind == "gate":
        m, k = Plain(n, case["chi"], case["cutoff"], x["state"]), n // 2 - 1
        m.bond(k, x["gate"])
        return gate_output(case, m.left(k), m.g[k], m.lam[k], m.g[k + 1], m.right(k + 1))
    if kind == "measure":
        m = Plain(n, case["chi"], case["cutoff"], x["state"])
        _, pr = m.project(n // 2, x["u"])
        for b in [*range(n - 1), *range(n - 3, -1, -1)]:
            m.bond(b)
        return [None, np.array([pr]), m.spectra(case["chi"]), m.all_probs()]
    if kind == "trajectory":
        m, rec, ent = Plain(n, case["chi"], case["cutoff"]), [], []
        for la in x["layers"]:
            rec += m.bilayer(*la)
            ent.append(m.entropy(n // 2 - 1))
        return [None, records(n, x["layers"], rec)[1], np.array(ent), m.spectra(case["chi"]), m.all_probs()]
    if kind == "from_vector":
        m = Plain(n, 1 << n, 0.0, schmidt_form(x["psi"], n, 1 << n, 1e-15))
        return [m.spectra(1 << (n // 2)), m.all_probs()]
    out, width = {"outcomes": [], "probs": [], "entropies": []}, max(n for (n, _, _) in x["specs"])
    for i, (m_n, chi, _) in enumerate(x["specs"][:2]):
        m, rec, ent = Plain(m_n, chi, case["cutoff"], x["states"][i % 2] if kind == "steady" else None), [], []
        for la in x["layers"]:
            rec += m.bilayer(*la[i])
            ent.append(m.entropy(m_n // 2 - 1))
        out["outcomes"].append(None)
        pr = np.zeros((len(ent), width))
        pr[np.concatenate([[t] * la[i][2].size for t, la in enumerate(x["layers"])]).astype(int),
           np.concatenate([la[i][2] for la in x["layers"]]).astype(int)] = [p for _, p in rec]
        out["probs"].append(pr)
        out["entropies"].append(np.array(ent).reshape(-1, 1))
    if len(x["specs"]) > 2:
        for v in out.values():
            v.append(None)
    return out
