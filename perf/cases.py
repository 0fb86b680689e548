"""The framework's work, measured: sigma (the Hamiltonian matvec) on device and
host buffers, block sigma, the Davidson projections, the set-up of a
Hamiltonian, and whole solves, each through the public entry points.

Sizes are the repository's own: L=32, N=16 (601,080,390 determinants) is the
headline sigma, L=28, N=14 the solver benchmark, L in 16..30 with N = L/2 +- 2
the served requests, L in 12..24 with four roots the batch, and L=13, N=5 the
H2O / 6-31G test molecule.  Integrals follow the benchmark's synthetic model,
seeded.  Vectors look like the solver's: components fall off with the number of
pairs excited out of the lowest determinant.
"""
import ctypes
import math

import numpy as np
import torch

import doci_gb300 as dg

DECAY = 0.25  # size of a component per pair excited out of the lowest determinant


def listed():
    return [
        # the headline workload: the FP32 sigma of a mixed-precision solve, at the largest space
        {"name": "sigma_f32_L32_N16", "path": "sigma", "L": 32, "N": 16, "prec": "f32"},
        # the sigma of the FP64 Davidson and CG runs of the solver benchmark
        {"name": "sigma_f64_L28_N14", "path": "sigma", "L": 28, "N": 14, "prec": "f64"},
        # a served request away from half filling, odd in L and N
        {"name": "sigma_f32_L27_N11", "path": "sigma", "L": 27, "N": 11, "prec": "f32"},
        # an ordinary FP64 sigma, odd in L and N
        {"name": "sigma_f64_L23_N9", "path": "sigma", "L": 23, "N": 9, "prec": "f64"},
        # a small active space: a few microseconds, the launches count
        {"name": "sigma_f32_L18_N9", "path": "sigma", "L": 18, "N": 9, "prec": "f32"},
        # the smallest calls: a water molecule in a small basis
        {"name": "sigma_f64_L13_N5", "path": "sigma", "L": 13, "N": 5, "prec": "f64"},
        # the drop-in matvec of a host program: host vectors in and out of one call
        {"name": "host_f64_L26_N13", "path": "host", "L": 26, "N": 13, "prec": "f64"},
        # several vectors at once, as a block method asks for them
        {"name": "block_f32_L24_N12_nv4", "path": "block", "L": 24, "N": 12, "prec": "f32", "nv": 4},
        # subspace column / Gram-Schmidt projections of a caller's own Davidson
        {"name": "multidot_f32_m16_L28", "path": "multidot", "n": 40116600, "m": 16, "prec": "f32"},
        # set-up that every user and every served request pays: integrals to tables and diagonal
        {"name": "build_L24_N12", "path": "build", "L": 24, "N": 12},
        # a whole ground-state solve
        {"name": "solve_L22_N8", "path": "solve", "L": 22, "N": 8, "mode": "fp64"},
        # many small Hamiltonians, four roots each, in one call
        {"name": "batch_12_L12-18_r4", "path": "batch", "count": 12, "lmin": 12, "lmax": 18, "roots": 4},
    ]


def draw(rng):
    def dims(lo, hi):
        L = rng.randint(lo, hi)
        return L, max(1, min(L - 1, L // 2 + rng.randint(-3, 3)))

    path = rng.choice(["sigma"] * 6 + ["host", "block", "multidot", "build", "solve", "batch"])
    prec = rng.choice(["f32", "f64"])
    if path == "sigma":
        L, N = dims(12, 31 if prec == "f32" else 29)
        return {"path": path, "L": L, "N": N, "prec": prec}
    if path == "host":
        L, N = dims(12, 27)
        return {"path": path, "L": L, "N": N, "prec": prec}
    if path == "block":
        L, N = dims(12, 25 if prec == "f32" else 24)
        return {"path": path, "L": L, "N": N, "prec": prec, "nv": rng.randint(2, 8)}
    if path == "multidot":
        n = int(math.exp(rng.uniform(math.log(1e3), math.log(4e7)))) | 1
        return {"path": path, "n": n, "m": rng.randint(1, 32), "prec": prec}
    if path == "build":
        L, N = dims(10, 26)
        return {"path": path, "L": L, "N": N}
    if path == "solve":
        L, N = dims(12, 20)
        return {"path": path, "L": L, "N": N, "mode": "fp64"}
    lo = rng.randint(10, 14)
    return {"path": path, "count": rng.randint(4, 12), "lmin": lo, "lmax": lo + rng.randint(2, 4), "roots": rng.randint(2, 4)}


# ------------------------------------------------------------------ inputs
def integrals(L, seed):
    """One- and two-electron integrals of the benchmark's model: h symmetric
    with sorted diagonal, (ij|kl) a sum of squares, both whole."""
    rng = np.random.default_rng([seed, L])
    h = rng.normal(0.0, 0.05, (L, L))
    h = np.triu(h, 1)
    h = h + h.T
    h[np.diag_indices(L)] = np.sort(rng.uniform(-2.0, 0.5, L))
    B = np.triu(rng.normal(0.0, 0.1, (2 * L, L, L)))
    B = (B + np.transpose(np.triu(B, 1), (0, 2, 1))).reshape(2 * L, L * L)
    return h, (B.T @ B).reshape(L, L, L, L)


def hamiltonian(L, N, seed):
    h, eri = integrals(L, seed)
    return dg.Hamiltonian.from_integrals(L, N, 0.0, h, eri)


def type_of(case):
    return torch.float32 if case["prec"] == "f32" else torch.float64


def number(case):
    return dg.FP32 if case["prec"] == "f32" else dg.FP64


def vectors(bits, L, N, nv, dtype, seed):
    """nv vectors over the determinants with these bitstrings (orbital o at bit
    o; the lowest determinant fills orbitals 0..N-1)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    level = torch.zeros_like(bits)
    for o in range(N, L):
        level += (bits >> o) & 1
    scale = torch.tensor([DECAY ** k for k in range(L + 1)], dtype=dtype, device="cuda")[level]
    return torch.stack([torch.randn(bits.numel(), dtype=dtype, device="cuda", generator=g) * scale for _ in range(nv)])


def rows(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, m, t = case["n"], case["m"], type_of(case)
    V = torch.randn((m, n), dtype=t, device="cuda", generator=g) / math.sqrt(n)
    # the vector projected is not orthogonal to the basis: part of it lies in the basis' span
    w = torch.randn(n, dtype=t, device="cuda", generator=g) / math.sqrt(n) + V.sum(0) / m
    return V, w


def batch_dims(case):
    span = case["lmax"] - case["lmin"] + 1
    return [(case["lmin"] + k % span, (case["lmin"] + k % span) // 2) for k in range(case["count"])]


def prepare(case, seed):
    path = case["path"]
    if path == "multidot":
        V, w = rows(case, seed)
        return {"case": case, "V": V, "w": w, "out": torch.empty(case["m"], dtype=torch.float64, device="cuda")}
    if path == "batch":
        return {"case": case, "hams": [hamiltonian(L, N, seed + 1000 * k) for k, (L, N) in enumerate(batch_dims(case))]}
    L, N = case["L"], case["N"]
    if path == "build":
        return {"case": case, "integrals": integrals(L, seed)}
    h = hamiltonian(L, N, seed)
    if path == "solve":
        return {"case": case, "h": h}
    nv = case.get("nv", 1)
    bits = torch.empty(h.D, dtype=torch.int32, device="cuda")
    h.bitstrings_device(0, h.D, bits.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    x = vectors(bits, L, N, nv, type_of(case), seed)
    if path == "host":
        x = x[0].cpu().pin_memory()
        return {"case": case, "h": h, "x": x, "y": torch.empty_like(x).pin_memory()}
    return {"case": case, "h": h, "x": x, "y": torch.empty_like(x)}


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    path = case["path"]
    if path == "build":
        with dg.Hamiltonian.from_integrals(case["L"], case["N"], 0.0, *state["integrals"]) as h:
            return h.diagonal()
    if path == "solve":
        res, vec = state["h"].solve(solver="D", mode=case["mode"], tol=1e-10, max_its=300, davidson_max_vec=16)
        # an eigenvector is given up to its sign: the lowest determinant's component is made positive
        return {"energy": res["energy"], "vector": vec if vec[0] >= 0 else -vec}
    if path == "batch":
        _, res = dg.batch_solve(state["hams"], nroots=case["roots"], mode="mixed", tol=1e-6, mixed_tol=1e-5, max_vec=32)
        return [np.array(r["energies"]) for r in res]
    stream = torch.cuda.current_stream().cuda_stream
    if path == "multidot":
        V, w, out = state["V"], state["w"], state["out"]
        st = dg.lib().doci_multidot(V.data_ptr(), V.shape[1], V.shape[0], w.data_ptr(), w.numel(), number(case),
                                    out.data_ptr(), stream)
        if st:
            raise dg.DociError(st, "doci_multidot")
        return out
    h, x, y = state["h"], state["x"], state["y"]
    if path == "host":
        st = dg.lib().doci_sigma_host(h.handle, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()), number(case))
        if st:
            raise dg.DociError(st, "doci_sigma_host")
    elif path == "block":
        h.sigma_block_device(x.data_ptr(), h.D, y.data_ptr(), h.D, x.shape[0], number(case), stream=stream)
    else:
        h.sigma_device(x.data_ptr(), y.data_ptr(), number(case), stream=stream)
    return y


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    path = case["path"]
    e = 4 if case.get("prec") == "f32" else 8
    if path == "multidot":
        return {"bytes": case["n"] * (case["m"] + 1) * e, "flops": 2 * case["n"] * case["m"]}
    if path == "batch":
        # 20 block iterations, each one sigma and one pass over half a basis and its sigmas
        dets = [(math.comb(L, N), N * (L - N)) for L, N in batch_dims(case)]
        r = case["roots"]
        return {"bytes": sum(20 * D * 4 * (3 * r + 32) for D, _ in dets), "flops": sum(20 * D * r * (2 * k + 64) for D, k in dets)}
    L, N = case["L"], case["N"]
    D, hops = math.comb(L, N), N * (L - N)
    if path == "build":
        return {"bytes": D * 12, "flops": D * N * L}
    if path == "solve":
        # 30 iterations, each one sigma and one pass over half a basis of 16 and its sigmas
        return {"bytes": 30 * D * 8 * (3 + 16), "flops": 30 * D * (2 * hops + 64)}
    nv = case.get("nv", 1)
    return {"bytes": D * e * (2 * nv + 1), "flops": D * nv * (2 * hops + 1)}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch
def determinants(L, N):
    """Bitstrings in rank order (decreasing value of the mirrored string) and the mirrored strings, ascending."""
    parts = []
    for first in range(0, 1 << L, 1 << 26):
        v = torch.arange(first, min(first + (1 << 26), 1 << L), dtype=torch.int64, device="cuda")
        c = torch.zeros_like(v, dtype=torch.int8)
        for o in range(L):
            c += ((v >> o) & 1).to(torch.int8)
        parts.append(v[c == N])
    return torch.cat(parts)


def plain_bits(M, L):
    """Orbital o at bit o, in rank order, from the mirrored strings (ascending)."""
    bits = torch.zeros(M.numel(), dtype=torch.int32, device="cuda")
    for o in range(L):
        b = ((M >> (L - 1 - o)) & 1) << o
        bits |= b.to(torch.int32)
    return bits.flip(0)


def diagonal(M, L, h, eri):
    """Diagonal over the mirrored strings: 2 h_ii over the pairs, 2 (ii|jj) - (ij|ij) over pairs of pairs."""
    W = 2 * np.einsum("iijj->ij", eri) - np.einsum("ijij->ij", eri)
    h1 = torch.from_numpy(2 * np.diag(h).copy()).cuda()
    W = torch.from_numpy(W.copy()).cuda()
    out = torch.empty(M.numel(), dtype=torch.float64, device="cuda")
    shifts = torch.tensor([L - 1 - o for o in range(L)], device="cuda")
    for a in range(0, M.numel(), 1 << 22):
        n = ((M[a:a + (1 << 22), None] >> shifts) & 1).to(torch.float64)
        out[a:a + (1 << 22)] = n @ h1 + ((n @ W) * n).sum(1)
    return out


class Plain:
    """H over the mirrored strings, ascending: diag x plus the pair hops (ia|ia)."""

    def __init__(self, L, N, seed):
        h, eri = integrals(L, seed)
        self.L, self.N, self.M = L, N, determinants(L, N)
        self.diag = diagonal(self.M, L, h, eri)
        self.K = np.einsum("iaia->ia", eri)
        self.at = torch.zeros(1 << L, dtype=torch.int32, device="cuda")
        self.at[self.M] = torch.arange(self.M.numel(), dtype=torch.int32, device="cuda")

    def apply(self, x):
        y = self.diag * x
        for i in range(self.L):
            for a in range(i):
                p, q = self.L - 1 - i, self.L - 1 - a
                hop = ((self.M >> p) ^ (self.M >> q)) & 1
                y += (float(self.K[i, a]) * hop.to(x.dtype)) * x[self.at[self.M ^ ((1 << p) | (1 << q))].long()]
        return y

    def lowest(self, roots, steps):
        """Lanczos with full reorthogonalisation from the lowest determinants: the lowest pairs."""
        D = self.M.numel()
        steps = min(steps, D)
        hop = torch.empty((D, self.N * (self.L - self.N)), dtype=torch.int64, device="cuda")
        val = torch.empty(hop.shape, dtype=torch.float64, device="cuda")
        bit = ((self.M[:, None] >> torch.arange(self.L, device="cuda")) & 1).bool()
        occ = bit.nonzero()[:, 1].reshape(D, self.N)
        emp = (~bit).nonzero()[:, 1].reshape(D, self.L - self.N)
        K = torch.from_numpy(self.K[::-1, ::-1].copy()).cuda()  # by mirrored orbital
        for k in range(self.N):
            s = slice(k * (self.L - self.N), (k + 1) * (self.L - self.N))
            hop[:, s] = self.at[(self.M ^ (1 << occ[:, k]))[:, None] | (1 << emp)].long()
            val[:, s] = K[occ[:, k][:, None], emp]
        V = torch.zeros((steps, D), dtype=torch.float64, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(1)
        v = torch.exp(-3 * (self.diag - self.diag.min())) * (1 + torch.rand(D, dtype=torch.float64, device="cuda", generator=g))
        T = torch.zeros((steps, steps), dtype=torch.float64)
        V[0] = v / v.norm()
        for k in range(steps):
            w = self.diag * V[k] + (val * V[k][hop]).sum(1)
            c = V[:k + 1] @ w
            T[k, k] = c[k]
            for _ in range(2):
                w = w - V[:k + 1].T @ (V[:k + 1] @ w)
            if k + 1 < steps:
                b = w.norm()
                if b < 1e-11:
                    T = T[:k + 1, :k + 1]
                    break
                T[k, k + 1] = T[k + 1, k] = b
                V[k + 1] = w / b
        e, Y = torch.linalg.eigh(T)
        vec = (Y[:, 0].cuda() @ V[:T.shape[0]])
        return e[:roots].clone(), vec


def exact(case, seed):
    path = case["path"]
    if path == "multidot":
        V, w = rows(case, seed)
        return torch.stack([(v.double() * w.double()).sum() for v in V])
    if path == "batch":
        out = []
        for k, (L, N) in enumerate(batch_dims(case)):
            e, _ = Plain(L, N, seed + 1000 * k).lowest(case["roots"], 160)
            out.append(e.numpy())
        return out
    L, N = case["L"], case["N"]
    if L > 28:
        return None  # the plain sigma takes longer than it is worth there
    if path == "build":
        h, eri = integrals(L, seed)
        return diagonal(determinants(L, N), L, h, eri).flip(0).cpu().numpy()
    p = Plain(L, N, seed)
    if path == "solve":
        e, vec = p.lowest(1, 140)
        vec = vec.flip(0)
        return {"energy": float(e[0]), "vector": (vec if vec[0] >= 0 else -vec).cpu().numpy()}
    nv = case.get("nv", 1)
    x = vectors(plain_bits(p.M, L), L, N, nv, type_of(case), seed)
    y = torch.stack([p.apply(v.double().flip(0)).flip(0) for v in x])
    return y[0].cpu() if path == "host" else y
