"""The workloads whose speed is followed: applies, Krylov solvers and vector algebra
through the package's public entry points, over the sizes they are used at.

``listed()`` are the followed cases, ``draw(rng)`` one more of the same ranges;
``prepare`` makes what a program has in hand before the call (inputs, the Hamiltonian),
``run`` is one pass, ``work`` what the pass cannot do without, and ``exact`` the values
that plain torch gives in 64 bits.

The mixed (32-bit) solvers hand their results back in 64-bit arrays although they carry
the accuracy of 32-bit Krylov vectors; ``run`` returns those as 32-bit values, except the
energies, which the solvers refine in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

import qkrylov_gb300 as qk

DEV = "cuda"


# ------------------------------------------------------------------ models
def bonds(c):
    return [(i, (i + 1) % c["L"]) for i in range(c["L"] if c["pbc"] else c["L"] - 1)]


def terms(c):
    """(coefficient, [(operator, site), ...]) of the case's model."""
    L, out = c["L"], []
    if c["model"] in ("spin", "field"):
        for i, j in bonds(c):
            out += [(c.get("coupling", 1.0), [("Sz", i), ("Sz", j)]), (0.5, [("Sp", i), ("Sm", j)]), (0.5, [("Sm", i), ("Sp", j)])]
    if c["model"] == "field":  # a tilted field and a Dzyaloshinskii-Moriya coupling: complex, no conserved Sz
        for i in range(L):
            out += [(0.3, [("Sx", i)]), (0.2, [("Sy", i)])]
        for i in range(0, L - 1, 2):
            out += [(0.1j, [("Sp", i), ("Sm", i + 1)]), (-0.1j, [("Sm", i), ("Sp", i + 1)])]
    if c["model"] == "fermion":
        for i, j in bonds(c):
            out += [(-1.0, [("Cdag", i), ("C", j)]), (-1.0, [("Cdag", j), ("C", i)]), (0.7, [("N", i), ("N", j)])]
    if c["model"] == "hubbard":
        for i, j in bonds(c):
            for s in ("Up", "Dn"):
                out += [(-1.0, [("Cdag" + s, i), ("C" + s, j)]), (-1.0, [("Cdag" + s, j), ("C" + s, i)])]
        out += [(4.0 * c.get("coupling", 1.0), [("Nupdn", i)]) for i in range(L)]
    return out


def scanned(c, seed):
    """The model at one point of a parameter scan (Sz Sz coupling or U): another seed, another point."""
    return {**c, "coupling": 0.95 + 0.1 * (0.6180339887498949 * (seed + 1) % 1.0)}


def dim(c):
    L = c["L"]
    if c["model"] == "field":
        return 2 ** L
    if c["model"] == "hubbard":
        return math.comb(L, c["nup"]) * math.comb(L, c["ndn"])
    return math.comb(L, c["n"])


def hamiltonian(c):
    L = c["L"]
    if c["model"] == "field":
        basis, site = qk.SpinHalfBasis(L), qk.SpinHalfSite()
    elif c["model"] == "spin":
        basis, site = qk.SpinHalfBasis(L, conserve_sz=True, sz=c["n"] - L / 2), qk.SpinHalfSite()
    elif c["model"] == "fermion":
        basis, site = qk.FermionBasis(L, conserve_n=True, n=c["n"]), qk.FermionSite()
    else:
        basis, site = qk.HubbardBasis(L, nup=c["nup"], ndn=c["ndn"]), qk.HubbardSite()
    ops = qk.OpSum()
    for coeff, factors in terms(c):
        ops.add_term(coeff, *[v for f in factors for v in f])
    return qk.MatrixFreeHamiltonian(basis, site, ops)


def chain(L, pbc=True, n=None, model="spin"):
    return {"model": model, "L": L, "pbc": pbc, "n": L // 2 if n is None else n}


def hubbard(L, pbc=True, nup=None, ndn=None):
    return {"model": "hubbard", "L": L, "pbc": pbc, "nup": L // 2 if nup is None else nup,
            "ndn": L // 2 if ndn is None else ndn}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # y = Hx in a user's own loop: a teaching-size ring, where the launches are the cost
        {"name": "apply64_ring14", "kind": "apply", "fp32": False, **chain(14)},
        # the same at an ordinary research size, odd length, open ends, in 64 bits
        {"name": "apply64_chain23", "kind": "apply", "fp32": False, **chain(23, pbc=False, n=11)},
        # the largest ring that is used in earnest, in 32 bits
        {"name": "apply32_ring28", "kind": "apply", "fp32": True, **chain(28)},
        # electrons: signs on the hops, and a basis whose order is not the internal one
        {"name": "apply32_hubbard13", "kind": "apply", "fp32": True, **hubbard(13, nup=6, ndn=6)},
        # complex couplings that conserve nothing: the whole space of a short chain
        {"name": "apply64_field18", "kind": "apply", "fp32": False, **chain(18, pbc=False, n=0, model="field")},
        # the drop-in ground-state solver: 64 bits, full reorthogonalisation, start vector and state on the host
        {"name": "lanczos64_ring20", "kind": "lanczos", "fp32": False, "steps": 80, **chain(20)},
        # the mixed-precision ground-state solver
        {"name": "lanczos32_ring24", "kind": "lanczos", "fp32": True, "steps": 100, **chain(24)},
        # thermodynamics over all Sz sectors in one batch (1 to 184,756 rows a sector)
        {"name": "ftlm32_ring20", "kind": "ftlm", "R": 32, "steps": 40, **chain(20)},
        # dynamical structure factor, every momentum of the ring in one batch
        {"name": "spectrum32_ring22", "kind": "spectrum", "fp32": True, "rhs": 12, "steps": 120, **chain(22)},
        # one spectral function the reference's way: 64 bits, one vector
        {"name": "spectrum64_ring18", "kind": "spectrum", "fp32": False, "rhs": 1, "steps": 100, **chain(18)},
        # the lowest states of a Hubbard chain by Davidson, the reference's form
        {"name": "davidson64_hubbard10", "kind": "davidson", "n_eig": 2, "sub": 16, "steps": 24,
         **hubbard(10, pbc=False)},
        # a block subspace step on 32-bit vectors: projections on a basis and combinations of it
        {"name": "subspace32_k32", "kind": "subspace", "n": 3432 * 3432, "k": 32, "nw": 4},
    ]


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "lanczos", "lanczos", "ftlm", "spectrum", "spectrum", "davidson",
                       "subspace"])
    pbc = rng.random() < 0.6
    if kind == "apply":
        model = rng.choice(["spin", "spin", "fermion", "hubbard", "field"])
        fp32 = rng.random() < 0.5
        if model == "field":
            m = chain(rng.randint(10, 19), pbc, 0, model)
        elif model == "hubbard":
            L = rng.randint(6, 13)
            m = hubbard(L, pbc, rng.randint(L // 2 - 1, L // 2), rng.randint(L // 2 - 1, L // 2))
        else:
            L = rng.randint(12, 27)
            m = chain(L, pbc, L // 2 - rng.randint(0, 2), model)
        return {"kind": kind, "fp32": fp32, **m}
    if kind == "lanczos":
        fp32 = rng.random() < 0.5
        L = 2 * rng.randint(8, 12 if fp32 else 10)  # even: a ground state of its own
        return {"kind": kind, "fp32": fp32, "steps": rng.randint(50, 100 if fp32 else 80), **chain(L, pbc)}
    if kind == "ftlm":
        return {"kind": kind, "R": rng.choice([4, 7, 16, 24, 32]), "steps": rng.randint(20, 40),
                **chain(rng.randint(10, 20), pbc)}
    if kind == "spectrum":
        fp32 = rng.random() < 0.5
        return {"kind": kind, "fp32": fp32, "rhs": rng.randint(2, 12) if fp32 else 1, "steps": rng.randint(100, 120) - (0 if fp32 else 20),
                **chain(2 * rng.randint(7, 11 if fp32 else 9))}
    if kind == "davidson":
        L = rng.randint(7, 10)
        return {"kind": kind, "n_eig": 1, "sub": rng.randint(12, 20), "steps": rng.randint(12, 24),
                **hubbard(L, False, L // 2, (L + 1) // 2)}
    return {"kind": kind, "n": int(10 ** rng.uniform(4, math.log10(3432 * 3432))), "k": rng.randint(3, 32),
            "nw": rng.randint(1, 4)}


# ------------------------------------------------------------------ inputs
BETAS = 1.0 / np.geomspace(0.2, 10.0, 40)
ETA = 0.2


def gaussian(seed, shape, dtype):
    g = torch.Generator(device=DEV).manual_seed(1000003 * seed + 17)
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


def pinned(x):
    h = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    h.copy_(x)
    return h.numpy()


OMEGAS = np.linspace(0.0, 4.0, 200)


def structure_factor(c):
    """Sz(q) psi of the ground state psi for q = 2 pi k / L (k = 1 ..; q = pi for one), and its energy."""
    A = Plain(c, True)
    start = gaussian(1, (A.n,), torch.complex128)
    a, b, _, V = krylov(A, start, min(60, A.n), orth=True)
    lam, u = lowest(a, b)
    psi = u.to(start.dtype).to(DEV) @ torch.stack(V)
    psi = psi / psi.norm()
    out = []
    for k in range(1, c["rhs"] + 1):
        f = torch.zeros_like(psi)
        q = 2 * math.pi * (k if c["rhs"] > 1 else c["L"] // 2) / c["L"]
        for i in range(c["L"]):
            f += complex(math.cos(q * i), math.sin(q * i)) * (((A.s >> i) & 1).double() - 0.5)
        out.append(f * psi / math.sqrt(c["L"]))
    return A, torch.stack(out), lam


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "subspace":
        scale = 1.0 / math.sqrt(c["n"])
        V = [gaussian(97 * seed + j, (c["n"],), torch.complex64).mul_(scale) for j in range(c["k"])]
        W = [gaussian(97 * seed + 50 + j, (c["n"],), torch.complex64).mul_(scale) for j in range(c["nw"])]
        C = gaussian(97 * seed + 90, (c["nw"], c["k"]), torch.complex128).cpu().numpy()
        return {"case": c, "V": V, "W": W, "C": C}
    if kind == "ftlm":  # one Hamiltonian for each Sz sector
        return {"case": c, "H": [hamiltonian({**c, "n": n}) for n in range(c["L"] + 1)], "seed": seed}
    if kind in ("spectrum", "davidson"):
        c = scanned(c, seed)
    s = {"case": c, "H": hamiltonian(c)}
    n = dim(c)
    if kind == "apply":
        s["x"] = gaussian(seed, (n,), torch.complex64 if c["fp32"] else torch.complex128)
    elif kind == "lanczos":
        s["v0"] = pinned(gaussian(seed, (n,), torch.complex128))
        s["vec"] = pinned(torch.zeros(n, dtype=torch.complex128))
    elif kind == "spectrum":
        _, phi, s["E0"] = structure_factor(c)
        s["phi"] = pinned(phi if c["rhs"] > 1 else phi[0])
    return s


# ------------------------------------------------------------------ one pass
def pointers(vectors):
    return (ctypes.c_void_p * len(vectors))(*[v.data_ptr() for v in vectors])


def doubles(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "apply":
        return state["H"].apply(state["x"])
    if kind == "lanczos":
        r = qk.lanczos_fixed_steps(state["H"], c["steps"], mixed=c["fp32"], v0=state["v0"],
                                   eigenvector_out=state["vec"])
        v = torch.from_numpy(state["vec"])
        return {"energy": r.energy, "state": v.to(torch.complex64) if c["fp32"] else v}
    if kind == "ftlm":
        r = qk.ftlm_sectors(state["H"], BETAS, n_random=c["R"], n_steps=c["steps"], start="philox",
                            seed=state["seed"], shifted=True)
        return [np.float32(a) for a in (r.partition_function, r.internal_energy, r.specific_heat, r.log_shift)]
    if kind == "spectrum":
        if c["fp32"]:
            S, _, _ = qk.spectral_functions_block(state["H"], state["phi"], OMEGAS, state["E0"], eta=ETA,
                                                  n_iter=c["steps"], mixed=True)
            return np.float32(S)
        r = qk.continued_fraction_coeffs(state["H"], state["phi"], n_iter=c["steps"])
        return qk.evaluate_spectral_function(r, OMEGAS, state["E0"], ETA)
    if kind == "davidson":
        r = qk.davidson_lowest_ex(state["H"], n_eig=c["n_eig"], max_subspace=c["sub"], tol=1e-10, mixed=False,
                                  return_vectors=True, max_iter=c["steps"])
        return {"energies": r.eigenvalues, "states": r.eigenvectors}
    V, W, C = state["V"], state["W"], state["C"]
    n, k, nw = c["n"], c["k"], c["nw"]
    P = np.empty((nw, k), dtype=np.complex128)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    v, lib = pointers(V), qk.lib()
    R = [torch.empty_like(w) for w in W]
    for rc in (lib.qkrylov_vector_mdot_device_f32(v, k, pointers(W), nw, n, 2, doubles(P), stream),
               lib.qkrylov_vector_mcombine_device_f32(v, k, doubles(C), pointers(R), nw, n, 0, stream)):
        if rc:
            raise RuntimeError("vector call failed: %d" % rc)
    return {"projections": np.complex64(P), "combinations": R}


# ------------------------------------------------------------------ what a pass cannot do without
def entries(c, n):
    """Generated matrix entries off the diagonal, about half of every hop's rows."""
    return sum(1 for _, f in terms(c) if any(o[0] not in ("Sz", "N", "Nupdn") for o in f)) * n / 4.0


def work(case):
    c, kind = case, case["kind"]
    if kind == "subspace":
        return {"bytes": 8.0 * c["n"] * (c["k"] + 2 * c["nw"]), "flops": 16.0 * c["n"] * c["k"] * c["nw"]}
    n = 2 ** c["L"] if kind == "ftlm" else dim(c)
    e = 8.0 if c.get("fp32", kind == "ftlm") else 16.0
    flops = 4.0 * entries(c, n) + 8.0 * n
    if kind == "apply":  # x read, y written
        return {"bytes": 2 * e * n, "flops": flops}
    M = c["steps"]
    if kind == "lanczos":
        # a step reads v_k and v_{k-1} and writes v_{k+1}; in 64 bits it also reads the whole basis twice
        # (projections, combination); at the end the basis once; the state and the start vector once
        basis = 0.0 if c["fp32"] else M * (M + 1)
        return {"bytes": n * (e * (3 * M + basis + M) + 32), "flops": M * (flops + 24.0 * n) + 8.0 * n * basis}
    if kind == "ftlm":
        return {"bytes": 3 * M * c["R"] * e * n, "flops": M * c["R"] * (flops + 24.0 * n)}
    if kind == "spectrum":
        return {"bytes": n * c["rhs"] * (3 * M * e + 16), "flops": M * c["rhs"] * (flops + 24.0 * n)}
    # Davidson: V and HV read once for the residuals, once for projecting, a vector applied, per state and step
    depth = c["sub"] / 2.0
    return {"bytes": M * n * e * (3 * depth + 4 * c["n_eig"]),
            "flops": M * n * c["n_eig"] * (3 * depth * 8.0 + 8.0) + M * c["n_eig"] * flops}


# ------------------------------------------------------------------ the same in 64 bits by plain torch
def states(c):
    """The sector's states in ascending order (the reference's order) as int64."""
    L = c["L"]
    if c["model"] == "field":
        return torch.arange(2 ** L, device=DEV)
    if c["model"] == "hubbard":
        up, dn = ({**c, "model": "spin", "n": c["nup"]}, {**c, "model": "spin", "n": c["ndn"]})
        spread = [sum(((s >> i) & 1) << (2 * i) for i in range(L)) for s in (states(up), states(dn))]
        return (spread[0][:, None] + 2 * spread[1][None, :]).reshape(-1).sort().values
    out = []
    for lo in range(0, 2 ** L, 2 ** 26):
        s = torch.arange(lo, min(lo + 2 ** 26, 2 ** L), device=DEV)
        out.append(s[bits(s, L) == c["n"]])
    return torch.cat(out)


def bits(s, L):
    return sum(((s >> i) & 1).to(torch.int8) for i in range(L))


def parity(s, L):
    for sh in (32, 16, 8, 4, 2, 1):
        s = s ^ (s >> sh)
    return s & 1


class Plain:
    """y = Hx term by term on the list of states; `keep` holds the row indices of every term."""

    def __init__(self, c, keep):
        self.c, self.s = c, states(c)
        self.n, self.keep = self.s.numel(), keep
        self.diag = torch.zeros(self.n, dtype=torch.float64, device=DEV)
        self.list = []
        for coeff, factors in terms(c):
            if any(o in ("Sp", "Sm", "Sx", "Sy") or o[0] == "C" for o, _ in factors):
                self.list.append(self.hop(coeff, factors) if keep else (coeff, factors))
            else:
                a = torch.full_like(self.diag, coeff)
                for o, i in factors:
                    if o == "Sz":
                        a *= ((self.s >> i) & 1).double() - 0.5
                    elif o == "N":
                        a *= ((self.s >> i) & 1).double()
                    else:
                        a *= (((self.s >> (2 * i)) & (self.s >> (2 * i + 1))) & 1).double()
                self.diag += a

    def hop(self, coeff, factors):
        """(target row of each row, n where there is none; amplitude: a number or one a row)."""
        t, ok, amp, sign = self.s, torch.ones_like(self.s, dtype=torch.bool), complex(coeff), None
        for o, i in factors:
            b = i
            if self.c["model"] == "hubbard":
                b = 2 * i + (o.endswith("Dn"))
            one = ((t >> b) & 1).bool()
            i_ = torch.tensor(1j, dtype=torch.complex128, device=DEV)
            if o in ("Sx", "Sy"):
                amp *= 0.5
                if o == "Sy":
                    sign = torch.where(one, -i_, i_)
            else:
                ok = ok & (one if o == "Sm" or (o[0] == "C" and not o.startswith("Cdag")) else ~one)
                if o[0] == "C":
                    p = 1.0 - 2.0 * parity(t & ((1 << b) - 1), b).double()
                    sign = p if sign is None else sign * p
            t = t ^ (1 << b)
        at = torch.searchsorted(self.s, t).clamp_(max=self.n - 1)
        at = torch.where(ok & (self.s[at] == t), at, torch.full_like(at, self.n))
        amp = amp.conjugate()
        if sign is not None:
            return at, (amp if amp.imag else amp.real) * sign.conj()
        return at, amp if amp.imag else amp.real

    def __call__(self, x):
        wide = (lambda a: a[:, None]) if x.dim() == 2 else (lambda a: a)
        xp = torch.cat([x, torch.zeros_like(x[:1])])
        y = wide(self.diag) * x
        for item in self.list:
            at, amp = item if self.keep else self.hop(*item)
            y += (wide(amp) if isinstance(amp, torch.Tensor) else amp) * xp[at]
        return y


def krylov(A, v, steps, orth=False):
    """Lanczos coefficients of every column of v (and the vectors, with full reorthogonalisation)."""
    norm = v.norm(dim=0)
    v = v / norm
    V, alphas, betas, prev, beta = [v], [], [], torch.zeros_like(v), torch.zeros_like(norm)
    for k in range(steps):
        w = A(v)
        a = (v.conj() * w).sum(0).real
        alphas.append(a)
        w = w - a * v - beta * prev
        if orth:
            B = torch.stack(V)
            for _ in range(2):
                w = w - (B.conj() @ w) @ B
        beta = w.norm(dim=0)
        if k + 1 == steps:
            break
        betas.append(beta)
        # a column whose Krylov space is exhausted stays at zero
        prev, v = v, torch.where(beta > 1e-15, w / beta.clamp(min=1e-300), torch.zeros_like(w))
        if orth:
            V.append(v)
    return torch.stack(alphas), torch.stack(betas or [torch.zeros_like(norm)])[:steps - 1], norm, V


def lowest(a, b):
    """Lowest eigenvalue of the tridiagonal matrix and its vector, the largest component positive."""
    a, b = a.reshape(-1).cpu(), b.reshape(-1).cpu()
    lam, U = torch.linalg.eigh(torch.diag(a) + torch.diag(b, 1) + torch.diag(b, -1))
    u = U[:, 0]
    return float(lam[0]), u * torch.sign(u[u.abs().argmax()])


def philox(seed, stream, n):
    """The first two words of Philox4x32-10 (Salmon et al., SC'11) for counters (0 .. n-1, stream)."""
    m32 = 0xFFFFFFFF

    def mul(a, m):  # 32 x 32 bits -> (high, low)
        lo, hi = a * (m & 0xFFFF), a * (m >> 16)
        mid = hi + (lo >> 16)
        return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)

    i = torch.arange(n, device=DEV)
    x, y, z, w = i & m32, i >> 32, torch.full_like(i, stream & m32), torch.full_like(i, stream >> 32)
    k0, k1 = seed & m32, seed >> 32
    for _ in range(10):
        h0, l0 = mul(x, 0xD2511F53)
        h1, l1 = mul(z, 0xCD9E8D57)
        x, y, z, w = h1 ^ y ^ k0, l1, h0 ^ w ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return x, y


def ftlm_start(c, seed, sector, R, padded):
    """The seeded Gaussian vectors of one sector: row i of the sector's enumeration (outer bits, then the inner
    bits by their number of domain walls) takes the generator's block i of stream sector * padded + vector."""
    s, L = states(c), c["L"]
    n_in = (L + 1) // 2
    b = s & ((1 << n_in) - 1)
    key = s >> n_in
    if n_in >= 3:
        key = (key << 6) + bits((b ^ (b >> 1)) & ((1 << (n_in - 1)) - 1), n_in).long()
    order = ((key << n_in) + b).sort().indices  # enumeration -> ascending
    out = torch.empty(s.numel(), R, dtype=torch.complex128, device=DEV)
    for v in range(R):
        r0, r1 = philox(seed, sector * padded + v, s.numel())
        rad = torch.sqrt(-2.0 * torch.log((r0.double() + 1.0) * 2.0 ** -32))
        out[order, v] = torch.polar(rad, 2.0 * math.pi * r1.double() * 2.0 ** -32)
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "davidson":
        return None  # the iterate after a given number of steps: a value of the algorithm, not of the problem
    if kind == "subspace":
        s = prepare(c, seed)
        V = torch.stack(s["V"]).to(torch.complex128)
        P = torch.stack([V.conj() @ w.to(torch.complex128) for w in s["W"]])
        C = torch.from_numpy(s["C"]).to(DEV)
        return {"projections": P, "combinations": [C[o] @ V for o in range(c["nw"])]}
    if kind == "apply":
        x = gaussian(seed, (dim(c),), torch.complex64 if c["fp32"] else torch.complex128)
        return Plain(c, False)(x.to(torch.complex128))
    if kind == "lanczos":
        v0 = gaussian(seed, (dim(c),), torch.complex128)
        a, b, _, V = krylov(Plain(c, True), v0, min(c["steps"], dim(c)), orth=True)
        lam, u = lowest(a, b)
        vec = u.to(V[0].dtype).to(DEV) @ torch.stack(V)
        vec = vec / vec.norm()
        return {"energy": lam, "state": vec}
    if kind == "ftlm":
        R, padded, tri = c["R"], 1 << (c["R"] - 1).bit_length(), []
        for n in range(c["L"] + 1):
            m = {**c, "n": n}
            a, b, norm, _ = krylov(Plain(m, True), ftlm_start(m, seed, n, R, padded), min(c["steps"], dim(m)))
            a, b = a.cpu(), b.cpu()
            for v in range(R):
                keep = 1  # rows before the recurrence ends
                while keep < a.shape[0] and b[keep - 1, v] > 1e-12:
                    keep += 1
                T = torch.diag(a[:keep, v]) + torch.diag(b[:keep - 1, v], 1) + torch.diag(b[:keep - 1, v], -1)
                lam, U = torch.linalg.eigh(T)
                tri.append((lam.numpy(), U[0].numpy() ** 2 * float(norm[v]) ** 2))
        low = min(float(t[0][0]) for t in tri)
        e, w = np.concatenate([t[0] for t in tri]), np.concatenate([t[1] for t in tri])
        f = w[None, :] * np.exp(-BETAS[:, None] * (e[None, :] - low))
        Z, E, E2 = f.sum(1), (f * e).sum(1), (f * e * e).sum(1)
        return [Z / R, E / Z, BETAS ** 2 * (E2 / Z - (E / Z) ** 2), -BETAS * low]
    A, phi, E0 = structure_factor(scanned(c, seed))
    a, b, norm, _ = krylov(A, phi.T.contiguous(), c["steps"])
    z = torch.from_numpy(OMEGAS + E0).to(DEV)[:, None] + 1j * ETA
    f = 1.0 / (z - a[-1])
    for k in range(a.shape[0] - 2, -1, -1):
        f = 1.0 / (z - a[k] - b[k] ** 2 * f)
    S = (-(norm ** 2) * f.imag / math.pi).T
    return S if c["rhs"] > 1 else S[0]

