"""The work that programs have this framework do, as cases to be timed and compared.

A case is a plain dict.  Its system is an a x b momentum mesh with `ne` particles ("9", or "4,4"
for two conserved components) in the sector of total momentum (kx, ky); the operator is a cosine
band plus a momentum-conserving two-body interaction whose magnitude falls with the momentum
transfer and whose phases are random (the shape of the repository's benchmark recipes).  The
kinds are the calls a program makes:

  edsolve    EDsolve(subspace, H; N, method): the whole public call, handle included, FP64
  solve      a kept Handle moved to a sector, then its lowest pairs (eigsolve), FP64 or mixed
  sweep      a kept Handle moved to a sector, then H0 + u V for many u at once (batch_solve)
  map        y = H x on device vectors over a kept hit cache, c128 or c64
  linearmap  the host callable of create_gpu_linearmap, as an outer Krylov code calls it
  rdm1       PES_1rdm of a state, the analysis step after a solve
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "momentumed.jl_b200"))

import momed  # noqa: E402
from momed import _lib  # noqa: E402
from momed.core import pair_operator  # noqa: E402

DEVICE = "cuda"


def listed():
    return [
        # the smallest solves: latency and launch count (the repository's config-1 sectors, 200 states)
        dict(name="edsolve_3x5_n10", kind="edsolve", a=3, b=5, ne="5", kx=0, ky=1, nev=10, method="map"),
        # the system of the reference's GPU notebook: 4x6, 8 electrons, 30.6k states, 9 pairs
        dict(name="edsolve_4x6_n9", kind="edsolve", a=4, b=6, ne="8", kx=1, ky=2, nev=9, method="map"),
        # the sparse method on a notebook-sized sector (6x4, 6 electrons, 5.6k states)
        dict(name="edsolve_sparse_6x4", kind="edsolve", a=6, b=4, ne="6", kx=5, ky=3, nev=10, method="sparse"),
        # an ordinary single solve with its vectors (174k states)
        dict(name="solve_3x9_fp64", kind="solve", a=3, b=9, ne="9", kx=1, ky=4, nev=4, krylovdim=30,
             precision="fp64", vectors=True),
        # the same sector in mixed precision with an odd number of pairs, as serving requests ask
        dict(name="solve_3x9_mixed", kind="solve", a=3, b=9, ne="9", kx=2, ky=7, nev=7, krylovdim=30,
             precision="mixed", vectors=False),
        # the large single solve (1.0M states, krylovdim 64)
        dict(name="solve_3x10_fp64", kind="solve", a=3, b=10, ne="10", kx=0, ky=3, nev=6, krylovdim=64,
             precision="fp64", vectors=False),
        # the headline sweep: one sector x 32 interaction strengths
        dict(name="sweep_3x9_32", kind="sweep", a=3, b=9, ne="9", kx=0, ky=5, nev=4, nu=32, krylovdim=30),
        # a ragged sweep on a small sector (5.5k states, 11 strengths)
        dict(name="sweep_3x7_11", kind="sweep", a=3, b=7, ne="7", kx=2, ky=3, nev=4, nu=11, krylovdim=30),
        # one application of the map, both precisions, on the large sectors
        dict(name="map_3x10_c128", kind="map", a=3, b=10, ne="10", kx=2, ky=9, dtype="c128"),
        dict(name="map_two_comp_4x6_c64", kind="map", a=4, b=6, ne="4,4", kx=3, ky=1, dtype="c64"),
        # the drop-in callable with host vectors, no cache: every term evaluated at every call
        dict(name="linearmap_3x9_c128", kind="linearmap", a=3, b=9, ne="9", kx=1, ky=1, dtype="c128"),
        # the one-body density matrix of a state
        dict(name="rdm1_3x9", kind="rdm1", a=3, b=9, ne="9", kx=2, ky=2),
    ]


# systems the drawn cases come from: (a, b, particles), sectors of 40 to 4.7M states
SYSTEMS = [(3, 4, "5"), (4, 3, "2,3"), (3, 5, "5"), (5, 3, "7"), (4, 4, "5"), (4, 4, "7"), (3, 6, "6"), (3, 6, "9"),
           (4, 3, "3,4"), (3, 7, "6"), (3, 7, "7"), (6, 4, "6"), (4, 5, "8"), (5, 5, "6"), (3, 5, "3,4"), (4, 6, "8"),
           (3, 8, "8"), (5, 5, "8"), (4, 6, "11"), (5, 5, "10"), (3, 9, "9"), (2, 13, "10"), (4, 4, "4,4"),
           (4, 7, "9"), (4, 5, "3,4"), (3, 9, "11"), (4, 7, "11"), (3, 10, "10"), (4, 5, "4,4"), (4, 6, "4,4")]

# states of a kind's drawn sectors: from, to
RANGES = {"edsolve": (60, 140e3), "solve": (200, 500e3), "sweep": (200, 180e3), "map": (2e3, 4.8e6),
          "linearmap": (200, 1.1e6), "rdm1": (200, 1.1e6)}


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi = RANGES[kind]
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    near = sorted((s for s in SYSTEMS if lo <= states(*s) <= hi), key=lambda s: abs(math.log(states(*s) / want)))
    a, b, ne = rng.choice(near[:3])
    case = dict(kind=kind, a=a, b=b, ne=ne, kx=rng.randrange(a), ky=rng.randrange(b))
    n = states(a, b, ne)
    if kind == "edsolve":
        case |= dict(nev=rng.randint(1, 10), method=rng.choice(("map", "sparse")))
    elif kind == "solve":
        precision = rng.choice(("fp64", "mixed"))
        case |= dict(nev=rng.randint(1, 10 if n < 2e5 else 6), krylovdim=rng.choice((30, 36, 48)), precision=precision,
                     vectors=precision == "fp64" and rng.random() < 0.5)
    elif kind == "sweep":
        case |= dict(nev=rng.randint(1, 5), nu=rng.randint(2, 32 if n > 1e5 else 27), krylovdim=30)
    elif kind in ("map", "linearmap"):
        case |= dict(dtype=rng.choice(("c128", "c64")))
    return case


# ------------------------------------------------------------------------------- the system
def _ne(ne):
    return tuple(int(v) for v in str(ne).split(","))


def states(a, b, ne):
    """States of one sector (all sectors of a mesh are within a fraction of a percent of this)."""
    return math.prod(math.comb(a * b, n) for n in _ne(ne)) / (a * b)


def hits_per_row(a, b, ne):
    """Two-body terms that connect a state to others of its sector, on average."""
    nk, n = a * b, _ne(ne)
    h = sum(math.comb(c, 2) * (math.comb(nk - c + 2, 2) / nk) for c in n)
    if len(n) == 2:
        h += n[0] * n[1] * (nk - n[0] + 1) * (nk - n[1] + 1) / nk
    return h


def _terms(case, seed):
    """Upper-Hermitian one-body and two-body terms as arrays (amp, out, in) of orbital masks."""
    a, b, comps = case["a"], case["b"], len(_ne(case["ne"]))
    nk = a * b
    rng = np.random.default_rng([seed, a, b, comps])
    orb = np.arange(nk * comps)
    k = orb % nk
    x, y, c = k % a, k // a, orb // nk
    band = np.cos(2 * np.pi * x / a) + np.cos(2 * np.pi * y / b)
    bit = np.uint64(1) << orb.astype(np.uint64)
    one = (band.astype(np.complex128), bit.copy(), bit.copy())
    p, q = np.triu_indices(len(orb), 1)
    key = ((x[p] + x[q]) % a * b + (y[p] + y[q]) % b) * 4 + c[p] + c[q]     # momentum and components
    amps, outs, ins = [], [], []
    for g in np.unique(key):
        sel = np.flatnonzero(key == g)
        o, i = np.meshgrid(sel, sel, indexing="ij")

        def v(p1, q1):         # interaction of momentum transfer k(q1) - k(p1), folded to the nearest image
            fx, fy = (x[q1] - x[p1]) / a, (y[q1] - y[p1]) / b
            t = 2 * np.pi * np.hypot(fx - np.floor(fx + 0.5), fy - np.floor(fy + 0.5))
            return np.exp(-t * t / 2) / (t + 0.5) * np.exp(2j * np.pi * rng.random(t.shape))

        m = v(p[o], p[i]) - v(p[o], q[i])
        up = i > o
        d = np.arange(len(sel))
        masks = bit[p[sel]] | bit[q[sel]]
        oo, ii = (bit[p] | bit[q])[o[up]], (bit[p] | bit[q])[i[up]]
        # upper: the larger mask annihilated
        amps += [m[up] / nk, m[d, d].real.astype(np.complex128) / nk]
        outs += [np.minimum(oo, ii), masks]
        ins += [np.maximum(oo, ii), masks]
    return one, (np.concatenate(amps), np.concatenate(outs), np.concatenate(ins))


def _operators(case, seed):
    bits = case["a"] * case["b"] * len(_ne(case["ne"]))
    return [momed.MBOperator(momed.ScatterList(*t, bits=bits), upper_hermitian=True) for t in _terms(case, seed)]


def _hamiltonian(case, seed):
    one, two = (op.scats for op in _operators(case, seed))
    return momed.MBOperator(one, two, upper_hermitian=True)


def _subspace(case, handle):
    a, b, ne = case["a"], case["b"], _ne(case["ne"])
    i = np.arange(a * b)
    para = momed.EDPara(k_list=np.stack([i % a, i // a]), Gk=(a, b), Nc_conserve=len(ne),
                        one_momentum_coordinate=False, two_momentum_coordinate=False)
    subs, _ = momed.ED_momentum_subspaces(para, ne, momentum_restriction=True,
                                          momentum_list=[(case["kx"], case["ky"])], handle=handle)
    return subs[0]


def _vector(n, seed, dtype):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    v = torch.randn(n, dtype=torch.complex128, device=DEVICE, generator=g)
    return (v / torch.linalg.vector_norm(v)).to(dtype)


def _reference_phase(n, seed):
    """Unit phases against which an eigenvector's free overall phase is fixed."""
    return np.exp(2j * np.pi * np.random.default_rng([seed, 7]).random(n))


def _fixed(ref, v):
    c = np.vdot(ref, v)
    return v * (np.conj(c) / abs(c))


# ------------------------------------------------------------------------------- the calls
def prepare(case, seed):
    kind = case["kind"]
    h = momed.Handle(0)
    sub = _subspace(case, h)
    n = len(sub)
    if kind == "edsolve":
        h.close()
        momed.activate_b200()
        return dict(case=case, sub=sub, op=_hamiltonian(case, seed), ref=_reference_phase(n, seed), seed=seed)
    if kind in ("solve", "sweep"):
        one, two = _operators(case, seed)
        amp_a, amp_b, in_, out, pm = pair_operator(one, two)
        h.set_scatter_pair(amp_a, amp_b, in_, out, pm)
        h.set_param(1.0)
        u = np.linspace(0.5, 2.0, case["nu"]) if kind == "sweep" else None
        return dict(case=case, h=h, basis=sub.list, u=u, ref=_reference_phase(n, seed), seed=seed)
    if kind == "rdm1":
        psi = momed.MBS64Vector(_vector(n, seed, torch.complex128).cpu().numpy(), sub)
        return dict(case=case, h=h, psi=psi)
    dtype = torch.complex128 if case["dtype"] == "c128" else torch.complex64
    x = _vector(n, seed, dtype)
    if kind == "linearmap":
        h.close()
        op = _hamiltonian(case, seed)
        if dtype is torch.complex64:
            s = op.scats
            op = momed.MBOperator(momed.ScatterList(s.amp, s.out, s.in_, s.pm, s.bits, np.complex64), upper_hermitian=True)
        m = momed.create_gpu_linearmap(momed.LinearMap(op, sub))
        return dict(case=case, m=m, x=x.cpu().numpy())
    full = momed.hermitian_complete(_hamiltonian(case, seed))
    h.set_basis(sub.list)
    h.set_scatter(full.amp, full.in_, full.out, full.pm)
    h.build_hit_cache()
    torch.cuda.synchronize()
    return dict(case=case, h=h, x=x, y=torch.empty_like(x), precision=_lib.C128 if dtype is torch.complex128 else _lib.C64)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "edsolve":
        vals, vecs = momed.EDsolve(state["sub"], state["op"], N=case["nev"], method=case["method"], method_info=False,
                                   seed=state["seed"])
        return {"energies": vals, "vectors": np.stack([_fixed(state["ref"], v.vec) for v in vecs])}
    if kind == "solve":
        h = state["h"]
        h.set_basis(state["basis"])
        mixed = case["precision"] == "mixed"
        vals, vecs, _, _ = h.eigsolve(case["nev"], krylovdim=case["krylovdim"], tol=1e-12, seed=state["seed"],
                                      precision=_lib.PREC_MIXED if mixed else _lib.PREC_FP64,
                                      want_vectors=case["vectors"])
        if vecs is None:
            return {"energies": vals}
        return {"energies": vals, "vectors": np.stack([_fixed(state["ref"], v) for v in vecs])}
    if kind == "sweep":
        h = state["h"]
        h.set_basis(state["basis"])
        vals, _, _, _ = h.batch_solve(state["u"], case["nev"], krylovdim=case["krylovdim"], tol=1e-12,
                                      seed=state["seed"], precision=_lib.PREC_MIXED)
        return {"energies": vals}
    if kind == "map":
        state["h"].matvec_device(state["x"].data_ptr(), state["y"].data_ptr(), state["precision"])
        return state["y"]
    if kind == "linearmap":
        return state["m"](state["x"])
    return momed.PES_1rdm(state["psi"], handle=state["h"])


def work(case):
    """Inputs read once and outputs written once; the operations of one application of the map (for
    the solves: of one Krylov cycle, the least a solve can take), 8 per hit."""
    a, b, ne, kind = case["a"], case["b"], case["ne"], case["kind"]
    n = states(a, b, ne)
    hits = n * hits_per_row(a, b, ne)
    terms = 0.5 * (a * b * len(_ne(ne))) ** 2 / (a * b) * 0.5 * (a * b * len(_ne(ne))) ** 2
    if kind in ("edsolve", "solve"):
        vec = 16 * n * case["nev"] if case.get("vectors", True) else 0
        return {"bytes": 8 * n + 40 * terms + vec, "flops": 8 * hits * min(case.get("krylovdim", 30), n)}
    if kind == "sweep":
        return {"bytes": 8 * n + 56 * terms, "flops": 8 * hits * case["nu"] * min(case["krylovdim"], n)}
    if kind == "rdm1":
        return {"bytes": 24 * n, "flops": 4 * n * sum(_ne(ne))}
    size = 16 if case["dtype"] == "c128" else 8
    return {"bytes": (8 + 2 * size) * n + 40 * terms, "flops": 8 * hits}


# ------------------------------------------------------------------------------- in 64 bits, by torch
def _basis64(case):
    """The sector's states in ascending order, found among all states of the right particle numbers."""
    a, b, ne = case["a"], case["b"], _ne(case["ne"])
    nk = a * b

    def component(n):
        got = []
        for s0 in range(0, 1 << nk, 1 << 26):
            s = torch.arange(s0, min(s0 + (1 << 26), 1 << nk), device=DEVICE)
            count = torch.zeros_like(s, dtype=torch.int8)
            for i in range(nk):
                count += ((s >> i) & 1).to(torch.int8)
            got.append(s[count == n])
        s = torch.cat(got)
        kx, ky = torch.zeros_like(s), torch.zeros_like(s)
        for i in range(nk):
            o = (s >> i) & 1
            kx += o * (i % a)
            ky += o * (i // a)
        return s, kx % a, ky % b

    s, kx, ky = component(ne[0])
    if len(ne) == 2:
        t, tx, ty = component(ne[1])            # the second component has the higher bits
        rows = []
        for j in range(a * b):
            jx, jy = j % a, j // a
            low = s[(kx == (case["kx"] - jx) % a) & (ky == (case["ky"] - jy) % b)]
            high = t[(tx == jx) & (ty == jy)]
            rows.append(((high[:, None] << nk) | low[None, :]).reshape(-1))
        return torch.sort(torch.cat(rows))[0]
    return s[(kx == case["kx"]) & (ky == case["ky"])]


def _between(mask):
    """Bits strictly between the two set bits of each mask."""
    hi = 1 << (int(mask).bit_length() - 1)
    lo = int(mask) & -int(mask)
    return (hi - 1) & ~((lo << 1) - 1) if hi != lo else 0


def _pair_hits(basis, out, in_):
    """Rows, target rows and signs of the term c+_out c_in on the basis."""
    rows = torch.nonzero(((basis & out) == out) & ((basis & in_ & ~out) == 0)).reshape(-1)
    mid = basis[rows] & ~out
    target = torch.searchsorted(basis, mid | in_)
    par = mid & (_between(out) ^ _between(in_))
    for shift in (32, 16, 8, 4, 2, 1):
        par = par ^ (par >> shift)
    return rows, target, (1 - 2 * (par & 1)).to(torch.float64)


def _diagonal(basis, amp, out):
    d = torch.zeros(len(basis), dtype=torch.float64, device=DEVICE)
    for v, o in zip(amp, out):
        d += float(v.real) * ((basis & int(o)) == int(o)).to(torch.float64)
    return d


def _apply64(case, seed, x, single):
    """H x term by term."""
    basis = _basis64(case)
    (oa, oo, _), (ta, to, ti) = _terms(case, seed)
    if single:                 # a complex64 operator: its amplitudes are the given numbers
        oa, ta = oa.astype(np.complex64).astype(np.complex128), ta.astype(np.complex64).astype(np.complex128)
    diag = to == ti
    y = (_diagonal(basis, oa, oo) + _diagonal(basis, ta[diag], to[diag])) * x
    for v, o, i in zip(ta[~diag], to[~diag], ti[~diag]):
        rows, target, sign = _pair_hits(basis, int(o), int(i))
        y.index_add_(0, rows, complex(v) * sign * x[target])
        y.index_add_(0, target, complex(np.conj(v)) * sign * x[rows])
    return y


def _matrix64(case, seed):
    """Diagonals of the one-body and two-body parts, and the two-body off-diagonal CSR matrix."""
    basis = _basis64(case)
    (oa, oo, _), (ta, to, ti) = _terms(case, seed)
    diag = to == ti
    r, c, v = [], [], []
    for amp, o, i in zip(ta[~diag], to[~diag], ti[~diag]):
        rows, target, sign = _pair_hits(basis, int(o), int(i))
        r += [rows.to(torch.int32), target.to(torch.int32)]
        c += [target.to(torch.int32), rows.to(torch.int32)]
        v += [complex(amp) * sign, complex(np.conj(amp)) * sign]
    r, order = torch.sort(torch.cat(r))
    c, v = torch.cat(c)[order].to(torch.int64), torch.cat(v)[order]
    ptr = torch.searchsorted(r, torch.arange(len(basis) + 1, device=DEVICE, dtype=torch.int32))
    m = torch.sparse_csr_tensor(ptr, c, v, (len(basis), len(basis)), check_invariants=False)
    return _diagonal(basis, oa, oo), _diagonal(basis, ta[diag], to[diag]), m


def _lowest64(apply_h, n, nev, vectors):
    """The nev lowest eigenpairs: dense for small n, else Lanczos with full reorthogonalisation."""
    if n <= 2500:
        w, z = torch.linalg.eigh(apply_h(torch.eye(n, dtype=torch.complex128, device=DEVICE)))
        return w[:nev], z[:, :nev].T
    steps = 1000
    basis = torch.empty((min(steps, 120), n), dtype=torch.complex128, device=DEVICE)
    basis[0] = _vector(n, 1, torch.complex128)
    alpha, beta = [], []
    for j in range(steps):
        if j + 1 >= len(basis):
            basis = torch.cat([basis, torch.empty_like(basis[:60])])
        w = apply_h(basis[j])
        q = basis[: j + 1]
        c = (q @ w.conj()).conj()
        w = w - c @ q
        w = w - (q @ w.conj()).conj() @ q
        nrm = torch.linalg.vector_norm(w)
        basis[j + 1] = w / nrm
        alpha.append(c[j].real)
        beta.append(nrm)
        if j >= 40 and j % 12 == 0:
            t = torch.diag(torch.stack(alpha))
            off = torch.stack(beta[:-1])
            t = t + torch.diag(off, 1) + torch.diag(off, -1)
            e, z = torch.linalg.eigh(t.cpu())
            if float((beta[-1].cpu() * z[-1, :nev].abs()).max()) < 2e-13 * max(1.0, float(e.abs().max())):
                break
    got = (z[:, :nev].T.to(DEVICE).to(torch.complex128) @ basis[: j + 1]) if vectors else None
    return e[:nev], got


def exact(case, seed):
    kind = case["kind"]
    if kind in ("map", "linearmap"):
        dtype = torch.complex128 if case["dtype"] == "c128" else torch.complex64
        n = len(_basis64(case))
        x = _vector(n, seed, dtype).to(torch.complex128)
        y = _apply64(case, seed, x, kind == "linearmap" and dtype is torch.complex64)
        return y if kind == "map" else y.cpu().numpy()
    if kind == "rdm1":
        # c+_i c_j with i != j changes the total momentum: only the occupations are inside the sector
        basis = _basis64(case)
        w = _vector(len(basis), seed, torch.complex128).abs() ** 2
        bits = case["a"] * case["b"] * len(_ne(case["ne"]))
        return np.diag([complex((w * ((basis >> i) & 1)).sum().item()) for i in range(bits)])
    d1, d2, m = _matrix64(case, seed)
    n = len(d1)

    def solve(u, vectors):
        def apply_h(x):
            if x.dim() == 2:
                return (torch.diag(d1 + u * d2).to(torch.complex128) + u * m.to_dense()) @ x
            return (d1 + u * d2) * x + u * (m @ x)
        return _lowest64(apply_h, n, case["nev"], vectors)

    if kind == "sweep":
        return {"energies": np.stack([solve(u, False)[0].cpu().numpy() for u in np.linspace(0.5, 2.0, case["nu"])])}
    vectors = case.get("vectors", True)
    e, z = solve(1.0, vectors)
    if not vectors:
        return {"energies": e.cpu().numpy()}
    ref = _reference_phase(n, seed)
    return {"energies": e.cpu().numpy(), "vectors": np.stack([_fixed(ref, v) for v in z.cpu().numpy()])}
