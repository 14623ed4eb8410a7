"""The measured work of the library: one entry per kind of call a program makes.

listed() holds the fixed cases, draw() samples the same ranges, prepare()
makes what a program has in hand before the call (a context on a torch
stream, densities or orbitals, a density-fitting factor), run() is one pass
through the public Python entry points, and exact() evaluates the same
quantities in 64-bit torch from the integrals' definition (McMurchie-Davidson
over whole classes of shell pairs), without the library.

Molecules are the seeded water clusters of hfgpu.clusters (the benchmark's
workload) in the bases the repository ships, and, for f shells, the four
s, p, d and f shells of two primitives per centre that its f-shell tests use.
Densities and orbitals are synthetic: occupied vectors centred on the
molecules, decaying with distance as localised orbitals do.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hf-rs_b200"))

from hfgpu import CartesianBasis, Context, JKOptions  # noqa: E402
from hfgpu.basis import cartesian_components  # noqa: E402
from hfgpu.clusters import water_cluster  # noqa: E402
from hfgpu.lib import HFG_DF_BF16, HFG_DF_FP32, HFG_DF_FP64, DFTensor  # noqa: E402

AUX = "def2-universal-jkfit"
PRECISION = {"fp64": HFG_DF_FP64, "tf32": HFG_DF_FP32, "bf16": HFG_DF_BF16}
FP32_BELOW, PRIM_BELOW = 3e-5, 1e-13  # the mixed form that whole SCFs use


def listed():
    return [
        # one J/K build of a single molecule: latency (SCF start, serving of small jobs)
        {"name": "jk_water", "kind": "jk", "waters": 1, "basis": "cc-pvdz", "mixed": False, "uhf": False},
        # a Fock build with host matrices, open shell, the reference's arithmetic
        {"name": "fock_uhf", "kind": "fock", "waters": 7, "basis": "6-31g*", "uhf": True},
        # the benchmark's build at an ordinary and the largest size
        {"name": "jk_mixed", "kind": "jk", "waters": 32, "basis": "cc-pvdz", "mixed": True, "uhf": False},
        # a batch of small molecules in one call (serving)
        {"name": "jk_batch", "kind": "batch", "molecules": 48, "waters": 4, "basis": "6-31g*"},
        # f shells
        {"name": "jk_fshell", "kind": "fshell", "centres": 4},
        # forces of a geometry optimisation step
        {"name": "gradient", "kind": "gradient", "waters": 2, "basis": "cc-pvdz", "uhf": False},
        # a density-fitting factor and its first J/K
        {"name": "df_build", "kind": "dfbuild", "waters": 5, "basis": "cc-pvdz", "store": "fp64"},
        # J/K of a DF-SCF iteration: FP64, and the tensor-core form
        {"name": "df_jk_fp64", "kind": "dfjk", "waters": 9, "basis": "cc-pvdz", "store": "fp64", "mma": "fp64"},
        {"name": "df_jk_bf16", "kind": "dfjk", "waters": 24, "basis": "cc-pvdz", "store": "fp32", "mma": "bf16"},
        # RI-MP2 energy on a factor
        {"name": "mp2", "kind": "mp2", "waters": 6, "basis": "cc-pvdz"},
        # pivoted Cholesky vectors and the J/K from them
        {"name": "cholesky", "kind": "cholesky", "waters": 3, "basis": "cc-pvdz", "threshold": 1e-5},
        # a whole SCF of a small molecule
        {"name": "scf", "kind": "scf", "waters": 2, "basis": "cc-pvdz"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jk", "jk", "fock", "batch", "fshell", "gradient", "dfbuild", "dfjk", "mp2", "cholesky", "scf"])
    basis = rng.choice(["sto-3g", "6-31g*", "cc-pvdz"])
    if kind == "jk":
        mixed, uhf = rng.random() < 0.5, rng.random() < 0.3
        return {"kind": kind, "waters": _log_int(rng, 1, (24 if uhf else 31) if mixed else 12), "basis": basis,
                "mixed": mixed, "uhf": uhf}
    if kind == "fock":
        return {"kind": kind, "waters": _log_int(rng, 1, 11), "basis": basis, "uhf": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "molecules": _log_int(rng, 2, 64), "waters": rng.randint(1, 4), "basis": basis}
    if kind == "fshell":
        return {"kind": kind, "centres": rng.randint(1, 4)}
    if kind == "gradient":
        return {"kind": kind, "waters": rng.randint(1, 2), "basis": basis,
                "uhf": basis != "cc-pvdz" and rng.random() < 0.5}
    if kind == "dfbuild":
        return {"kind": kind, "waters": _log_int(rng, 1, 6), "basis": basis,
                "store": rng.choice(["fp64", "tf32", "bf16"]).replace("tf32", "fp32")}
    if kind == "dfjk":
        mma = rng.choice(["fp64", "tf32", "bf16"])
        store = "fp64" if mma == "fp64" and rng.random() < 0.7 else "fp32"
        return {"kind": kind, "waters": _log_int(rng, 1, 10 if mma == "fp64" else 20), "basis": basis, "store": store,
                "mma": mma}
    if kind == "mp2":
        return {"kind": kind, "waters": _log_int(rng, 1, 6), "basis": basis}
    if kind == "cholesky":
        return {"kind": kind, "waters": rng.randint(1, 3), "basis": basis, "threshold": 10.0 ** rng.uniform(-6, -3)}
    return {"kind": kind, "waters": rng.randint(2, 4), "basis": basis}


# ---------------------------------------------------------------- inputs ---

def _spdf_basis(centres, seed):
    """One s, p, d and f shell of two primitives on each centre."""
    rng = np.random.default_rng(seed)
    shells = []
    for l, (lo, hi) in enumerate([(0.3, 3.0), (0.35, 2.0), (0.5, 1.5), (0.6, 1.4)]):
        shells.append((l, np.array([hi, lo]), np.array([0.4, 0.7]), None))
    atoms = [("He", tuple(float(x) for x in 1.8 * np.array([i % 2, i // 2 % 2, i // 4]) + rng.uniform(-0.3, 0.3, 3)))
             for i in range(centres)]
    return CartesianBasis(atoms, {"HE": shells})


def _basis(case, seed):
    if case["kind"] == "fshell":
        return _spdf_basis(case["centres"], seed)
    return CartesianBasis.build(water_cluster(case["waters"], seed=seed), case["basis"])


def _occupied(basis, nocc, seed):
    """n x nocc vectors, each centred on one atom and decaying from it."""
    rng = np.random.default_rng(seed + 77)
    pos = basis.positions()
    home = pos[(np.arange(nocc) * len(pos)) // max(nocc, 1)]
    d = np.linalg.norm(basis.center[:, None, :] - home[None, :, :], axis=2)
    C = rng.standard_normal((basis.n, nocc)) * np.exp(-0.45 * d)
    return np.ascontiguousarray(0.6 * C / np.linalg.norm(C, axis=0))


def _n_occ(case, basis):
    return 2 * case["centres"] if case["kind"] == "fshell" else 5 * case["waters"]


def _densities(case, basis, seed):
    """Total density and the spin densities (one for a closed shell)."""
    C = _occupied(basis, _n_occ(case, basis), seed)
    if case.get("uhf"):
        a, b = C @ C.T, C[:, 1:] @ C[:, 1:].T
        return a + b, [a, b]
    P = 2.0 * C @ C.T
    return P, [P]


def _mo_space(basis, nocc, seed):
    """Orthonormal orbitals and energies with an occupied / virtual gap."""
    rng = np.random.default_rng(seed + 99)
    C = np.linalg.qr(rng.standard_normal((basis.n, basis.n)))[0]
    eps = np.concatenate([np.sort(rng.uniform(-20.0, -0.4, nocc)), np.sort(rng.uniform(0.2, 4.0, basis.n - nocc))])
    return np.ascontiguousarray(C), eps


def _options(case):
    return JKOptions.make(prim=PRIM_BELOW, mixed=FP32_BELOW) if case.get("mixed") else JKOptions.make()


def _hamiltonian(n, seed):
    H = np.random.default_rng(seed + 55).standard_normal((n, n))
    return H + H.T


def _gradient_weights(case, basis, seed):
    C = _occupied(basis, _n_occ(case, basis), seed)
    e = np.linspace(-20.0, -0.4, C.shape[1])
    return 2.0 * (C * e) @ C.T


class _Stream:
    """A torch stream that the library's context runs on."""

    def __init__(self):
        self.s = torch.cuda.Stream()

    def __enter__(self):
        self.s.wait_stream(torch.cuda.current_stream())
        return self.s

    def __exit__(self, *a):
        torch.cuda.current_stream().wait_stream(self.s)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "stream": _Stream()}
    raw = st["stream"].s.cuda_stream
    gpu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    empty = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")
    if kind == "batch":
        st["ctx"], st["P"], off = [], [], [0]
        for j in range(case["molecules"]):
            sub = {"kind": "jk", "waters": 1 + j % case["waters"], "basis": case["basis"]}
            basis = _basis(sub, 1000 * seed + j)
            st["ctx"].append(Context(basis, stream=raw))
            st["P"].append(gpu(_densities(sub, basis, 1000 * seed + j)[0]))
            off.append(off[-1] + basis.n ** 2)
        # every molecule's J (and K) one after another in one buffer
        st["J"], st["K"] = empty(off[-1]), empty(off[-1])
        st["pP"] = [t.data_ptr() for t in st["P"]]
        st["pJ"], st["pK"] = ([t.data_ptr() + 8 * o for o in off[:-1]] for t in (st["J"], st["K"]))
        torch.cuda.synchronize()
        return st
    basis = _basis(case, seed)
    n = basis.n
    ctx = st["ctx"] = Context(basis, stream=raw)
    if kind in ("jk", "fshell"):
        P, spins = _densities(case, basis, seed)
        st["P"] = gpu(P)
        st["Ps"] = st["P"] if len(spins) == 1 else gpu(np.stack(spins))
        st["J"], st["K"], st["ns"], st["opts"] = empty(n, n), empty(len(spins), n, n), len(spins), _options(case)
    elif kind == "fock":
        st["P"], st["spins"] = _densities(case, basis, seed)
        st["H"], st["opts"] = _hamiltonian(n, seed), _options(case)
    elif kind == "gradient":
        st["P"], spins = _densities(case, basis, seed)
        st["spins"] = spins if len(spins) == 2 else None
        st["W"] = _gradient_weights(case, basis, seed)
    elif kind == "cholesky":
        st["C"] = _occupied(basis, _n_occ(case, basis), seed)
    elif kind != "scf":
        st["aux"] = CartesianBasis.build(basis.atoms, AUX)
        store = PRECISION[case.get("store", "fp64").replace("fp32", "tf32")]
        if kind == "dfbuild":
            st["store"] = store
        else:
            # whole systems screen the AO pairs as the DF-RHF workload does
            st["df"] = DFTensor(ctx, st["aux"], pair_threshold=1e-10, storage=store)
        if kind == "mp2":
            st["C"], st["eps"] = _mo_space(basis, 5 * case["waters"], seed)
        else:
            st["C"] = _occupied(basis, _n_occ(case, basis), seed)
        if kind == "dfjk":
            st["dC"] = gpu(st["C"].T)  # column-major n x nocc
            st["J"], st["K"] = empty(n, n), empty(n, n)
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind, ctx = case["kind"], st["ctx"]
    if kind in ("jk", "fshell"):
        with st["stream"]:
            ctx.jk_device(st["P"].data_ptr(), st["Ps"].data_ptr(), st["J"].data_ptr(), st["K"].data_ptr(),
                          nspin=st["ns"], opts=st["opts"])
        return [st["J"], st["K"]]
    if kind == "batch":
        with st["stream"] as s:
            Context.jk_device_batch(ctx, st["pP"], st["pJ"], st["pK"], stream=s.cuda_stream)
        return [st["J"], st["K"]]
    if kind == "fock":
        if case["uhf"]:
            return list(ctx.fock_uhf(st["H"], st["spins"][0], st["spins"][1], opts=st["opts"]))
        return [ctx.fock_rhf(st["H"], st["P"], opts=st["opts"])]
    if kind == "gradient":
        return [ctx.gradient(st["P"], st["W"], P_spin=st["spins"])]
    if kind == "dfbuild":
        df = DFTensor(ctx, st["aux"], storage=st["store"])
        out = [df.metric()] + list(df.jk(st["C"], mma=HFG_DF_FP64))
        df.close()
        return out
    if kind == "dfjk":
        with st["stream"]:
            st["df"].jk_device_shard(st["dC"].data_ptr(), st["C"].shape[1], st["J"].data_ptr(), st["K"].data_ptr(), 0, 1,
                                     mma=PRECISION[case["mma"]])
        return [st["J"], st["K"]]
    if kind == "mp2":
        return [np.array([st["df"].mp2_energy(st["C"], st["eps"], 5 * case["waters"])])]
    if kind == "cholesky":
        f, _, _ = DFTensor.cholesky(ctx, case["threshold"])
        out = list(f.jk(st["C"]))
        f.close()
        return out
    r = ctx.scf(tol=1e-10, jk=JKOptions.make(prim=1e-15))
    return [np.array([r["energy"]]), r["P"][0], r["F"][0]]


def tolerance(case):
    kind = case["kind"]
    arith = [case[k] for k in ("store", "mma") if k in case]
    if "bf16" in arith:
        # operands or the stored factor rounded to 8 significant bits
        return {"rel": 6e-3}
    if "tf32" in arith:
        return {"rel": 1e-3}
    if kind == "cholesky":
        # residual diagonals that agree to rounding (like atoms far apart) may
        # be taken in either order: the vectors differ within the threshold
        return {"rel": max(1e-8, 0.3 * case["threshold"])}
    if "fp32" in arith:
        return {"rel": 1e-7}
    if kind in ("dfjk", "dfbuild", "mp2"):
        return {"rel": 2e-10}  # the metric's condition number times 1e-16
    if case.get("mixed"):
        # FP32 below Q_ab Q_cd < 3e-5, primitive products below 1e-13 dropped
        return {"rel": 1e-10}
    if kind == "scf":
        return {"rel": 1e-9}  # converged to 1e-10 Eh
    return {"rel": 1e-12}


# ------------------------------------------------------------------ work ---

def _pair_list(basis, primitive):
    """Rough Schwarz bounds of the shell pairs, or of their primitive pairs:
    (functions, primitive pairs, bound), from Gaussian products."""
    shells = _shells(basis)
    c = np.array([s["r"] for s in shells])
    nf = np.array([s["c"].shape[1] for s in shells])
    if primitive:
        own = np.concatenate([[i] * len(s["a"]) for i, s in enumerate(shells)])
        ex = np.concatenate([s["a"] for s in shells])
        co = np.abs(np.concatenate([s["c"][:, 0] for s in shells]))
        k = np.ones(len(own))
    else:
        own, k = np.arange(len(shells)), np.array([float(len(s["a"])) for s in shells])
        ex, co = np.array([s["a"].min() for s in shells]), np.array([np.max(np.abs(s["c"][:, 0])) for s in shells])
    a, b = np.tril_indices(len(own))
    r2 = ((c[own[a]] - c[own[b]]) ** 2).sum(1)
    p = ex[a] + ex[b]
    q = np.minimum(co[a] * co[b] * np.exp(-ex[a] * ex[b] / p * r2) * 6.0 * p ** -1.25, 5.0)
    return (nf[own[a]] * nf[own[b]]).astype(float), k[a] * k[b], q


def _quartet_work(basis, eps=0.0):
    """Flops of the screened quartets: Boys values and prefactors, one
    contribution per integral and primitive quartet (those above eps), and
    the six density contractions of the finished integrals."""
    def over(q, thr, x, y):
        o = np.argsort(-q)
        cnt = np.searchsorted(-q[o], -(thr / np.maximum(q[o], 1e-300)))
        return 0.5 * float(np.sum(x[o] * np.concatenate([[0.0], np.cumsum(y[o])])[cnt]))
    nf, npp, q = _pair_list(basis, False)
    done = 12.0 * over(q, 1e-12, nf, nf)
    if eps > 0.0:
        nf, npp, q = _pair_list(basis, True)
    thr = max(eps, 1e-12) if eps > 0.0 else 1e-12
    return done + 60.0 * over(q, thr, npp, npp) + 4.0 * over(q, thr, npp * nf, npp * nf)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        subs = [{"kind": "jk", "waters": 1 + j % case["waters"], "basis": case["basis"]} for j in range(case["molecules"])]
        bs = [_basis(s, 1) for s in subs[:case["waters"]]]
        each = [{"bytes": 8.0 * 3 * b.n ** 2, "flops": _quartet_work(b)} for b in bs]
        return {k: sum(each[j % len(each)][k] for j in range(case["molecules"])) for k in ("bytes", "flops")}
    basis = _basis(case, 1)
    n = basis.n
    if kind in ("jk", "fock", "fshell"):
        ns = 2 if case.get("uhf") else 1
        return {"bytes": 8.0 * n * n * (2 + 2 * ns), "flops": _quartet_work(basis, 1e-12 if case.get("mixed") else 0.0)}
    if kind == "gradient":
        return {"bytes": 8.0 * n * n * 3, "flops": 3.0 * _quartet_work(basis)}
    if kind == "scf":
        return {"bytes": 8.0 * n * n * 20, "flops": 12.0 * (_quartet_work(basis) + 30.0 * n ** 3)}
    nocc, np_ = 5 * case["waters"], n * (n + 1) // 2
    if kind == "cholesky":
        rank = 6.0 * n
        return {"bytes": 8.0 * (0.5 * np_ * np_ + 2.0 * rank * np_),
                "flops": _quartet_work(basis) + np_ * rank ** 2 + 4.0 * n * n * nocc * rank}
    na = CartesianBasis.build(basis.atoms, AUX).n
    size = {"fp64": 8.0, "fp32": 4.0, "bf16": 2.0}[case.get("store", "fp64")]
    jk = 4.0 * na * np_ + 2.0 * na * n * n * nocc + na * nocc * n * n
    if kind == "dfbuild":
        return {"bytes": 8.0 * na * na + 2.0 * size * na * np_, "flops": 9.0 * na ** 3 + 2.0 * na * na * np_ + jk}
    if kind == "dfjk":
        return {"bytes": size * na * np_ + 16.0 * n * n, "flops": jk}
    nv = n - nocc
    return {"bytes": size * na * np_ + 8.0 * n * n,
            "flops": na * (2.0 * n * n * nocc + 2.0 * n * nocc * nv) + na * (nocc * nv) ** 2}


# ----------------------------------------------------------------- exact ---
# Integrals from their definition in 64-bit torch: Hermite expansions of whole
# classes of shell pairs, the auxiliary integrals R_tuv, and two contractions.

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _shells(basis):
    out, f = [], 0
    while f < basis.n:
        l = int(basis.lxyz[f].sum())
        nc = (l + 1) * (l + 2) // 2
        sl = [slice(basis.prim_off[f + i], basis.prim_off[f + i + 1]) for i in range(nc)]
        out.append({"l": l, "f": f, "r": basis.center[f], "atom": int(basis.atom[f]), "a": basis.exps[sl[0]],
                    "c": np.stack([basis.coefs[s] for s in sl], 1)})
        f += nc
    return out


class _Boys(torch.autograd.Function):
    """F_0(T) .. F_m(T): a series and downward recursion to T = 36, the error
    function and upward recursion beyond; dF_k/dT = -F_{k+1}."""

    @staticmethod
    def forward(ctx, T, m):
        t = T.clamp(max=36.0)
        e = torch.exp(-t)
        term = torch.full_like(t, 1.0 / (2 * m + 3))
        s = term.clone()
        for i in range(1, 170):
            term = term * (2.0 * t / (2 * m + 3 + 2 * i))
            s += term
        F = [None] * (m + 2)
        F[m + 1] = e * s
        for k in range(m, -1, -1):
            F[k] = (2.0 * t * F[k + 1] + e) / (2 * k + 1)
        tb, eb = T.clamp(min=36.0), torch.exp(-T.clamp(min=36.0))
        g = 0.5 * torch.sqrt(math.pi / tb)
        big = T > 36.0
        for k in range(m + 2):
            F[k] = torch.where(big, g, F[k])
            g = ((2 * k + 1) * g - eb) / (2.0 * tb)
        ctx.save_for_backward(*F)
        return torch.stack(F[:m + 1])

    @staticmethod
    def backward(ctx, grad):
        F = ctx.saved_tensors
        return -sum(grad[k] * F[k + 1] for k in range(len(F) - 1)), None


def _herm(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _axis_tables(la, lb, a, b, A, B):
    """E[i][j][t], tensors over primitive pairs x 3 axes (prefactor apart)."""
    p = (a + b)[:, None]
    P = (a[:, None] * A + b[:, None] * B) / p
    E = {(0, 0, 0): torch.ones_like(P)}
    get = lambda i, j, t: E.get((i, j, t), 0.0)
    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j:
                x, q = (P - A, (i - 1, j)) if i else (P - B, (i, j - 1))
                for t in range(i + j + 1):
                    E[i, j, t] = get(*q, t - 1) / (2.0 * p) + x * get(*q, t) + (t + 1) * get(*q, t + 1)
    return E, P


def _pair_classes(sa, sb, pos=None):
    """Shell pairs of the lists sa x sb (sb None: unique pairs of sa) by class;
    an entry of sb that is "unit" pairs with the constant 1.  pos: differentiable
    atom positions that replace the shells' centres."""
    dev = _dev()
    groups = {}
    for i, s in enumerate(sa):
        for j, t in enumerate(sa[:i + 1] if sb is None else sb):
            x, y = (t, s) if t["l"] > s["l"] and sb is None else (s, t)
            groups.setdefault((x["l"], len(x["a"]), y["l"], len(y["a"])), []).append((x, y, 2.0 if sb is None and i != j else 1.0))
    out = []
    for (la, ka, lb, kb), prs in sorted(groups.items()):
        T = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device=dev)
        if pos is None:
            A, B = T([x["r"] for x, _, _ in prs]), T([y["r"] for _, y, _ in prs])
        else:
            A, B = pos[[x["atom"] for x, _, _ in prs]], pos[[y["atom"] for _, y, _ in prs]]
        N, nk = len(prs), ka * kb
        ex = lambda v, i: T([p[i]["a"] for p in prs])
        a = ex(None, 0)[:, :, None].expand(N, ka, kb).reshape(-1)
        b = ex(None, 1)[:, None, :].expand(N, ka, kb).reshape(-1)
        ca, cb = T([p[0]["c"] for p in prs]), T([p[1]["c"] for p in prs])  # N, K, ncomp
        cc = torch.einsum("nka,nlb->nklab", ca, cb).reshape(N * nk, ca.shape[2] * cb.shape[2])
        A, B = A.repeat_interleave(nk, 0), B.repeat_interleave(nk, 0)
        E, P = _axis_tables(la, lb, a, b, A, B)
        K = torch.exp(-a * b / (a + b) * ((A - B) ** 2).sum(1))
        zero = torch.zeros_like(K)
        rows = []
        for xa in cartesian_components(la):
            for xb in cartesian_components(lb):
                rows.append(torch.stack([E[xa[0], xb[0], t][:, 0] * E[xa[1], xb[1], u][:, 1] * E[xa[2], xb[2], v][:, 2]
                                         if t <= xa[0] + xb[0] and u <= xa[1] + xb[1] and v <= xa[2] + xb[2] else zero
                                         for t, u, v in _herm(la + lb)], 1))
        H = torch.stack(rows, 1) * (cc * K[:, None])[:, :, None]  # prim, ab, hermite
        comp = lambda s: torch.arange((s + 1) * (s + 2) // 2, device=dev)
        fa = torch.tensor([p[0]["f"] for p in prs], device=dev)[:, None] + comp(la)
        fb = torch.tensor([p[1]["f"] for p in prs], device=dev)[:, None] + comp(lb)
        out.append({"L": la + lb, "N": N, "nk": nk, "p": a + b, "P": P, "H": H, "fa": fa, "fb": fb,
                    "w": T([p[2] for p in prs]), "E": E, "a": a, "b": b, "cc": cc, "K": K, "l": (la, lb)})
    return out


def _r_table(L, PQ, alpha):
    """R_tuv(alpha, PQ) for t + u + v <= L, stacked over _herm(L)."""
    F = _Boys.apply(alpha * (PQ ** 2).sum(-1), L)
    R = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * F[n]}
        for t, u, v in sorted(_herm(L - n), key=sum)[1:]:
            ax = 0 if t else (1 if u else 2)
            k = [t, u, v]
            k[ax] -= 1
            r = PQ[..., ax] * R[tuple(k)]
            if k[ax]:
                k2 = list(k)
                k2[ax] -= 1
                r = r + k[ax] * R[tuple(k2)]
            new[t, u, v] = r
        R = new
    return torch.stack([R[h] for h in _herm(L)], -1)


def _blocks(X, Y, budget=3e7):
    """(pairs of X, block[pair of X, ab, pair of Y, cd]) over chunks of X."""
    hx, hy, dev = _herm(X["L"]), _herm(Y["L"]), X["p"].device
    index = {h: i for i, h in enumerate(_herm(X["L"] + Y["L"]))}
    idx = torch.tensor([[index[tuple(np.add(h, k))] for k in hy] for h in hx], device=dev)
    sign = torch.tensor([(-1.0) ** sum(k) for k in hy], dtype=torch.float64, device=dev)
    Hy = Y["H"] * sign
    step = max(1, int(budget / (X["nk"] * len(Y["p"]) * max(idx.numel(), 4 * len(index)))))
    for x0 in range(0, X["N"], step):
        x1 = min(X["N"], x0 + step)
        s = slice(x0 * X["nk"], x1 * X["nk"])
        p, q = X["p"][s, None], Y["p"][None, :]
        R = _r_table(X["L"] + Y["L"], X["P"][s, None, :] - Y["P"][None, :, :], p * q / (p + q))
        R = R * (2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)))[..., None]
        R = R.view(x1 - x0, X["nk"], Y["N"], Y["nk"], -1)[..., idx]  # x, k, y, m, hx, hy
        Z = torch.einsum("xkymhg,ymcg->xkyhc", R, Hy.view(Y["N"], Y["nk"], -1, len(hy)))
        yield slice(x0, x1), torch.einsum("xkyhc,xkah->xayc", Z, X["H"][s].view(x1 - x0, X["nk"], -1, len(hx)))


def _eri4(basis):
    n = basis.n
    V = torch.zeros((n, n, n, n), dtype=torch.float64, device=_dev())
    cls = _pair_classes(_shells(basis), None)
    for i, X in enumerate(cls):
        for Y in cls[:i + 1]:
            for s, blk in _blocks(X, Y):
                fa, fb = X["fa"][s], X["fb"][s]
                m = blk.view(len(fa), fa.shape[1], fb.shape[1], Y["N"], Y["fa"].shape[1], Y["fb"].shape[1])
                a, b = fa[:, :, None, None, None, None], fb[:, None, :, None, None, None]
                c, d = Y["fa"][None, None, None, :, :, None], Y["fb"][None, None, None, :, None, :]
                for w, x in ((a, b), (b, a)):
                    for y, z in ((c, d), (d, c)):
                        V[w, x, y, z] = m
                        V[y, z, w, x] = m
    return V


def _one_electron(basis, pos):
    """S and T + V (torch, differentiable in pos)."""
    n, dev = basis.n, pos.device
    S, H = (torch.zeros((n, n), dtype=torch.float64, device=dev) for _ in range(2))
    Z = torch.tensor(basis.nuclear_charges(), dtype=torch.float64, device=dev)
    for X in _pair_classes(_shells(basis), None, pos):
        la, lb = X["l"]
        # centres again, for the tables raised by two in b
        A, B = (pos[torch.tensor(basis.atom, device=dev).long()[f[:, 0]]].repeat_interleave(X["nk"], 0)
                for f in (X["fa"], X["fb"]))
        E, _ = _axis_tables(la, lb + 2, X["a"], X["b"], A, B)
        s1 = lambda i, j, ax: E[i, j, 0][:, ax] if j >= 0 else 0.0
        be = X["b"]
        t1 = lambda i, j, ax: (be * (2 * j + 1) * s1(i, j, ax) - 2.0 * be ** 2 * s1(i, j + 2, ax)
                               - 0.5 * j * (j - 1) * s1(i, j - 2, ax))
        pref = (math.pi / X["p"]) ** 1.5 * X["K"]
        sb, tb = [], []
        for xa in cartesian_components(la):
            for xb in cartesian_components(lb):
                s = [s1(xa[k], xb[k], k) for k in range(3)]
                t = [t1(xa[k], xb[k], k) for k in range(3)]
                sb.append(s[0] * s[1] * s[2])
                tb.append(t[0] * s[1] * s[2] + s[0] * t[1] * s[2] + s[0] * s[1] * t[2])
        R = _r_table(X["L"], X["P"][:, None, :] - pos[None], X["p"][:, None].expand(-1, len(Z)))
        V = -torch.einsum("pzh,z,pah->pa", R, Z, X["H"]) * (2.0 * math.pi / X["p"])[:, None]
        w = X["cc"] * pref[:, None]
        blk_s = (torch.stack(sb, 1) * w).view(X["N"], X["nk"], -1).sum(1)
        blk_h = (torch.stack(tb, 1) * w + V).view(X["N"], X["nk"], -1).sum(1)
        i = X["fa"][:, :, None].expand(-1, -1, X["fb"].shape[1]).reshape(-1)
        j = X["fb"][:, None, :].expand(-1, X["fa"].shape[1], -1).reshape(-1)
        S = S.index_put((i, j), blk_s.reshape(-1)).index_put((j, i), blk_s.reshape(-1))
        H = H.index_put((i, j), blk_h.reshape(-1)).index_put((j, i), blk_h.reshape(-1))
    return S, H


def _nuclear(basis, pos):
    Z = torch.tensor(basis.nuclear_charges(), dtype=torch.float64, device=pos.device)
    i, j = torch.triu_indices(len(Z), len(Z), 1)
    return (Z[i] * Z[j] / torch.linalg.norm(pos[i] - pos[j], dim=1)).sum()


def _jk(V, P, spins):
    return torch.einsum("abcd,cd->ab", V, P), [torch.einsum("acbd,cd->ab", V, s) for s in spins]


def _factor(basis, aux, cutoff=1e-10):
    """B[Q, m, n] of the Cartesian auxiliary basis."""
    unit = {"l": 0, "f": 0, "r": np.zeros(3), "a": np.zeros(1), "c": np.ones((1, 1))}
    ax = _pair_classes(_shells(aux), [unit])
    # the constant carries no exponent: the product centre is the shell's
    M = torch.zeros((aux.n, aux.n), dtype=torch.float64, device=_dev())
    T = torch.zeros((aux.n, basis.n, basis.n), dtype=torch.float64, device=_dev())
    for X in ax:
        for Y in ax:
            for s, blk in _blocks(X, Y):
                M[X["fa"][s][:, :, None, None], Y["fa"][None, None]] = blk
        for Y in _pair_classes(_shells(basis), None):
            for s, blk in _blocks(X, Y):
                blk = blk.view(*blk.shape[:3], Y["fa"].shape[1], Y["fb"].shape[1])
                q = X["fa"][s][:, :, None, None, None]
                a, b = Y["fa"][None, None, :, :, None], Y["fb"][None, None, :, None, :]
                T[q, a, b] = blk
                T[q, b, a] = blk
    w, U = torch.linalg.eigh(M)
    keep = w > cutoff
    return M, torch.einsum("pq,pmn->qmn", U[:, keep] * w[keep] ** -0.5, T)


def _factor_jk(B, C):
    P = 2.0 * C @ C.T
    J = torch.einsum("q,qmn->mn", torch.einsum("qmn,mn->q", B, P), B)
    U = torch.einsum("qmn,ni->qmi", B, C)
    return J, 2.0 * torch.einsum("qmi,qni->mn", U, U)


def _exact_gradient(case, basis, seed):
    t = lambda a: torch.tensor(np.array(a), dtype=torch.float64, device=_dev())
    P, spins = _densities(case, basis, seed)
    x = 0.25 if len(spins) == 1 else 0.5
    W, P, spins = t(_gradient_weights(case, basis, seed)), t(P), [t(s) for s in spins]
    pos = t(basis.positions()).requires_grad_(True)
    S, H = _one_electron(basis, pos)
    g = torch.autograd.grad((P * H).sum() - (W * S).sum() + _nuclear(basis, pos), pos)[0]
    cls = _pair_classes(_shells(basis), None, pos)
    for i, X in enumerate(cls):
        for j, Y in enumerate(cls[:i + 1]):
            for s, blk in _blocks(X, Y, budget=1e7):
                fa, fb = X["fa"][s], X["fb"][s]
                m = blk.view(len(fa), fa.shape[1], fb.shape[1], Y["N"], Y["fa"].shape[1], Y["fb"].shape[1])
                a, b = fa[:, :, None, None, None, None], fb[:, None, :, None, None, None]
                c, d = Y["fa"][None, None, None, :, :, None], Y["fb"][None, None, None, :, None, :]
                G = P[a, b] * P[c, d]
                for D in spins:
                    G = G - x * (D[a, c] * D[b, d] + D[a, d] * D[b, c])
                wgt = X["w"][s][:, None, None, None, None, None] * Y["w"][None, None, None, :, None, None]
                e = 0.5 * (1.0 if i == j else 2.0) * (wgt * m * G).sum()
                g = g + torch.autograd.grad(e, pos, retain_graph=True)[0]
    return [g.cpu().numpy()]


def _exact_cholesky(case, basis, seed):
    n = basis.n
    i, j = np.tril_indices(n)
    ti, tj = torch.tensor(i, device=_dev()), torch.tensor(j, device=_dev())
    V = _eri4(basis)[ti, tj][:, ti, tj]
    d = V.diagonal().clone()
    rows = []
    while True:
        big = d.max()
        k = int(torch.nonzero(d >= big - 1e-12 * big.abs())[0, 0])
        if float(d[k]) <= case["threshold"]:
            break
        r = V[k].clone()
        if rows:
            Lm = torch.stack(rows)
            r -= Lm[:, k] @ Lm
        r /= torch.sqrt(d[k])
        d = (d - r * r).clamp(min=0.0)
        d[k] = 0.0
        rows.append(r)
    B = torch.zeros((len(rows), n, n), dtype=torch.float64, device=_dev())
    B[:, ti, tj] = torch.stack(rows)
    B[:, tj, ti] = torch.stack(rows)
    J, K = _factor_jk(B, torch.tensor(_occupied(basis, _n_occ(case, basis), seed), device=_dev()))
    return [J.cpu().numpy(), K.cpu().numpy()]


def _exact_scf(basis, nocc):
    pos = torch.tensor(basis.positions(), dtype=torch.float64, device=_dev())
    V = _eri4(basis)
    S, H = _one_electron(basis, pos)
    w, U = torch.linalg.eigh(S)
    X = U[:, w > 1e-8] * w[w > 1e-8] ** -0.5
    F, fs, es = H, [], []
    for it in range(60):
        C = X @ torch.linalg.eigh(X.T @ F @ X)[1][:, :nocc]
        P = 2.0 * C @ C.T
        J, (K,) = _jk(V, P, [P])
        F0 = H + J - 0.5 * K
        e = X.T @ (F0 @ P @ S - S @ P @ F0) @ X
        if float(e.abs().max()) < 1e-12:
            break
        fs, es = (fs + [F0])[-8:], (es + [e])[-8:]
        m = len(fs)
        A = -torch.ones((m + 1, m + 1), dtype=torch.float64, device=_dev())
        A[m, m] = 0.0
        A[:m, :m] = torch.stack([torch.stack([(x * y).sum() for y in es]) for x in es])
        b = torch.zeros(m + 1, dtype=torch.float64, device=_dev())
        b[m] = -1.0
        scale = A[:m, :m].diagonal().max()
        A[:m, :m] /= scale
        F = sum(c * f for c, f in zip(torch.linalg.lstsq(A.cpu(), b.cpu()[:, None], driver="gelsd").solution[:m, 0].tolist(), fs))
    energy = 0.5 * (P * (H + F0)).sum() + _nuclear(basis, pos)
    return [np.array([float(energy)]), P.cpu().numpy(), F0.cpu().numpy()]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None
    basis = _basis(case, seed)
    limit = {"jk": 133, "fock": 133, "fshell": 80, "gradient": 50, "cholesky": 75, "scf": 75, "dfbuild": 230, "dfjk": 230,
             "mp2": 150}[kind]
    if basis.n > limit:
        return None  # the dense integrals take minutes
    host = lambda x: x.cpu().numpy()
    t = lambda a: torch.tensor(np.array(a), dtype=torch.float64, device=_dev())
    if kind in ("jk", "fshell", "fock"):
        P, spins = _densities(case, basis, seed)
        J, K = _jk(_eri4(basis), t(P), [t(s) for s in spins])
        if kind != "fock":
            return [host(J), host(torch.stack(K))]
        H, k = t(_hamiltonian(basis.n, seed)), 1.0 if case["uhf"] else 0.5
        return [host(H + J - k * x) for x in K]
    if kind == "gradient":
        return _exact_gradient(case, basis, seed)
    if kind == "cholesky":
        return _exact_cholesky(case, basis, seed)
    if kind == "scf":
        return _exact_scf(basis, 5 * case["waters"])
    M, B = _factor(basis, CartesianBasis.build(basis.atoms, AUX))
    if kind == "mp2":
        C, eps = _mo_space(basis, 5 * case["waters"], seed)
        C, eps, o = t(C), t(eps), 5 * case["waters"]
        ov = torch.einsum("mi,qmn,na->qia", C[:, :o], B, C[:, o:])
        v = torch.einsum("qia,qjb->iajb", ov, ov)
        gap = (eps[:o, None, None, None] - eps[None, o:, None, None] + eps[None, None, :o, None]
               - eps[None, None, None, o:])
        return [np.array([float((v * (2.0 * v - v.transpose(1, 3)) / gap).sum())])]
    J, K = _factor_jk(B, t(_occupied(basis, _n_occ(case, basis), seed)))
    return ([host(M)] if kind == "dfbuild" else []) + [host(J), host(K)]
