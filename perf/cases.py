"""The workloads this library's speed is measured on.

Every case calls the public entry points (``pynof_gb300.ops``, ``.integrals``,
``.batch``) the way the solver, the batched builds and the PyNOF drop-in call
them, on seeded inputs of the library's own recipe (``synthetic.py``): b a
Gaussian scaled by exp(-0.05 (m + n)) and symmetrised in (m, n), C orthogonal,
H symmetric, occupations sorted descending.  Sizes follow the configurations
of ``synthetic.WORKLOADS`` and ``bench.py`` (nbf 24..600, naux about 4 nbf,
nbf5 about nbf / 2) and odd sizes between them.

Kinds:

* ``jk``      J_i, K_i of every occupied orbital (computeJKj, RI), the build
              the library's headline is quoted on; ``form`` is the arithmetic:
              "s6" (six digit slices, the default), "bf16x3", "tf32x3" or
              "fp64".
* ``dropin``  the same build through PyNOF's own function: numpy orbitals in,
              numpy J, K out.
* ``step``    one step of the orbital optimiser: C expm(Y), then J_MO, K_MO,
              H_core and the Lagrangian at the new orbitals in one call.
* ``mo``      J_MO, K_MO, H_core alone (computeJKH_MO), what the occupation
              optimiser starts from.
* ``lag``     the Lagrangian on the FP64 path: the closing pass of a solve.
* ``ao``      the four-index route: J, K from (mn|sl), the generalized Fock
              matrices, the Lagrangian from them and the electronic energy.
* ``occ``     the occupation optimiser's minimisation (occoptr).
* ``batch``   J, K of many molecules of uneven size from one recorded graph.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from pynof_gb300 import batch, integrals, nof, ops, synthetic

DEV = "cuda"
F64 = torch.float64
SLICES = {"s6": 6, "bf16x3": 2, "tf32x3": ops.SPLIT_TF32X3}


def listed():
    return [
        # water / cc-pVDZ: the smallest molecule, all launch latency
        {"name": "jk_24", "kind": "jk", "nbf": 24, "naux": 116, "nbf5": 24, "form": "s6"},
        # an ordinary molecule, no size a multiple of anything
        {"name": "jk_171", "kind": "jk", "nbf": 171, "naux": 683, "nbf5": 85, "form": "s6"},
        # the headline build
        {"name": "jk_600", "kind": "jk", "nbf": 600, "naux": 2400, "nbf5": 300, "form": "s6"},
        # the low rung of a precision ladder
        {"name": "jk_300_bf16x3", "kind": "jk", "nbf": 300, "naux": 1200, "nbf5": 150, "form": "bf16x3"},
        # PyNOF itself calling computeJKj behind p.gpu
        {"name": "dropin_300", "kind": "dropin", "nbf": 300, "naux": 1200, "nbf5": 150},
        # orbital steps of a small and of a medium served molecule
        {"name": "step_53", "kind": "step", "nbf": 53, "naux": 212, "nbf5": 25},
        {"name": "step_300", "kind": "step", "nbf": 300, "naux": 1200, "nbf5": 150},
        # MO integrals of a large ragged molecule before its occupation step
        {"name": "mo_411", "kind": "mo", "nbf": 411, "naux": 1644, "nbf5": 205, "form": "s6"},
        # the closing FP64 Lagrangian of a medium solve
        {"name": "lag_fp64_300", "kind": "lag", "nbf": 300, "naux": 1200, "nbf5": 150},
        # the four-index route (no density fitting) of a small molecule
        {"name": "ao_120", "kind": "ao", "nbf": 120, "nbf5": 60},
        # occupations of a medium molecule at fixed orbitals
        {"name": "occ_150", "kind": "occ", "nbf": 300, "naux": 1200, "ndoc": 30, "ncwo": 4},
        # a batch of uneven molecules in one graph
        {"name": "batch_24", "kind": "batch", "count": 24, "lo": 24, "hi": 250, "sizes": 7},
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ri(rng: random.Random, lo: int, hi: int) -> dict:
    nbf = _log(rng, lo, hi)
    return {"nbf": nbf, "naux": int(round(nbf * rng.uniform(3.6, 4.8))) if nbf < 400 else 4 * nbf,
            "nbf5": max(4, int(round(nbf * rng.uniform(0.4, 0.5)))) if nbf > 40 else nbf}


def draw(rng):
    kind = rng.choice(["jk", "jk", "jk", "step", "step", "mo", "dropin", "lag", "ao", "occ", "batch"])
    if kind == "jk":
        form = rng.choice(["s6", "s6", "s6", "bf16x3", "tf32x3", "fp64"])
        return {"kind": "jk", **_ri(rng, 24, 250 if form == "fp64" else 560), "form": form}
    if kind == "step":
        return {"kind": "step", **_ri(rng, 24, 420)}
    if kind == "mo":
        return {"kind": "mo", **_ri(rng, 24, 500), "form": rng.choice(["s6", "s6", "bf16x3", "tf32x3", "fp64"])}
    if kind == "dropin":
        return {"kind": "dropin", **_ri(rng, 24, 420)}
    if kind == "lag":
        return {"kind": "lag", **_ri(rng, 24, 260)}
    if kind == "ao":
        nbf = _log(rng, 24, 118)
        return {"kind": "ao", "nbf": nbf, "nbf5": max(4, int(round(nbf * rng.uniform(0.4, 0.5))))}
    if kind == "occ":
        nbf = _log(rng, 40, 240)
        return {"kind": "occ", "nbf": nbf, "naux": 4 * nbf, "ndoc": max(1, nbf // 10), "ncwo": rng.choice([3, 4])}
    return {"kind": "batch", "count": rng.randint(5, 24), "lo": 24, "hi": rng.randint(60, 240),
            "sizes": rng.randint(0, 10**6)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator().manual_seed(int(seed) + 1)


def _factor(nbf: int, naux: int, seed: int) -> torch.Tensor:
    """b (nbf, nbf, naux), exactly symmetric in its first two indices."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    b = torch.randn((nbf, nbf, naux), dtype=F64, device=DEV, generator=g)
    e = torch.exp(-0.05 * torch.arange(nbf, dtype=F64, device=DEV))
    b.mul_(e[:, None, None]).mul_(e[None, :, None])
    return (b + b.transpose(0, 1)).mul_(0.5)


def _orbitals(nbf: int, g: torch.Generator) -> torch.Tensor:
    return torch.linalg.qr(torch.randn((nbf, nbf), dtype=F64, generator=g))[0].contiguous()


def _core(nbf: int, g: torch.Generator) -> torch.Tensor:
    a = torch.randn((nbf, nbf), dtype=F64, generator=g)
    return 0.5 * (a + a.T)


def _occupations(nbf5: int, g: torch.Generator):
    """n (descending) and coupling matrices with the zero diagonals the
    solver hands over."""
    n = torch.rand(nbf5, dtype=F64, generator=g).sort(descending=True).values
    ck = torch.outer(n, n)
    ck.fill_diagonal_(0.0)
    return n, 2.0 * ck, ck


def _prep(b: torch.Tensor, form: str):
    return b if form == "fp64" else ops.PreparedRI(b, SLICES[form])


def _half(nbf5: int) -> int:
    """Doubly occupied orbitals of nbf5 (one in five, as the solver's structures)."""
    return max(1, nbf5 // 5)


def _structure(case: dict) -> synthetic.Structure:
    nbf5 = case["nbf5"]
    return synthetic.Structure(nbf=case["nbf"], nbfaux=case["naux"], ndoc=1, ncwo=nbf5 - 1)


def _molecules(case: dict):
    return [(n, 4 * n, max(1, n // 10) * 5) for n in
            synthetic.batch_sizes(case["count"], case["lo"], case["hi"], case["sizes"])]


def _parts(case: dict, seed: int) -> dict:
    """The seeded inputs of a case, on the GPU (C also on the host)."""
    kind, g = case["kind"], _gen(seed)
    if kind == "batch":
        mols = []
        for i, (nbf, naux, nbf5) in enumerate(_molecules(case)):
            mols.append((_orbitals(nbf, g).to(DEV), _factor(nbf, naux, 1000 * seed + i), nbf5))
        return {"mols": mols}
    nbf = case["nbf"]
    C, H = _orbitals(nbf, g), _core(nbf, g)
    s = {"C_host": C, "C": C.to(DEV), "H": H.to(DEV)}
    if kind == "occ":
        st = synthetic.Structure(nbf=nbf, nbfaux=case["naux"], ndoc=case["ndoc"], ncwo=case["ncwo"])
        s["st"], s["b"] = st, _factor(nbf, case["naux"], seed)
        return s
    n, cj, ck = _occupations(case["nbf5"], g)
    s.update(n=n.to(DEV), cj=cj.to(DEV), ck=ck.to(DEV))
    if kind == "ao":
        # (mn|sl) of a factorised operator: the 8-fold symmetry of real integrals
        f = _factor(nbf, 2 * nbf, seed).view(nbf * nbf, 2 * nbf)
        s["I"] = (f @ f.T).view(nbf, nbf, nbf, nbf)
        return s
    s["b"] = _factor(nbf, case["naux"], seed)
    if kind == "step":
        nvar = nbf * (nbf - 1) // 2 - (nbf - case["nbf5"]) * (nbf - case["nbf5"] - 1) // 2
        # AMSgrad steps: every element of about the learning rate's size
        y = 0.02 * (2.0 * torch.rand(nvar, dtype=F64, generator=g) - 1.0)
        s["y"] = y.to(DEV)
        s["norm1"] = ops.AntisymNorm(nbf, case["nbf5"])(y.numpy())
    return s


def prepare(case, seed):
    kind, s = case["kind"], _parts(case, seed)
    s["kind"] = kind
    if kind == "batch":
        mols = [(C, ops.PreparedRI(b, 6), nbf5) for C, b, nbf5 in s.pop("mols")]
        s["plan"] = batch.BatchJK(mols, tiles=(3, 3))
        return s
    if kind == "occ":
        st, b = s["st"], s.pop("b")
        s["J"], s["K"], s["Hc"] = _mo64(s["C"], s["H"], b, st.nbf5)
        s["gamma"] = torch.as_tensor(nof.gamma_guess_softmax(st), dtype=F64).to(DEV)
        s["om"] = ops.OccMinimizer(st.nbf5, st.no1, st.ndoc, st.ncwo, DEV)
        return s
    s["nbf5"], s["ndoc"] = case["nbf5"], _half(case["nbf5"])
    s["form"] = case.get("form")
    if kind in ("jk", "mo"):
        s["prep"] = _prep(s.pop("b"), case["form"])
    elif kind == "step":
        s["prep"] = _prep(s.pop("b"), "s6")
    elif kind == "dropin":
        s["C_host"], s["p"] = s["C_host"].numpy(), _structure(case)
        integrals.prepared(s["b"], integrals.PRECISION["nslices"])
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    s, kind = state, state["kind"]
    if kind == "batch":
        here, plan = torch.cuda.current_stream(), s["plan"]
        plan.stream.wait_stream(here)
        plan.run()
        here.wait_stream(plan.stream)
        return {"J": plan.J, "K": plan.K}
    if kind == "occ":
        gamma, result, n, cj, ck = s["om"].minimize(s["gamma"], s["J"], s["K"], s["Hc"])
        return {"gamma": gamma, "result": result, "n": n, "cj12": cj, "ck12": ck}
    P, nd = s["nbf5"], s["ndoc"]
    if kind == "jk":
        J, K = ops.jkj_ri(s["C"], s["prep"], P) if s["form"] == "fp64" else ops.jkj_ri_mixed(s["C"], s["prep"], P)
        return {"J": J, "K": K}
    if kind == "dropin":
        J, K = integrals.computeJKj(s["C_host"], None, s["b"], s["p"])
        return {"J": J, "K": K}
    if kind == "mo":
        mo = ops.jkh_mo_ri if s["form"] == "fp64" else ops.jkh_mo_ri_mixed
        J, K, Hc = mo(s["C"], s["H"], s["prep"], P)
        return {"J": J, "K": K, "Hc": Hc}
    if kind == "step":
        C = ops.rotate_orbital(s["y"], s["C"], P, norm1=s["norm1"])
        J, K, Hc, elag, Hmat = ops.jkh_lagrange2_ri_mixed(C, s["H"], s["prep"], s["n"], s["cj"], s["ck"], P, nd, nd)
        return {"C": C, "J": J, "K": K, "Hc": Hc, "elag": elag, "Hmat": Hmat}
    if kind == "lag":
        elag, Hmat = ops.lagrange2_ri(s["C"], s["H"], s["b"], s["n"], s["cj"], s["ck"], P, nd, nd)
        return {"elag": elag, "Hmat": Hmat}
    J, K = ops.jkj_full(s["C"], s["I"], P)
    F = ops.fock_rc(J, K, s["n"], s["H"], s["cj"], s["ck"], nd, nd)
    elag = ops.lagrange(F, s["C"])
    E = ops.energy_elec(elag, s["C"], s["H"], s["n"], nd, nd)
    return {"J": J, "K": K, "F": F, "elag": elag, "E": E}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Operands read once and results written once, as float64; the flops of
    the contractions with their (m, n) / (p, q) symmetry used."""
    kind = case["kind"]
    if kind == "batch":
        ws = [work({"kind": "jk", "nbf": n, "naux": q, "nbf5": p}) for n, q, p in _molecules(case)]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    N = float(case["nbf"])
    if kind == "occ":
        P = float(case["ndoc"] * (case["ncwo"] + 1))
        return {"bytes": 8 * 4 * P * P, "flops": 10 * P * P}  # of one evaluation; the iterations follow from the data
    P = float(case["nbf5"])
    if kind == "ao":
        pairs = N * (N + 1) / 2
        return {"bytes": 8 * (N**4 + 3 * P * N * N + N * N), "flops": 2 * 2 * P * pairs * N * N + 2 * 2 * P * P * N * N}
    Q = float(case["naux"])
    half = 2 * P * N * N * Q
    if kind in ("jk", "dropin"):
        return {"bytes": 8 * (N * N * Q + 2 * P * N * N), "flops": 2 * half}
    to_mo = 2 * P * P * N * Q  # (pq|l), p, q < nbf5
    if kind == "mo":
        return {"bytes": 8 * (N * N * Q + 2 * P * P), "flops": half + to_mo / 2 + 2 * P * P * Q}
    # the Lagrangian: half transform, MO transform, exchange contraction over (q, l)
    lag = half + to_mo / 2 + 2 * N * P * P * Q
    rot = 0.0 if kind == "lag" else 2 * 10 * N**3
    return {"bytes": 8 * (N * N * Q + 3 * N * N + 4 * P * P), "flops": lag + rot}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _jk64(C, b, P):
    N, _, Q = b.shape
    T = (C[:, :P].T.contiguous() @ b.view(N, N * Q)).view(P, N, Q)
    d = torch.einsum("nq,qnl->ql", C[:, :P], T)
    return (d @ b.view(N * N, Q).T).view(P, N, N), T @ T.transpose(1, 2)


def _bmo64(C, b, P):
    """(aq|l) for every a and q < nbf5, as (nbf, nbf5, naux)."""
    N, _, Q = b.shape
    T = (C[:, :P].T.contiguous() @ b.view(N, N * Q)).view(P, N, Q)
    return (C.T.contiguous() @ T.transpose(0, 1).reshape(N, P * Q)).view(N, P, Q)


def _mo64(C, H, b, P):
    """J_MO, K_MO, H_core, made on the way to an occupation problem."""
    B = _bmo64(C, b, P)[:P]
    d = torch.stack([B[p, p] for p in range(P)])
    Cp = C[:, :P]
    return (d @ d.T).contiguous(), B.square().sum(2).contiguous(), (Cp * (H @ Cp)).sum(0).contiguous()


def _lag64(C, H, b, n, cj, ck, P, nd):
    B = _bmo64(C, b, P)
    d = torch.stack([B[p, p] for p in range(P)])
    Hmat = C.T @ H @ C[:, :P]
    w = cj @ d + n[:, None] * d  # closed shell: every orbital is doubly occupied or correlating
    elag = torch.zeros_like(C)
    exch = B.reshape(C.shape[0], -1) @ (ck[:, :, None] * B[:P]).reshape(P, -1).T
    elag[:, :P] = n * Hmat + torch.einsum("abk,bk->ab", B, w) - exch
    return elag, Hmat


def _expm64(y, nbf, P):
    i, j = torch.triu_indices(nbf, nbf, 1)
    keep = i < P
    Y = torch.zeros((nbf, nbf), dtype=F64)
    Y[i[keep], j[keep]] = y.cpu()
    return torch.linalg.matrix_exp(Y - Y.T)


def exact(case, seed):
    kind, s = case["kind"], _parts(case, seed)
    if kind == "occ":
        return None  # the result of an iteration
    if kind == "batch":
        JK = [_jk64(C, b, P) for C, b, P in s["mols"]]
        return {"J": [j for j, _ in JK], "K": [k for _, k in JK]}
    P, nd, C, H = case["nbf5"], _half(case["nbf5"]), s["C"], s["H"]
    if kind in ("jk", "dropin"):
        J, K = _jk64(C, s["b"], P)
        return {"J": J.cpu().numpy(), "K": K.cpu().numpy()} if kind == "dropin" else {"J": J, "K": K}
    if kind == "mo":
        return dict(zip(("J", "K", "Hc"), _mo64(C, H, s["b"], P)))
    if kind == "lag":
        return dict(zip(("elag", "Hmat"), _lag64(C, H, s["b"], s["n"], s["cj"], s["ck"], P, nd)))
    if kind == "step":
        C = C @ _expm64(s["y"], case["nbf"], P).to(DEV)
        J, K, Hc = _mo64(C, H, s["b"], P)
        elag, Hmat = _lag64(C, H, s["b"], s["n"], s["cj"], s["ck"], P, nd)
        return {"C": C, "J": J, "K": K, "Hc": Hc, "elag": elag, "Hmat": Hmat}
    N, I, n = case["nbf"], s["I"], s["n"]
    D = torch.einsum("si,li->isl", C[:, :P], C[:, :P]).reshape(P, N * N)
    J = (D @ I.view(N * N, N * N).T).view(P, N, N)
    K = (D @ I.permute(1, 3, 0, 2).reshape(N * N, N * N)).view(P, N, N)
    F = torch.einsum("ij,jmn->imn", s["cj"], J) - torch.einsum("ij,jmn->imn", s["ck"], K)
    F += n[:, None, None] * (H + J)  # closed shell
    G = torch.einsum("imn,ni->mi", F, C[:, :P])
    elag = torch.zeros_like(C)
    elag[:, :P] = C.T @ G
    E = elag.diagonal()[:P].sum() + (n * (C[:, :P] * (H @ C[:, :P])).sum(0)).sum()
    return {"J": J, "K": K, "F": F, "elag": elag, "E": E}
