"""Timed cases of the (T) library: what its users have it do, through its public entry points.

A case is one of these calls on device-resident FP64 inputs in the reference's layouts:

  kernel  ``pyscfad_b200.cc.ccsd_t.kernel`` and its autograd backward (the drop-in of the reference's entry point)
  energy  ``triples.energy``: E(T) alone
  vjp     ``triples.energy_vjp``: E(T) and the gradients of all seven inputs, whole or a slice of virtual blocks
  lno     ``triples.lno_energy_vjp``: the LNO fragment energy and its gradients
  df      ``triples.energy_vjp_df``: ovvv given as its density-fitting factors
  batch   ``BatchedTriples.run``: many uneven problems replayed as one CUDA graph

Inputs follow the distributions of the benchmark workloads (orbital energies with a gap, small random amplitudes,
integrals contracted from random Cholesky-like factors).
"""
import types

import torch

from pyscfad_b200 import triples
from pyscfad_b200.batched import BatchedTriples
from pyscfad_b200.cc import ccsd_t

KEYS = ("mo_energy", "t1", "t2", "ovoo", "ovov", "ovvv", "fvo")
DF_KEYS = ("mo_energy", "t1", "t2", "ovoo", "ovov", "Lov", "Lvv", "fvo")
LEAVES = ("fock", "mo_energy", "ovoo", "ovov", "ovvv", "t1", "t2")
BLOCK = 16   # virtual block of the library's chunk decomposition, in which chunk_range counts


def _case(name, form, nocc, nvir, naux, precision="mixed", packed=True, fvo=False, **more):
    return dict(name=name, form=form, nocc=nocc, nvir=nvir, naux=naux, precision=precision, packed=packed, fvo=fvo,
                **more)


def listed():
    return [
        # one small molecule (water, cc-pVDZ) through the drop-in kernel and its backward, in its default
        # precision: launches, host work and latency
        _case("kernel_fp64_o5v19", "kernel", 5, 19, 80, "fp64"),
        # the same molecule in the mode the benchmark runs
        _case("vjp_mixed_o5v19", "vjp", 5, 19, 80),
        # a single-point energy of a small molecule, no gradients
        _case("energy_mixed_o10v60", "energy", 10, 60, 280),
        # ragged sizes, four-index integrals that are not packed, non-canonical orbitals, the bf16 mode
        _case("vjp_bf16_o13v83", "vjp", 13, 83, 384, "mixed_bf16", packed=False, fvo=True),
        # energy and gradients at full precision, a mid-sized molecule
        _case("vjp_fp64_o12v100", "vjp", 12, 100, 448, "fp64"),
        # the same size with density-fitted integrals handed over as factors
        _case("df_mixed_o12v100", "df", 12, 100, 448),
        # an LNO fragment: projector of half of the occupied orbitals
        _case("lno_mixed_o14v96", "lno", 14, 96, 400),
        # a small fragment at full precision, odd sizes
        _case("lno_fp64_o9v45", "lno", 9, 45, 200, "fp64", fvo=True),
        # the benchmark's batched workload: uneven small problems as one graph
        _case("batch_mixed_48", "batch", 12, 80, 0, count=48, mix=1),
        # many correlated electrons in a small basis
        _case("vjp_mixed_o40v72", "vjp", 40, 72, 400, fvo=True),
        # the benchmark's medium workload, whole
        _case("vjp_mixed_o20v180", "vjp", 20, 180, 600),
        # one slice of the headline workload, as one of the jobs that it is split into
        _case("slice_mixed_o40v360", "vjp", 40, 360, 1200, a0=6, a1=7),
    ]


def draw(rng):
    """A call of the ranges above: work (nocc^3 nvir^4) and nocc spread over their logarithms."""
    def log_uniform(lo, hi):
        return lo * (hi / lo) ** rng.random()

    def sizes(o_hi, w_lo, w_hi, v_hi=192):
        w = log_uniform(w_lo, w_hi)
        # nvir between 1.5 nocc and v_hi
        o = int(round(log_uniform(max(3.0, (w / v_hi ** 4) ** (1 / 3)), min(o_hi, max(3.5, (w / 5) ** (1 / 7))))))
        return o, int((w / o ** 3) ** 0.25)

    form = rng.choice(["kernel", "energy", "vjp", "vjp", "vjp", "vjp", "lno", "df", "batch", "slice"])
    if form == "batch":
        return _pure("batch", rng.randint(7, 12), rng.randint(40, 80), 0, count=rng.randint(6, 48),
                     mix=rng.randint(2, 1 << 20))
    if form == "slice":
        o, v = rng.randint(16, 40), rng.randint(192, 330)
        a0 = rng.randint(0, 5)
        return _pure("vjp", o, v, 3 * (o + v), a0=a0, a1=a0 + 1)
    precision = {"kernel": "fp64", "lno": rng.choice(["mixed", "fp64"]), "df": rng.choice(["mixed", "fp64"]),
                 "energy": rng.choice(["mixed", "fp64"]),
                 "vjp": rng.choice(["mixed", "mixed", "mixed_bf16", "fp64"])}[form]
    if form == "lno":
        o, v = sizes(20, 1e6, 2e11)
    elif precision == "fp64":
        o, v = sizes(24, 1e6, 3e11)
    else:
        o, v = sizes(40, 1e6, 4e12)
    return _pure(form, o, v, 4 * (o + v), precision, packed=form in ("df", "batch") or rng.random() < 0.7,
                 fvo=rng.random() < 0.5)


def _pure(*a, **k):
    return {key: val for key, val in _case("", *a, **k).items() if key != "name"}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _tril(v, dev):
    return torch.tril_indices(v, v, device=dev)


def _inputs(case, seed):
    """The benchmark's distributions, FP64, from the seed alone; "Lov" and "Lvv" beside the seven inputs."""
    dev, o, v = _device(), case["nocc"], case["nvir"]
    naux = case["naux"] or 4 * (o + v)
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 1000003 + 17)
    kw = dict(dtype=torch.float64, device=dev)
    eo = torch.sort(torch.empty(o, **kw).uniform_(-1.5, -0.3, generator=g))[0]
    ev = torch.sort(torch.empty(v, **kw).uniform_(0.2, 3.0, generator=g))[0]
    t1 = torch.empty(o, v, **kw).normal_(0.0, 1e-2, generator=g)
    x = torch.empty(o, o, v, v, **kw).normal_(0.0, 2e-2, generator=g)
    t2 = (0.5 * (x + x.permute(1, 0, 3, 2))).contiguous()
    del x
    il, jl = _tril(v, dev)
    # factors of symmetric matrices: off-diagonal entries are means of two draws
    Lov = torch.empty(naux, o * v, **kw).normal_(0.0, 0.1 * 0.5 ** 0.5, generator=g)
    y = torch.empty(naux, o, o, **kw).normal_(0.0, 0.1, generator=g)
    Loo = (0.5 * (y + y.transpose(1, 2))).reshape(naux, o * o)
    sd = torch.where(il == jl, 0.1, 0.1 * 0.5 ** 0.5).to(torch.float64)
    Lvv = torch.empty(naux, il.numel(), **kw).normal_(0.0, 1.0, generator=g) * sd
    inp = dict(mo_energy=torch.cat([eo, ev]), t1=t1, t2=t2,
               ovoo=(Lov.T @ Loo).reshape(o, v, o, o), ovov=(Lov.T @ Lov).reshape(o, v, o, v),
               fvo=torch.zeros(v, o, **kw))
    if case["fvo"]:
        inp["fvo"].normal_(0.0, 1e-3, generator=g)
    if case["form"] == "df":
        inp.update(Lov=Lov, Lvv=Lvv)
    else:
        ovvv = (Lov.T @ Lvv).reshape(o, v, il.numel())
        inp["ovvv"] = ovvv if case["packed"] else _unpack(ovvv)
    if case["form"] == "lno":
        z = torch.empty(o, o, **kw).normal_(0.0, 1.0, generator=g)
        ulo = torch.linalg.qr(z)[0][: max(1, o // 2)]
        inp["mat"] = (ulo.T @ ulo).contiguous()
    return inp


def _unpack(ovvv):
    o, v = ovvv.shape[0], ovvv.shape[1]
    il, jl = _tril(v, ovvv.device)
    full = torch.empty(o, v, v, v, dtype=ovvv.dtype, device=ovvv.device)
    full[:, :, il, jl] = ovvv
    full[:, :, jl, il] = ovvv
    return full


def _members(case):
    """The problems of a batch: nocc from 4, nvir from 20 up to the case's, drawn from its "mix" alone."""
    g = torch.Generator()
    g.manual_seed(case["mix"])
    o = torch.randint(4, case["nocc"] + 1, (case["count"],), generator=g).tolist()
    v = torch.randint(20, case["nvir"] + 1, (case["count"],), generator=g).tolist()
    return [dict(_pure("vjp", a, b, 0), member=n) for n, (a, b) in enumerate(zip(o, v))]


def _member_inputs(case, seed):
    return [_inputs(m, int(seed) * 1009 + m["member"]) for m in _members(case)]


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["form"] == "batch":
        bt = BatchedTriples(_member_inputs(case, seed), precision=case["precision"], tune=False)
        bt.capture()
        return {"case": case, "batch": bt}
    inp = _inputs(case, seed)
    if case["form"] != "kernel":
        return {"case": case, "inp": inp}
    o, v = case["nocc"], case["nvir"]
    fock = torch.diag(inp["mo_energy"])
    fock[o:, :o] = inp["fvo"]
    fock[:o, o:] = inp["fvo"].T
    leaf = {k: x.requires_grad_() for k, x in dict(inp, fock=fock).items() if k in LEAVES}
    eris = types.SimpleNamespace(**{k: leaf[k] for k in ("fock", "mo_energy", "ovoo", "ovov", "ovvv")})
    return {"case": case, "leaf": leaf, "eris": eris, "cc": types.SimpleNamespace(t1=leaf["t1"], t2=leaf["t2"])}


def run(state):
    case = state["case"]
    form, precision = case["form"], case["precision"]
    if form == "batch":
        bt = state["batch"]
        bt.run()
        out = {k: torch.cat([p.grads[k].reshape(-1) for p in bt.problems]) for k in KEYS}
        out["e"] = torch.stack([p.energy for p in bt.problems])
        return out
    if form == "kernel":
        e = ccsd_t.kernel(state["cc"], state["eris"])
        grads = torch.autograd.grad(e, [state["leaf"][k] for k in LEAVES])
        return dict(zip(LEAVES, grads), e=e.detach())
    inp = state["inp"]
    if form == "energy":
        return {"e": triples.energy(*(inp[k] for k in KEYS), precision=precision)}
    if form == "lno":
        e, g = triples.lno_energy_vjp(inp["mat"], *(inp[k] for k in KEYS), precision=precision)
    elif form == "df":
        e, g = triples.energy_vjp_df(*(inp[k] for k in DF_KEYS), precision=precision)
    else:
        chunks = (case["a0"], case["a1"]) if "a1" in case else None
        e, g = triples.energy_vjp(*(inp[k] for k in KEYS), precision=precision, chunk_range=chunks)
    return dict(g, e=e)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _fraction(case):
    """Share of the raw amplitudes in the blocks [a0, a1) of a slice."""
    if "a1" not in case:
        return 1.0
    v = case["nvir"]
    hi, lo = min(v, BLOCK * case["a1"]), min(v, BLOCK * case["a0"])
    return (hi ** 3 - lo ** 3) / v ** 3


def work(case):
    if case["form"] == "batch":
        parts = [work(m) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    o, v = case["nocc"], case["nvir"]
    pairs = v * (v + 1) // 2
    naux = case["naux"] or 4 * (o + v)
    words = (o + v) + 2 * o * v + o * o * v * v * 2 + o ** 3 * v
    words += naux * (o * v + pairs) if case["form"] == "df" else o * v * (pairs if case["packed"] else v * v)
    grad = case["form"] != "energy"
    flops = (6 if grad else 2) * o ** 3 * v ** 3 * (v + o) * _fraction(case)
    if case["form"] == "df":
        flops += 6 * o * v * pairs * naux
    if case["form"] == "lno":
        flops += 6 * o ** 4 * v ** 3
    return {"bytes": 8 * words * (2 if grad else 1), "flops": flops}


# ---------------------------------------------------------------------------
# the same quantities in plain torch, 64 bits
# ---------------------------------------------------------------------------
PERMS = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))


def _r3(x):
    """The spin adaptation on the virtual indices of a quantity that is symmetric under simultaneous permutations:
    the same permutations of the occupied indices.  Its own transpose."""
    p = lambda *d: x.permute(*d, 3, 4, 5)  # noqa: E731
    return 4.0 * x + p(1, 2, 0) + p(2, 0, 1) - 2.0 * (p(2, 1, 0) + p(0, 2, 1) + p(1, 0, 2))


def _triples(inp, packed, a0, a1, want_grad):
    """E(T) (with "mat": the LNO energy) and its gradients over the virtual blocks [a0, a1), tile by tile:
    w[ijk,abc] = sum_f ovvv[i,a,f,b] t2[k,j,c,f] - sum_m ovoo[i,a,m,j] t2[k,m,c,b],
    v[ijk,abc] = ovov[i,a,j,b] t1[k,c] + t2[j,i,b,a] fvo[c,k],  WW, VV: their sums over simultaneous permutations,
    E = 1/3 sum WW r3(WW + VV/2) / D over all indices (the first occupied index of the first factor projected)."""
    e, t1, t2, ovoo, ovov, fvo = (inp[k] for k in ("mo_energy", "t1", "t2", "ovoo", "ovov", "fvo"))
    mat = inp.get("mat")
    ovvv = _unpack(inp["ovvv"]) if packed else inp["ovvv"]
    o, v = t1.shape
    eo, ev = e[:o], e[o:]
    step = BLOCK
    if a0 is None:
        while step < v and o ** 3 * (2 * step) ** 3 <= 1 << 26:
            step *= 2
        a0, a1 = 0, -(-v // step)
    tiles = [slice(s, min(v, s + step)) for s in range(0, v, step)]
    val = dict(ovvv=ovvv, t2=t2, ovoo=ovoo, ovov=ovov, t1=t1, fvo=fvo)
    bar = {k: torch.zeros_like(x) for k, x in val.items()}
    bar["mo_energy"] = torch.zeros_like(e)
    if mat is not None:
        bar["mat"] = torch.zeros_like(mat)
    energy = torch.zeros((), dtype=torch.float64, device=e.device)
    for A in range(a0, min(a1, len(tiles))):
        for B in range(A + 1):
            for C in range(B + 1):
                blk = (tiles[A], tiles[B], tiles[C])
                orderings = len({(A, B, C)[s] * 10 ** 6 + (A, B, C)[t] * 10 ** 3 + (A, B, C)[u] for s, t, u in PERMS})
                terms = []   # (left term, right factor, their letters, blocks): signed products of each permutation
                for s in PERMS:
                    p, q, r = ("ijk"[n] for n in s)
                    x, y, z = ("abc"[n] for n in s)
                    X, Y, Z = (blk[n] for n in s)
                    al = slice(None)
                    terms += [(1.0, "W", "ovvv", (al, X, al, Y), p + x + "f" + y, "t2", (al, al, Z, al), r + q + z + "f"),
                              (-1.0, "W", "ovoo", (al, X, al, al), p + x + "m" + q, "t2", (al, al, Z, Y), r + "m" + z + y),
                              (1.0, "V", "ovov", (al, X, al, Y), p + x + q + y, "t1", (al, Z), r + z),
                              (1.0, "V", "t2", (al, al, Y, X), q + p + y + x, "fvo", (Z, al), z + r)]
                shape = (o, o, o) + tuple(t.stop - t.start for t in blk)
                sums = {k: torch.zeros(shape, dtype=torch.float64, device=e.device) for k in "WV"}
                for sign, to, ka, ia, la, kb, ib, lb in terms:
                    sums[to].add_(torch.einsum(la + "," + lb + "->ijkabc", val[ka][ia], val[kb][ib]), alpha=sign)
                WW = sums["W"]
                occ = eo[:, None, None] + eo[None, :, None] + eo[None, None, :]
                vir = ev[blk[0]][:, None, None] + ev[blk[1]][None, :, None] + ev[blk[2]][None, None, :]
                D = occ[:, :, :, None, None, None] - vir
                Q = _r3(WW + 0.5 * sums["V"]) / D
                if mat is None:
                    c, PW, PQ = orderings / 3.0, WW, Q
                else:
                    # sum over the orderings of (A, B, C): the projector on each of the three occupied slots
                    c = orderings / 9.0
                    spec = ("ljkabc,li->ijkabc", "ilkabc,lj->ijkabc", "ijlabc,lk->ijkabc")
                    PW = sum(torch.einsum(t, WW, mat) for t in spec)
                    PQ = sum(torch.einsum(t, Q, mat.T) for t in spec)
                energy += c * torch.sum(PW * Q)
                if not want_grad:
                    continue
                if mat is not None:
                    bar["mat"] += c * (torch.einsum("ljkabc,ijkabc->li", WW, Q) + torch.einsum("jlkabc,jikabc->li", WW, Q)
                                       + torch.einsum("jklabc,jkiabc->li", WW, Q))
                Qb = c * PW
                Db = -Qb * Q / D
                for n in range(3):
                    bar["mo_energy"][:o] += Db.sum(dim=[d for d in range(6) if d != n])
                    bar["mo_energy"][o:][blk[n]] -= Db.sum(dim=[d for d in range(6) if d != 3 + n])
                Xb = _r3(Qb / D)
                del Db, Qb, D, PW
                grad = {"W": c * PQ + Xb, "V": 0.5 * Xb}
                for sign, to, ka, ia, la, kb, ib, lb in terms:
                    G = grad[to]
                    bar[ka][ia] += sign * torch.einsum("ijkabc," + lb + "->" + la, G, val[kb][ib])
                    bar[kb][ib] += sign * torch.einsum("ijkabc," + la + "->" + lb, G, val[ka][ia])
    if packed:
        il, jl = _tril(v, e.device)
        low = bar["ovvv"][:, :, il, jl]
        bar["ovvv"] = low + torch.where(il == jl, 0.0, 1.0) * bar["ovvv"][:, :, jl, il]
    return energy, bar


def exact(case, seed):
    form = case["form"]
    if form == "batch":
        got = [_triples(x, True, None, None, True) for x in _member_inputs(case, seed)]
        out = {k: torch.cat([b[k].reshape(-1) for _, b in got]) for k in KEYS}
        out["e"] = torch.stack([e for e, _ in got])
        return out
    inp = _inputs(case, seed)
    if form == "df":
        o, v = inp["t1"].shape
        inp["ovvv"] = (inp["Lov"].T @ inp["Lvv"]).reshape(o, v, -1)
    e, bar = _triples(inp, case["packed"], case.get("a0"), case.get("a1"), form != "energy")
    if form == "energy":
        return {"e": e}
    if form == "df":
        g = bar.pop("ovvv").reshape(inp["Lov"].shape[1], -1)
        bar.update(Lov=inp["Lvv"] @ g.T, Lvv=inp["Lov"] @ g)
    if form == "kernel":
        o, v = inp["t1"].shape
        fock = torch.zeros(o + v, o + v, dtype=torch.float64, device=e.device)
        fock[o:, :o] = bar.pop("fvo")
        bar["fock"] = fock
    return dict(bar, e=e)
