"""Performance cases of the engine: the calls a CIPSI user's program makes.

Every case goes through the public entry points -- `engine.Context.run`,
`run_stream`, `adjoint`, `adjoint_1e`, `selection_raw`, `engine.Batch`, and the
C entries `cipsi_hamiltonian_build` / `_get` and `cipsi_davidson` -- on seeded
inputs in the reference's file formats (cipsi_gb300/synth.py).  The systems are
well conditioned, as converged CIPSI inputs are: the perturbers lie above every
root energy (a gap between occupied and virtual orbitals, one reference-
dominated root, or a complete active space for several roots).

Results are returned whole, without the engine's own work counters (compares,
pairs, bytes, times, launches), which describe how it computes and not what.
"""
from __future__ import annotations

import ctypes
import itertools
import math
import os
import tempfile

import numpy as np

from cipsi_gb300 import engine, shard, synth

# fields of Context.run's result that are answers (the others are counters of work done and times)
ANSWER = ("e2mp", "e2vp", "e2b", "psimp", "psivp", "dpivot", "ietat", "n_processed", "n_selected", "n_candidates",
          "nom", "nam", "tabmp", "tabvp")


def _case(name, kind, norb, nocc, metat=1, tau=0.01, **kw):
    """One case.  S: `ncf` determinants of the excitation ranks in `ranks`, or
    the complete active space (cas_occ, cas_virt) when cas_occ > 0."""
    c = {"name": name, "kind": kind, "norb": norb, "nocc": nocc, "metat": metat, "tau": tau, "ncf": 0, "ranks": "2",
         "cas_occ": 0, "cas_virt": 0, "nsym": 1, "ityper": 2, "iselec": 1, "world": 1, "geometries": 1}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: the 20-orbital test system, records read back (latency and launches)
        _case("run_20orb", "run", 20, 5, ncf=50, tau=0.02),
        # odd sizes, four irreps, singles to triples, as an ordinary molecule's symmetry gives
        _case("run_37orb_sym4", "run", 37, 7, ncf=333, ranks="1,2,3", nsym=4, tau=0.01),
        # Moller-Plesset partition alone (ityper = 1), energy-based listing
        _case("run_45orb_mp", "run", 45, 9, ncf=450, ranks="1,2", ityper=1, tau=0.01),
        # the 60-orbital benchmark size, S of singles to triples, all generators
        _case("run_60orb", "run", 60, 10, ncf=2000, ranks="1,2,3", tau=0.01),
        # several roots over a complete active space (the strict parity test's space)
        _case("run_60orb_cas_3roots", "run", 60, 10, metat=3, cas_occ=2, cas_virt=8, tau=0.01),
        # one rank's shard of the 120-orbital, S = 20,000 benchmark, streamed in chunks
        _case("stream_120orb_shard", "stream", 120, 15, ncf=20000, world=160, tau=0.005),
        # two roots, two-word strings, active space, one rank's shard
        _case("stream_120orb_cas_2roots", "stream", 120, 15, metat=2, cas_occ=2, cas_virt=8, world=16, tau=0.005),
        # points of a potential curve in one batched launch (norb 40-100, |S| 500-5000)
        _case("batch_6_geometries", "batch", 40, 10, ncf=500, ranks="1,2,3", geometries=6),
        # gradients: the full adjoint, and the one-electron one of the finite-field runs
        _case("adjoint_30orb", "adjoint", 30, 6, ncf=300, ranks="1,2,3"),
        _case("adjoint_1e_50orb_cas_2roots", "adjoint_1e", 50, 10, metat=2, cas_occ=2, cas_virt=5, nsym=2),
        # the CI matrix over a list of determinants (moy) and its lowest roots (bd)
        _case("hamiltonian_16k", "hamiltonian", 60, 10, ncf=16001, ranks="1,2,3"),
        _case("davidson_6k", "davidson", 6001, 40, metat=2),
    ]


def draw(rng):
    """Another case of the same kinds, sizes spread over their ranges."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "stream", "batch", "adjoint", "adjoint_1e", "hamiltonian", "davidson"])
    if kind == "davidson":
        return _plain(_case("", kind, log_int(200, 8000), log_int(10, 60), metat=rng.randint(1, 4)))
    if kind == "hamiltonian":
        return _plain(_case("", kind, rng.randint(24, 100), rng.randint(6, 12), ncf=log_int(500, 16000),
                            ranks=rng.choice(["1,2,3", "1,2", "2,3"]), nsym=rng.choice([1, 1, 2])))
    if kind == "batch":
        return _plain(_case("", kind, rng.randint(20, 48), rng.randint(5, 9), ncf=log_int(60, 500), ranks="1,2,3",
                            geometries=rng.randint(2, 8)))
    while True:
        nocc = rng.randint(3, 12)
        norb = nocc + log_int(9, 90 if kind == "stream" else 55)
        c = _case("", kind, norb, nocc, tau=rng.choice([0.005, 0.01, 0.02]), nsym=rng.choice([1, 1, 2, 4]))
        if rng.random() < 0.4 and nocc >= 3:
            c.update(metat=rng.randint(1, 4), cas_occ=2, cas_virt=rng.randint(2, min(8, norb - nocc - 2)))
            nc = math.comb(c["cas_occ"] + c["cas_virt"], 2) ** 2
        else:
            nc = log_int(40, 3000)
            c.update(ncf=nc, ranks=rng.choice(["2", "1,2", "1,2,3", "1,2,3,4"]))
        if kind in ("run", "stream"):
            c["ityper"] = rng.choice([2, 2, 2, 1])
            c["iselec"] = rng.choice([1, 1, 3])
        if kind == "stream":
            c["world"] = rng.choice([2, 4, 8])
        # candidates of all generators, against those of the 60-orbital listed case
        cand = _candidates(c, nc) / c["world"]
        room = 0.9 * (norb - nocc - (c["cas_virt"] if c["cas_occ"] else 0)) >= 4
        if cand < (1.5e8 if kind.startswith("adjoint") else 3.2e8) and room and nc < 0.2 * _space(norb, nocc, c):
            return _plain(c)


def _plain(c):
    del c["name"]
    return c


def _space(norb, nocc, c):
    """About how many determinants of the case's ranks there are to draw S from."""
    if c["cas_occ"]:
        return math.inf
    nv = norb - nocc
    return sum(math.comb(2 * nocc, r) * math.comb(2 * nv, r) / 2.5 for r in map(int, c["ranks"].split(","))) / c["nsym"]


def _dets(c):
    return math.comb(c["cas_occ"] + c["cas_virt"], c["cas_occ"]) ** 2 if c["cas_occ"] else c["ncf"]


def _candidates(c, ncf):
    """Single and double excitations of the generators (half of S: one per spin-flip pair)."""
    no, nv = c["nocc"], c["norb"] - c["nocc"]
    per = 2 * no * nv + 2 * math.comb(no, 2) * math.comb(nv, 2) + (no * nv) ** 2
    return ncf / 2 * per / c["nsym"]


def _capacity(case):
    """Records a case's own arrays hold (more than its runs select; the rest stays zero), or matrix
    elements of the hamiltonian case."""
    if case["kind"] == "hamiltonian":
        return case["ncf"] * min(case["ncf"], 1500) + 64
    share = 0.2 if case["cas_occ"] else 0.02
    return min(16 << 20, int(share * _candidates(case, _dets(case))) + 4096)


def work(case):
    """Floating-point operations: per candidate one two-electron element with every root (4 + 2 per root) and
    three denominators, quotients and sums per root (20).  Bytes: integrals, S and coefficients read, results
    and matrix elements written."""
    n, m = case["norb"], case["metat"]
    if case["kind"] == "davidson":
        nnz = n * case["nocc"]  # one product per root and iteration, about 12 iterations
        return {"bytes": 12.0 * nnz + 8.0 * n * m, "flops": 12.0 * 2 * nnz * (m + 2)}
    nc, words = _dets(case), 2 * (1 if n <= 64 else 2)
    ints = (n * (n + 1) // 2) ** 2 / 2 / case["nsym"] * 4.0
    if case["kind"] == "hamiltonian":
        return {"bytes": ints + 8.0 * words * nc, "flops": 2.0 * words * nc * nc / 2}
    cand = case["geometries"] * _candidates(case, nc) / case["world"]
    scale = 2.0 if case["kind"] == "adjoint" else 1.0
    return {"bytes": case["geometries"] * (ints + 8.0 * (words + m) * nc), "flops": scale * cand * (4 + 22.0 * m)}


# ------------------------------------------------------------------ inputs
def _config(case, seed, index=0):
    """The synthetic system of a case: reference-dominated single-root spaces
    (sum of the other squared coefficients about 0.1) with a gap of 3 Eh, or
    active spaces 6 Eh apart from the other orbitals."""
    n, nocc, ncf = case["norb"], case["nocc"], case["ncf"]
    if case["kind"] == "batch":  # a curve's points differ in basis and space size
        n, ncf = n + (7 * index) % 61, ncf + (233 * index) % (2 * ncf)
    kw = dict(norb=n, nocc=nocc, ncholesky=2 * n, metat=case["metat"], tau=case["tau"], ityper=case["ityper"],
              iselec=case["iselec"], nsym=case["nsym"], seed=1000 * seed + index, coef_mode="gauss005",
              energy="diagonal")
    if case["cas_occ"]:
        return synth.SynthConfig("case", ncf=0, space="cas", cas_occ=case["cas_occ"], cas_virt=case["cas_virt"],
                                 core_shift=6.0, virt_shift=6.0, **kw)
    return synth.SynthConfig("case", ncf=ncf, ranks=tuple(map(int, case["ranks"].split(","))), virt_shift=3.0,
                             coef_sigma=0.3 / math.sqrt(ncf),
                             curve_R=2.0 + 1.5 * index if case["kind"] == "batch" else None, **kw)


def _load(cfg):
    """An uploaded context and its options, from the files of one calculation directory."""
    with tempfile.TemporaryDirectory() as wd:
        synth.generate(cfg, wd)
        inp = engine.Inputs(wd)
    ctx = engine.Context(inp.dims)
    ctx.upload(inp)
    opts = engine.Opts.from_buffer_copy(inp.opts)
    inp.close()
    return ctx, opts


def prepare(case, seed):
    kind = case["kind"]
    if kind == "davidson":
        return _sparse(case, seed)
    if kind == "batch":
        pairs = [_load(_config(case, seed, i)) for i in range(case["geometries"])]
        ctxs, opts = [p[0] for p in pairs], [p[1] for p in pairs]
        return {"kind": kind, "batch": engine.Batch(ctxs, opts), "ctxs": ctxs}
    ctx, opts = _load(_config(case, seed))
    st = {"kind": kind, "ctx": ctx, "opts": opts, "mask": None}
    if kind == "stream":
        st["mask"] = np.ascontiguousarray(shard.generator_mask(ctx.dims.ncf, 1, case["world"]), np.uint8)
    if kind.startswith("adjoint"):
        st["seed"] = np.random.default_rng(seed).normal(size=(3, ctx.dims.metat))
    if kind == "run":
        cap, words = _capacity(case), 2 * (1 if case["norb"] <= 64 else 2)
        st["records"] = {"bits": np.zeros((cap, words), np.uint64), "owner": np.zeros(cap, np.int32),
                         "xam": np.zeros(cap), "evp": np.zeros((cap, case["metat"]))}
    if kind == "hamiltonian":
        st["lib"] = _hamiltonian_entries()
        st["col"], st["val"] = np.zeros(_capacity(case), np.int32), np.zeros(_capacity(case))
        st["rowptr"] = np.zeros(case["ncf"] + 2, np.int64)  # the closure of S may add one determinant
    return st


def _hamiltonian_entries():
    lib = engine._lib()
    P, I64 = ctypes.c_void_p, ctypes.c_int64
    lib.cipsi_hamiltonian_build.argtypes = [P, P, ctypes.c_int32, ctypes.POINTER(I64)]
    lib.cipsi_hamiltonian_get.argtypes = [P, ctypes.c_int32, ctypes.c_int32, P, P, P]
    return lib


def _sparse(case, seed):
    """A CI-like matrix as moy stores it: a rising diagonal (halved), about
    `nocc` off-diagonal elements per row that fall off in size, rows in order."""
    n, per = case["norb"], case["nocc"]
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(1, n), np.minimum(np.arange(1, n), max(1, per // 2)))
    cols = (rng.random(len(rows)) * rows).astype(np.int64)
    key = np.unique(rows * n + cols)
    rows, cols = key // n, key % n
    vals = rng.normal(0.0, 0.03, len(key))
    diag = np.sort(rng.uniform(0.0, 6.0, n))
    diag[: case["metat"]] -= 2.0 - 0.2 * np.arange(case["metat"])
    i = np.concatenate([rows, np.arange(n)])
    j = np.concatenate([cols, np.arange(n)])
    v = np.concatenate([vals, 0.5 * diag])
    order = np.lexsort((j, i))
    return {"kind": "davidson", "n": n, "roots": case["metat"], "i": (i[order] + 1).astype(np.int32),
            "j": (j[order] + 1).astype(np.int32), "v": np.ascontiguousarray(v[order]), "lib": engine._lib()}


# -------------------------------------------------------------------- runs
def _answer(res):
    return {k: np.asarray(res[k]) for k in ANSWER}


def run(state):
    kind = state["kind"]
    if kind == "run":
        res = state["ctx"].run(state["opts"])
        records = state["records"]
        if res["n_selected"] > len(records["owner"]):
            raise RuntimeError("more records than the program's arrays hold")
        state["ctx"].selection_raw(res["n_selected"], out=records)
        return {"result": _answer(res), "records": dict(records, bits=records["bits"].view(np.int64))}
    if kind == "stream":
        return {"result": _answer(state["ctx"].run_stream(state["opts"], gen_mask=state["mask"]))}
    if kind == "batch":
        state["batch"].run()
        state["batch"].wait()
        results = [_answer(r) for r in state["batch"].fetch_all()]
        return {"result": {k: np.stack([r[k] for r in results]) for k in ANSWER}}
    if kind == "adjoint":
        return {"gradients": state["ctx"].adjoint(state["opts"], state["seed"])}
    if kind == "adjoint_1e":
        e2, grad = state["ctx"].adjoint_1e(state["opts"], state["seed"])
        return {"e2": e2, "gradients": grad}
    if kind == "hamiltonian":
        ctx, lib, npairs = state["ctx"], state["lib"], ctypes.c_int64()
        ctx._check(lib.cipsi_hamiltonian_build(ctx._c, None, -1, ctypes.byref(npairs)), "hamiltonian_build")
        rowptr, col, val = state["rowptr"], state["col"], state["val"]
        if npairs.value > len(col):
            raise RuntimeError("more matrix elements than the program's arrays hold")
        ctx._check(lib.cipsi_hamiltonian_get(ctx._c, 0, ctx.dims.ncf, rowptr.ctypes.data, col.ctypes.data,
                                             val.ctypes.data), "hamiltonian_get")
        return {"rowptr": rowptr, "col": col, "val": val}
    n, roots = state["n"], state["roots"]
    evals, evecs = np.empty(roots), np.empty((roots, n))
    err, iters = ctypes.create_string_buffer(512), ctypes.c_int32()
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (state["i"], state["j"], state["v"])]
    rc = state["lib"].cipsi_davidson(
        ctypes.c_int32(n), ctypes.c_int64(len(state["v"])), *p, ctypes.c_int32(roots), ctypes.c_double(1e-11),
        ctypes.c_int32(200), ctypes.c_int32(0), evals.ctypes.data_as(ctypes.c_void_p),
        evecs.ctypes.data_as(ctypes.c_void_p), ctypes.byref(iters), None, err, ctypes.c_int32(len(err)))
    if rc != 0:
        raise RuntimeError(err.value.decode())
    return {"evals": evals, "evecs": evecs}


# ------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """Plain numpy in 64 bits: the eigenpairs of a small matrix; the E2 sums of
    a small run, by the perturbation step's rules on sets of occupied spin orbitals."""
    if case["kind"] == "davidson" and case["norb"] <= 3000:
        s = _sparse(case, seed)
        H = np.zeros((s["n"], s["n"]))
        H[s["i"] - 1, s["j"] - 1] = s["v"]
        w, U = np.linalg.eigh(H + H.T)
        U = U[:, : s["roots"]].T
        big = U[np.arange(s["roots"]), np.abs(U).argmax(axis=1)]
        return {"evals": w[: s["roots"]], "evecs": U * np.sign(big)[:, None]}
    if case["kind"] == "run" and not case["cas_occ"] and case["ranks"] == "2" and case["nsym"] == 1 and \
            case["ityper"] == 2 and _candidates(case, case["ncf"]) < 4e5:
        sums = _e2_doubles(_config(case, seed))
        return {"result": {k: sums.get(k) for k in ANSWER}, "records": None}
    return None


def _e2_doubles(cfg):
    """E2 sums over the perturbers of S = reference + doubles (closed under
    spin flip, partners adjacent, one root), from the Cholesky factors."""
    rng = np.random.default_rng(cfg.seed)
    h, L, irrep = synth.make_integrals(cfg, rng)
    dets, rep = synth.build_space(cfg, rng, irrep)  # the inputs' own draws, in their order
    n, no = cfg.norb, cfg.nocc
    c = rng.normal(0.0, cfg.coef_sigma, size=max(rep) + 1)
    c[0] = 1.0
    c = c[np.array(rep)] / np.linalg.norm(c[np.array(rep)])
    V = np.einsum("kpq,krs->pqrs", L, L, optimize=True)
    V32 = V.astype(np.float32).astype(np.float64)  # (pq|rs) are stored as real*4
    occ = np.arange(no)
    J, K = np.einsum("ppqq->pq", V), np.einsum("pqpq->pq", V)
    F = h + 2 * np.einsum("pqii->pq", V[:, :, occ][:, :, :, occ]) - np.einsum("piqi->pq", V[:, occ][:, :, :, occ])
    F = np.where(np.abs(F) < 1e-7, 0.0, F)
    f2 = np.concatenate([np.diag(F)] * 2)
    spin, orb = np.repeat([0, 1], n), np.tile(np.arange(n), 2)
    X = J[np.ix_(orb, orb)] - (spin[:, None] == spin[None, :]) * K[np.ix_(orb, orb)]
    ref = np.zeros(2 * n)
    ref[np.concatenate([occ, occ + n])] = 1

    def rows(pairs):
        B = np.tile(ref, (len(pairs), 1))
        for k, (hl, pt) in enumerate(pairs):
            B[k, np.asarray(hl, int) - 1] = 0
            B[k, np.asarray(pt, int) - 1] = 1
        return B

    def diag(B):  # hdig and hmp over the occupation changes
        D = B - ref
        return D @ f2 + 0.5 * np.einsum("kr,rs,ks->k", D, X, D), D @ f2

    S = rows(dets)
    hd, hm = diag(S)
    e, emp = (c * c) @ hd, (c * c) @ hm  # the "diagonal" root energy is the barycentre too
    rank = np.array([len(a) for a, _ in dets])
    out = dict.fromkeys(("e2mp", "e2vp", "e2b"), 0.0)
    key = [tuple(np.nonzero(r)[0]) for r in S]
    flip = {k: tuple(sorted((o + n) % (2 * n) for o in k)) for k in key}
    index = {k: i for i, k in enumerate(key)}
    for k in range(len(S)):
        partner = index[flip[key[k]]]
        if partner < k:  # the partner generated the flipped perturbers
            continue
        on, off = np.nonzero(S[k])[0], np.nonzero(S[k] == 0)[0]
        cand = []
        for a in itertools.combinations(off, 2):
            cand += [(r, a) for r in itertools.combinations(on, 2) if spin[list(r)].sum() == spin[list(a)].sum()]
        cand += [((r,), (a,)) for r in on for a in off if spin[r] == spin[a]]
        I = np.tile(S[k], (len(cand), 1))
        for t, (r, a) in enumerate(cand):
            I[t, list(r)], I[t, list(a)] = 0, 1
        D = (I * (1 - ref)).sum(1).astype(int) - rank[k]
        # rank changes allowed with the reference in S and no singles in S
        ok = (D == 2) | ((D == 1) & (rank[k] != 1))
        low = rank[k] >= 1 and rank[k] != 2
        ok |= (D <= 0) & low
        I, D, cand = I[ok], D[ok], [x for x, y in zip(cand, ok) if y]
        x = I @ (1 - S).T  # spin orbitals of I that S_j lacks
        near = x <= 2
        keep = ~near[:, :k].any(1) & (x[:, k:] > 0).all(1)
        twin = partner != k
        for t in np.nonzero(keep)[0]:
            r, a = cand[t]
            if not twin and D[t] == 2:
                if spin[list(r)].sum() == 1:
                    ra, aa = sorted(r), sorted(a)
                    (o1, o2), (a1, a2) = (ra[0], ra[1] - n), (aa[0], aa[1] - n)
                    if not (o1 < o2 or (o1 == o2 and a1 <= a2)):
                        continue
                    same = o1 == o2 and a1 == a2
                elif spin[r[0]] == 1:
                    continue
                else:
                    same = False
            else:
                same = False
            js = k + np.nonzero(near[t, k:])[0]
            b = sum(_element(I[t], S[j], F, V32, ref, spin, orb) * c[j] for j in js)
            nesp, lesp = (1 if twin else 0), int(twin and (partner in js))
            if D[t] == 2 and not twin and not same:
                nesp = 2 * nesp + 1
            w = (nesp + 1.0) / (lesp + 1.0)
            if b == 0.0 and D[t] == 2:
                continue
            dg, mp = diag(I[t: t + 1])
            out["e2mp"] += w * b * b / (emp - mp[0])
            out["e2vp"] += w * b * b / (e - dg[0])
            out["e2b"] += w * b * b / (e - dg[0])
    return {k: np.array([v]) for k, v in out.items()}


def _element(I, j, F, V, ref, spin, orb):
    """<I|H|j>, canonical phases, one or two differences."""
    p, q = np.nonzero((j > 0) & (I == 0))[0], np.nonzero((I > 0) & (j == 0))[0]
    core = np.cumsum(I * j) - I * j
    sign = -1.0 if int(core[p].sum() + core[q].sum()) % 2 else 1.0
    o, s = orb, spin
    if len(p) == 1:
        pp, qq = o[p[0]], o[q[0]]
        big = I if I @ (1 - ref) > j @ (1 - ref) else j
        v = F[pp, qq]
        for r in np.nonzero(big != ref)[0]:
            t = V[pp, qq, o[r], o[r]] - (V[pp, o[r], qq, o[r]] if s[r] == s[p[0]] else 0.0)
            v += (big[r] - ref[r]) * t
        return sign * v
    v = V[o[p[0]], o[q[0]], o[p[1]], o[q[1]]] * (s[p[0]] == s[q[0]])
    v -= V[o[p[0]], o[q[1]], o[p[1]], o[q[0]]] * (s[p[0]] == s[q[1]])
    return sign * v
