"""The work that users of this engine have it do, as cases that can be timed and checked.

Every case goes through the Python front end (`sbd_gb300.engine`) as a program would call it.  Problems are the
synthetic ones of `sbd_gb300.generators` (integrals from 32 Cholesky-like factors; strings drawn with weights
exp(-p / (norb / 4))), at the sizes of this repository's benchmark configurations, its request mix and its tests, and at
sizes between them.  A case has a `kind`:

  sigma     one product H C on device vectors, in FP64, on a block of FP32 vectors, or in double-float: the call that
            a program with its own eigensolver makes once per step
  davidson  a solve by the engine's own Davidson, FP64 or mixed, with the vectors brought back.  FP64 solves run a
            fixed number of steps (`--iteration` and `--block` of the reference's command line), mixed ones converge
            tightly, as for density matrices of the result
  batch     many small problems solved in lock step
  setup     a new problem: upload, excitation tables, diagonal, and both brought back (one per request of a
            sampled-bitstring loop)
  rdm       one- and two-particle density matrices of a vector
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sbd_gb300 import generators as G
from sbd_gb300.engine import FP64, MIXED, Engine, TPBProblem, batch_davidson

_engine = None


def engine() -> Engine:
    """The process's one context: a program keeps it for as long as it runs."""
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


def sigma(name, norb, nocc, na, nb, precision, nvec=1):
    return {"name": name, "kind": "sigma", "norb": norb, "nocc": nocc, "na": na, "nb": nb, "precision": precision,
            "nvec": nvec}


def listed():
    return [
        # the smallest problems (the norb-12 batch's sizes) one product at a time: launches and latency
        sigma("sigma f64 norb12 161x187", 12, 4, 161, 187, "f64"),
        # an ordinary small molecule: the benchmark's configuration 0, 113 nonzeros a row
        sigma("sigma f64 norb16 800x800", 16, 5, 800, 800, "f64"),
        # the request that dominates the serving mix: tens of singles a string, 771 nonzeros a row
        sigma("sigma f64 norb24 3274x3935", 24, 8, 3274, 3935, "f64"),
        # the benchmark's headline problem, 78 nonzeros a row
        sigma("sigma f64 norb36 6000x6000", 36, 12, 6000, 6000, "f64"),
        # the largest: half a nonzero a row, a stream through memory (odd beta count: rows start unaligned)
        sigma("sigma f64 norb58 12000x11999", 58, 16, 12000, 11999, "f64"),
        # FP32 block product of the mixed solver, at a request's size
        sigma("sigma f32x3 norb32 2011x1703", 32, 11, 2011, 1703, "f32", 3),
        # a small FP64 solve: 30 steps of one root
        {"name": "davidson f64 norb16 800x800", "kind": "davidson", "norb": 16, "nocc": 5, "na": 800, "nb": 800,
         "nroots": 1, "max_nb": 15, "max_it": 2, "precision": "f64"},
        # the headline solve's steps: two roots, one full subspace of 24
        {"name": "davidson f64 norb36 6000x6000", "kind": "davidson", "norb": 36, "nocc": 12, "na": 6000, "nb": 6000,
         "nroots": 2, "max_nb": 24, "max_it": 1, "precision": "f64"},
        # a request of the serving mix in the mixed form, to convergence
        {"name": "davidson mixed norb24 1207x903", "kind": "davidson", "norb": 24, "nocc": 8, "na": 1207, "nb": 903,
         "nroots": 1, "max_nb": 20, "max_it": 40, "precision": "mixed"},
        # the norb-12 batch, four roots each
        {"name": "batch f64 24 problems", "kind": "batch", "norb": 12, "nocc": 4, "count": 24, "nroots": 4,
         "max_nb": 24, "max_it": 1, "precision": "f64"},
        # a request's arrival
        {"name": "setup norb40 1731x2050", "kind": "setup", "norb": 40, "nocc": 13, "na": 1731, "nb": 2050},
        # density matrices of a solution
        {"name": "rdm norb24 301x420", "kind": "rdm", "norb": 24, "nocc": 8, "na": 301, "nb": 420},
    ]


# --- drawing --------------------------------------------------------------------------------------------------

_NOCC = {12: 4, 16: 5, 24: 8, 32: 11, 36: 12, 40: 13, 48: 16, 58: 16}


def _strings(rng, norb, low, high):
    high = min(high, math.comb(norb, _NOCC[norb]))
    return int(round(math.exp(rng.uniform(math.log(min(low, high)), math.log(high)))))


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "davidson", "davidson", "batch", "setup", "rdm"])
    if kind == "batch":
        mixed = rng.random() < 0.5
        return {"kind": "batch", "norb": 12, "nocc": 4, "count": rng.randint(3, 24), "nroots": rng.randint(1, 4),
                "max_nb": rng.choice([16, 20, 24]), "max_it": 40 if mixed else 1,
                "precision": "mixed" if mixed else "f64"}
    if kind == "rdm":
        norb = rng.choice([12, 16, 24])
        return {"kind": "rdm", "norb": norb, "nocc": _NOCC[norb], "na": _strings(rng, norb, 50, 400),
                "nb": _strings(rng, norb, 50, 400)}
    if kind == "setup":
        norb = rng.choice([12, 24, 32, 36, 40, 48])
        return {"kind": "setup", "norb": norb, "nocc": _NOCC[norb], "na": _strings(rng, norb, 100, 3000),
                "nb": _strings(rng, norb, 100, 3000)}
    if kind == "davidson":
        mixed = rng.random() < 0.4
        norb = rng.choice([16, 24, 32, 36, 40, 48])
        c = {"kind": "davidson", "norb": norb, "nocc": _NOCC[norb], "na": _strings(rng, norb, 200, 1500),
             "nb": _strings(rng, norb, 200, 1500)}
        if mixed:
            return {**c, "nroots": 1, "max_nb": 20, "max_it": 40, "precision": "mixed"}
        return {**c, "nroots": rng.randint(1, 3), "max_nb": rng.choice([12, 16, 20, 24]), "max_it": 1,
                "precision": "f64"}
    norb = rng.choice([12, 16, 24, 32, 36, 40, 48, 58])
    high = 3500 if norb <= 24 else 7000
    precision = rng.choice(["f64", "f64", "f32", "df"])
    c = {"kind": "sigma", "norb": norb, "nocc": _NOCC[norb], "na": _strings(rng, norb, 100, high),
         "nb": _strings(rng, norb, 100, high), "precision": precision, "nvec": 1}
    if precision == "f32":
        c["nvec"] = rng.randint(1, 4)
    return c


# --- inputs ----------------------------------------------------------------------------------------------------

def _draw_strings(norb, nocc, count, rng):
    """`count` distinct strings with the generators' distribution: occupied orbitals drawn one after another without
    replacement, weights exp(-p / (norb / 4)).  The `nocc` smallest of exponential variates over the weights are such
    a draw, so a whole array of strings is drawn at once."""
    total = math.comb(norb, nocc)
    if 2 * count >= total:
        return G.draw_strings(norb, nocc, count, rng)
    w = np.exp(-np.arange(norb) / (norb / 4.0))
    found = np.zeros(0, dtype=np.uint64)
    while found.size < count:
        e = rng.exponential(size=(2 * count, norb)) / w
        occ = np.argpartition(e, nocc - 1, axis=1)[:, :nocc].astype(np.uint64)
        new = np.bitwise_or.reduce(np.uint64(1) << occ, axis=1)
        found = np.concatenate([found, new])
        found = found[np.sort(np.unique(found, return_index=True)[1])]  # the first of each, in the order drawn
    return np.sort(found[:count])


def _inputs(case, seed):
    """(integrals, alpha strings, beta strings) of a case.  A new problem's tables come back as arrays, whose lengths
    the strings decide: there every seed has the same strings but for the order of neighbouring orbitals."""
    norb = case["norb"]
    own = np.random.SeedSequence([seed, norb, case["na"], case["nb"]])
    rng = np.random.Generator(np.random.PCG64(own))
    ints = G.make_integrals(norb, 2 * case["nocc"], rng)
    if case["kind"] != "setup":
        return ints, *(_draw_strings(norb, case["nocc"], case[n], rng) for n in ("na", "nb"))
    fixed = np.random.Generator(np.random.PCG64(case["na"] * 10_000 + case["nb"]))
    lists = [_draw_strings(norb, case["nocc"], case[n], fixed) for n in ("na", "nb")]
    order = np.arange(norb)
    for p in np.nonzero(rng.random(norb // 2) < 0.5)[0]:
        order[[2 * p, 2 * p + 1]] = order[[2 * p + 1, 2 * p]]
    one = np.uint64(1)
    bits = np.arange(norb, dtype=np.uint64)
    return ints, *(np.sort(np.bitwise_or.reduce(((s[:, None] >> bits) & one) << order.astype(np.uint64), axis=1))
                   for s in lists)


def _vectors(case, seed, nvec):
    """Vectors like those a solve meets: normalised, a weight for each string over three orders of magnitude, random
    signs and sizes on top."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    dev = {"device": "cuda", "dtype": torch.float64}

    def weights(n):
        return 10.0 ** (-3.0 * torch.rand(n, 1, generator=g, **dev))

    v = []
    for _ in range(nvec):
        x = torch.randn(case["na"], case["nb"], generator=g, **dev)
        x *= weights(case["na"])
        x *= weights(case["nb"]).T
        v.append((x / x.norm()).reshape(-1))
    return torch.stack(v)


def _split(x):
    """FP64 values as double-float pairs (the leading FP32 value and the rest in FP32)."""
    hi = x.float()
    return torch.stack([hi, (x - hi.double()).float()], dim=-1).contiguous()


def _sigma_input(case, seed):
    x = _vectors(case, seed, case["nvec"])
    if case["precision"] == "f32":
        return x.float()
    return _split(x[0]) if case["precision"] == "df" else x[0].contiguous()


def _batch_problems(case, seed):
    r = np.random.Generator(np.random.PCG64(case["count"]))  # the sizes belong to the case
    sizes = np.exp(r.uniform(math.log(50), math.log(495), size=(case["count"], 2))).round().astype(int)
    return [_inputs({**case, "na": int(na), "nb": int(nb)}, seed * 1000 + i) for i, (na, nb) in enumerate(sizes)]


def _problem(norb, inputs):
    ints, a, b = inputs
    return TPBProblem(engine(), norb, a, b, ints.h1, ints.eri, ints.ecore)


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "batch":
        s["problems"] = [_problem(case["norb"], q) for q in _batch_problems(case, seed)]
        for p in s["problems"]:
            p.build_tables()
        return s
    inputs = _inputs(case, seed)
    if case["kind"] == "setup":
        s["inputs"] = inputs
        return s
    s["problem"] = _problem(case["norb"], inputs)
    s["problem"].diag_terms()  # builds the tables and the diagonal
    if case["kind"] == "sigma":
        s["C"] = _sigma_input(case, seed)
        s["S"] = torch.empty_like(s["C"])
    elif case["kind"] == "rdm":
        s["W"] = _vectors(case, seed, 1)[0].contiguous()
    torch.cuda.synchronize()
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "sigma":
        p, c, s = state["problem"], state["C"], state["S"]
        stream = torch.cuda.current_stream().cuda_stream
        if case["precision"] == "f64":
            p.sigma_device(c.data_ptr(), s.data_ptr(), stream=stream)
        elif case["precision"] == "df":
            p.sigma_df_device(c.data_ptr(), s.data_ptr(), stream=stream)
        else:
            p.sigma_mixed_block_device(c.data_ptr(), s.data_ptr(), case["nvec"], stream=stream)
        return s
    if case["kind"] == "davidson":
        mixed = case["precision"] == "mixed"
        r = state["problem"].davidson(nroots=case["nroots"], max_nb=case["max_nb"], max_it=case["max_it"],
                                      eps=1e-11, init=1 if mixed else 0, precision=MIXED if mixed else FP64)
        return {"energies": r.energies, "vectors": r.vectors}
    if case["kind"] == "batch":
        rs = batch_davidson(engine(), state["problems"], nroots=case["nroots"], max_nb=case["max_nb"], eps=1e-11,
                            max_it=case["max_it"], want_vectors=True,
                            precision=MIXED if case["precision"] == "mixed" else FP64)
        return {"energies": np.stack([r.energies for r in rs]),
                "vectors": np.concatenate([r.vectors.reshape(-1) for r in rs])}
    if case["kind"] == "rdm":
        one, two = state["problem"].rdm(state["W"].data_ptr())
        return {"one": one, "two": two}
    p = _problem(case["norb"], state["inputs"])
    p.build_tables()
    out = {"hii": p.diag_terms(), "alpha": p.export_tables(0), "beta": p.export_tables(1)}
    p.close()
    return {"hii": out["hii"], **{f"{s}_{k}": v.view(np.int64) if v.dtype == np.uint64 else v
                                  for s in ("alpha", "beta") for k, v in out[s].items()}}


# --- the same in plain torch, 64 bits --------------------------------------------------------------------------

def _occupation(strings, norb):
    bits = torch.from_numpy(strings.view(np.int64).copy()).to(_device())
    return ((bits[:, None] >> torch.arange(norb, device=bits.device)) & 1).double()


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pairs(occ, distance):
    """(bra, ket) index pairs whose strings differ in `distance` occupied orbitals."""
    n, nocc = occ.shape[0], int(occ[0].sum())
    o = occ.float()
    found = [torch.nonzero((o[i:i + 2048] @ o.T) == nocc - distance) + torch.tensor([i, 0], device=occ.device)
             for i in range(0, n, 2048)]
    f = torch.cat(found)
    return f[:, 0], f[:, 1]


def _moved(occ, bra, ket, count):
    """Orbitals left and orbitals entered going from bra to ket, each ascending, [pairs, count]."""
    d = occ[bra] - occ[ket]
    orb = torch.arange(occ.shape[1], device=occ.device).expand_as(d)
    big = occ.shape[1]
    left = torch.where(d > 0, orb, big).sort(dim=1).values[:, :count]
    entered = torch.where(d < 0, orb, big).sort(dim=1).values[:, :count]
    return left, entered


def _between(occ, i, a):
    """Sign of moving an electron from orbital i to a: (-1) to the number of occupied ones strictly between."""
    cum = torch.cat([torch.zeros_like(occ[:, :1]), occ.cumsum(1)], dim=1)
    lo, hi = torch.minimum(i, a), torch.maximum(i, a)
    n = cum.gather(1, hi[:, None]) - cum.gather(1, lo[:, None] + 1)
    return 1.0 - 2.0 * (n[:, 0].long() % 2).double()


def _pair_index(i, j):
    hi, lo = torch.maximum(i, j), torch.minimum(i, j)
    return hi * (hi + 1) // 2 + lo


def _integrals(ints, norb):
    dev = _device()
    npair = norb * (norb + 1) // 2
    p, q = np.tril_indices(npair)
    K = np.zeros((npair, npair))
    K[p, q] = K[q, p] = ints.eri[p * (p + 1) // 2 + q]
    return torch.from_numpy(ints.h1.reshape(norb, norb)).to(dev), torch.from_numpy(K).to(dev)


def _spin_tables(occ, h1, K):
    """Same-spin matrix elements (all electrons of one spin created before the other's): singles (bra, ket, pair
    index, sign, h + exchange part) and doubles (bra, ket, value)."""
    norb = occ.shape[1]
    orb = torch.arange(norb, device=occ.device)
    diag = _pair_index(orb, orb)
    bra, ket = _pairs(occ, 1)
    left, entered = _moved(occ, bra, ket, 1)
    i, a = left[:, 0], entered[:, 0]
    P = _pair_index(i, a)
    val = h1[a, i]
    for j in range(norb):
        jj = torch.full_like(i, j)
        val = val + occ[bra, j] * (K[P, diag[j]] - K[_pair_index(a, jj), _pair_index(jj, i)])
    singles = (bra, ket, P, _between(occ[bra], i, a), val)
    bra, ket = _pairs(occ, 2)
    left, entered = _moved(occ, bra, ket, 2)
    (i, j), (a, b) = left.T, entered.T
    sign = _between(occ[bra], i, a)
    mid = occ[bra].clone()
    mid.scatter_(1, i[:, None], 0.0).scatter_(1, a[:, None], 1.0)
    sign = sign * _between(mid, j, b)
    val = K[_pair_index(a, i), _pair_index(b, j)] - K[_pair_index(a, j), _pair_index(b, i)]
    return singles, (bra, ket, sign * val)


def _eta(occ_a, occ_b):
    """Sign between the interleaved and the spin-blocked determinant: pairs (alpha p, beta q < p)."""
    below = torch.cat([torch.zeros_like(occ_b[:, :1]), occ_b.cumsum(1)[:, :-1]], dim=1)
    return 1.0 - 2.0 * ((occ_a @ below.T).round().long() % 2).double()


def _diagonal(occ_a, occ_b, h1, K):
    norb = occ_a.shape[1]
    orb = torch.arange(norb, device=occ_a.device)
    d = _pair_index(orb, orb)
    J = K[d][:, d]
    X = K[_pair_index(orb[:, None], orb[None]), _pair_index(orb[:, None], orb[None])]

    def own(o):
        return o @ h1.diagonal() + 0.5 * ((o @ (J - X)) * o).sum(1)

    return own(occ_a)[:, None] + own(occ_b)[None] + occ_a @ J @ occ_b.T


def _same_spin(out, C, singles, doubles, occ_other, K):
    """out += the same-spin elements on the rows of C; a single also feels the other spin's electrons."""
    norb = occ_other.shape[1]
    orb = torch.arange(norb, device=C.device)
    J = K[:, _pair_index(orb, orb)] @ occ_other.T
    step = max(1, 100_000_000 // max(1, C.shape[1]))
    bra, ket, P, sign, val = singles
    for s in range(0, bra.numel(), step):
        t = slice(s, s + step)
        out.index_add_(0, bra[t], (val[t, None] + J[P[t]]).mul_(sign[t, None]).mul_(C[ket[t]]))
    bra, ket, val = doubles
    for s in range(0, bra.numel(), step):
        t = slice(s, s + step)
        out.index_add_(0, bra[t], C[ket[t]].mul_(val[t, None]))


def _product(norb, inputs, C):
    """H C for the rows of C, in the interleaved convention."""
    ints, astr, bstr = inputs
    h1, K = _integrals(ints, norb)
    oa, ob = _occupation(astr, norb), _occupation(bstr, norb)
    sa, da = _spin_tables(oa, h1, K)
    sb, db = _spin_tables(ob, h1, K)
    eta, hii = _eta(oa, ob), _diagonal(oa, ob, h1, K)
    outs = []
    for c in C:
        x = c.double().reshape(len(astr), len(bstr)) * eta
        out = hii * x
        _same_spin(out, x, sa, da, ob, K)
        xt = x.T.contiguous()
        ot = torch.zeros_like(xt)
        _same_spin(ot, xt, sb, db, oa, K)
        # alpha single times beta single: alpha pairs whose bra is the same row after one another
        step = max(1, 100_000_000 // max(1, sb[0].numel()))
        for s in range(0, sa[0].numel(), step):
            t = slice(s, s + step)
            term = K[sa[2][t]][:, sb[2]].mul_(sb[3][None]).mul_(sa[3][t, None]).mul_(x[sa[1][t]][:, sb[1]])
            rows = torch.zeros(term.shape[0], x.shape[1], dtype=x.dtype, device=x.device)
            rows.index_add_(1, sb[0], term)
            out.index_add_(0, sa[0][t], rows)
        outs.append((out + ot.T).mul_(eta).reshape(-1))
    return torch.stack(outs)


def _annihilated(occ, orbs):
    """Removing one or two orbitals (in order) from every string: [(string, remaining string's index, sign)] per
    orbital tuple, and the number of remaining strings."""
    norb = occ.shape[1]
    weight = 2 ** torch.arange(norb, device=occ.device)
    found, keys = [], []
    for tup in orbs:
        o, sign = occ.clone(), torch.ones(occ.shape[0], dtype=occ.dtype, device=occ.device)
        ok = torch.ones(occ.shape[0], dtype=torch.bool, device=occ.device)
        for p in tup:
            ok &= o[:, p] > 0
            sign = sign * (1.0 - 2.0 * (o[:, :p].sum(1).long() % 2).double())
            o[:, p] = 0.0
        idx = torch.nonzero(ok)[:, 0]
        key = (o[idx].long() * weight).sum(1)
        found.append((idx, key, sign[idx]))
        keys.append(key)
    rest = torch.unique(torch.cat(keys))
    return [(i, torch.searchsorted(rest, k), s) for i, k, s in found], rest.numel()


def _same_spin_rdm(occ, x):
    """<a+ b+ d c> of one spin over rows x[string, other], as [a, b, c, d]."""
    norb = occ.shape[1]
    pairs = [(a, b) for a in range(norb) for b in range(a)]
    rem, n = _annihilated(occ, pairs)
    small = torch.zeros(len(pairs), len(pairs), dtype=x.dtype, device=x.device)
    step = max(1, 200_000_000 // max(1, n * len(pairs)))
    for s in range(0, x.shape[1], step):
        T = torch.zeros(len(pairs), n, x[:, s:s + step].shape[1], dtype=x.dtype, device=x.device)
        for q, (i, k, sg) in enumerate(rem):
            T[q, k] = sg[:, None] * x[i, s:s + step]
        T = T.reshape(len(pairs), -1)
        small += T @ T.T
    full = torch.zeros(norb, norb, len(pairs), dtype=x.dtype, device=x.device)
    a, b = torch.tensor(pairs, device=x.device).T
    full[a, b], full[b, a] = small, -small
    out = torch.zeros(norb, norb, norb, norb, dtype=x.dtype, device=x.device)
    out[:, :, a, b], out[:, :, b, a] = full, -full
    return out


def _rdm(case, seed):
    norb = case["norb"]
    _, astr, bstr = _inputs(case, seed)
    oa, ob = _occupation(astr, norb), _occupation(bstr, norb)
    x = _vectors(case, seed, 1)[0].to(oa.device).reshape(len(astr), len(bstr)) * _eta(oa, ob)
    aa, bb = _same_spin_rdm(oa, x), _same_spin_rdm(ob, x.T.contiguous())
    ra, na = _annihilated(oa, [(p,) for p in range(norb)])
    rb, nb = _annihilated(ob, [(p,) for p in range(norb)])
    ab = torch.zeros(norb * norb, norb * norb, dtype=x.dtype, device=x.device)
    cols = torch.zeros(norb, x.shape[0], nb, dtype=x.dtype, device=x.device)  # beta orbital removed
    for q, (i, k, sg) in enumerate(rb):
        cols[q][:, k] = x[:, i] * sg
    # every alpha remainder in turn: a block of them holds (orbital, remainder) rows of cols
    src = torch.full((norb, na), -1, dtype=torch.long, device=x.device)
    sgn = torch.zeros(norb, na, dtype=x.dtype, device=x.device)
    for p, (i, k, sg) in enumerate(ra):
        src[p, k], sgn[p, k] = i, sg
    step = max(1, 200_000_000 // (norb * norb * max(1, nb)))
    for s in range(0, na, step):
        i, sg = src[:, s:s + step], sgn[:, s:s + step]
        T = cols[:, i.clamp(min=0)] * sg[None, :, :, None]  # [q, p, remainder, beta remainder]
        T = T.permute(1, 0, 2, 3).reshape(norb * norb, -1)
        ab += T @ T.T
    ab = ab.reshape(norb, norb, norb, norb)  # [a, b, c, d]: alpha c -> a, beta d -> b
    one = []
    for occ, y in ((oa, x), (ob, x.T.contiguous())):
        rem, n = _annihilated(occ, [(p,) for p in range(norb)])
        T = torch.zeros(norb, n, y.shape[1], dtype=y.dtype, device=y.device)
        for p, (i, k, sg) in enumerate(rem):
            T[p, k] = sg[:, None] * y[i]
        T = T.reshape(norb, -1)
        one.append((T @ T.T).reshape(-1))
    mixed = torch.zeros(4, norb, norb, norb, norb, dtype=x.dtype, device=x.device)
    orb = torch.arange(norb, device=x.device)
    a, b, c, d = (t.reshape(-1) for t in torch.meshgrid(orb, orb, orb, orb, indexing="ij"))  # c -> a, d -> b
    v = ab.reshape(-1)
    # the reference's rule where both electrons move: each pair of spin orbitals (2p alpha, 2p + 1 beta) is put in
    # ascending order, and the entry's block goes by the spins of the pair that is left
    i, a2, j, b2 = 2 * c, 2 * a, 2 * d + 1, 2 * b + 1
    lo, hi, left, right = torch.minimum(i, j), torch.maximum(i, j), torch.minimum(a2, b2), torch.maximum(a2, b2)
    same = ((a == c) | (b == d)) | ((lo & 1) == (left & 1))
    one_moves = (a == c) | (b == d)
    lo, hi = torch.where(one_moves, i, lo), torch.where(one_moves, j, hi)
    left, right = torch.where(one_moves, a2, left), torch.where(one_moves, b2, right)
    c2, d2 = torch.where(same, lo, hi) // 2, torch.where(same, hi, lo) // 2
    mixed.index_put_(((lo & 1) + 2 * (hi & 1), left // 2, right // 2, c2, d2), v, accumulate=True)
    mixed.index_put_(((hi & 1) + 2 * (lo & 1), right // 2, left // 2, d2, c2), v, accumulate=True)
    flat = [t.permute(3, 2, 1, 0).reshape(-1) for t in (aa, mixed[1], mixed[2], bb)]
    return {"one": torch.stack(one), "two": torch.stack(flat)}


def exact(case, seed):
    if case["kind"] == "sigma":
        x = _vectors(case, seed, case["nvec"])
        if case["precision"] == "f32":
            return _product(case["norb"], _inputs(case, seed), x.float())
        if case["precision"] == "df":
            pair = _split(x[0])
            y = _product(case["norb"], _inputs(case, seed), [pair[:, 0].double() + pair[:, 1].double()])[0]
            hi = y.float().double()  # laid out as pairs: the leading value, and the rest
            return torch.stack([hi, y - hi], dim=-1)
        return _product(case["norb"], _inputs(case, seed), x)[0]
    if case["kind"] == "rdm":
        return _rdm(case, seed)
    if case["kind"] == "setup":
        ints, astr, bstr = _inputs(case, seed)
        h1, K = _integrals(ints, case["norb"])
        hii = _diagonal(_occupation(astr, case["norb"]), _occupation(bstr, case["norb"]), h1, K)
        return {"hii": hii.reshape(-1)}
    return None  # solves: their vectors depend on the number of steps taken


# --- what a pass cannot do without -----------------------------------------------------------------------------

def _counts(case):
    """(singles, doubles) of each spin for this size (they differ by a few percent between seeds)."""
    out = []
    for astr in _inputs(case, 0)[1:]:
        occ = _occupation(astr, case["norb"])
        out.append((_pairs(occ, 1)[0].numel(), _pairs(occ, 2)[0].numel()))
    return out


def work(case):
    if case["kind"] == "batch":
        n = [len(a) * len(b) for _, a, b in _batch_problems(case, 0)]
        steps = case["max_nb"] * (case["max_it"] if case["precision"] == "f64" else 2)
        # each step: the basis, its products and the new vectors once
        return {"bytes": 8.0 * sum(n) * steps * case["nroots"] * case["max_nb"], "flops": 0.0}
    norb, na, nb = case["norb"], case["na"], case["nb"]
    N, npair = na * nb, norb * (norb + 1) // 2
    if case["kind"] == "setup":
        (sa, da), (sb, db) = _counts(case)
        return {"bytes": 8.0 * (N + na + nb + npair * (npair + 1) / 2) + 24.0 * (sa + sb) + 32.0 * (da + db),
                "flops": 0.0}
    (sa, da), (sb, db) = _counts(case)
    nnz = (sa + da) * nb + (sb + db) * na + sa * sb
    if case["kind"] == "rdm":
        return {"bytes": 8.0 * N + 8.0 * (2 * norb ** 2 + 4 * norb ** 4), "flops": 2.0 * (nnz + N)}
    if case["kind"] == "sigma":
        size = {"f64": 8, "df": 8, "f32": 4}[case["precision"]]
        return {"bytes": (2.0 * case["nvec"] + 1) * size * N + 24.0 * (sa + da + sb + db),
                "flops": 2.0 * case["nvec"] * (nnz + N)}
    k, nb_max = case["nroots"], case["max_nb"]
    steps = nb_max * case["max_it"] if case["precision"] == "f64" else 2 * nb_max
    # per step: k products, and the basis and its products (half of max_nb of each on average) read for the Ritz
    # vectors and residuals and once more for the orthogonalisation
    return {"bytes": 8.0 * N * steps * (3 * k + 1.5 * nb_max),
            "flops": 2.0 * steps * k * ((nnz + N) + 2.5 * N * nb_max / 2)}
