"""Performance cases of the resident CKKS library, through its public entry points.

Each case is one call (or the short call sequence) that a user's program makes
on ciphertexts it already holds: batched ciphertext operations through a plan,
a linear transform, forward and inverse transforms, ModRaise, pointwise
arithmetic, and a burst of requests through the server. Ring sizes, tower
counts, prime widths, digit widths and batch sizes are those of this
repository's tests and benchmark.

Every result is an exact residue, so outputs compare bit for bit. `exact`
recomputes them from the definitions with 64-bit integer tensor arithmetic and
none of the library's kernels.

Contexts (twiddle tables, per-level constants, resident keys) are what a
program builds once and keeps, so states of one chain share one context; keys
come from fixed seeds, ciphertexts and plaintexts from the state's seed. No
output buffer is an input, so a pass can be repeated on the same state.
"""
import collections
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-resident-library_b200"))
import gpufhe_b200 as G  # noqa: E402

ROT_STEPS = tuple(s << j for j in range(8) for s in (1, -1))    # slot rotations +-1, +-2, ... +-2^7


# ------------------------------------------------------------------ cases
def _case(name, kind, logn, towers, alpha, special, count, bits=50, low=0, n1=0, n2=0, depth=0):
    """A chain of one 60-bit and towers-1 `bits`-bit primes with `special`
    60-bit primes and digits of `alpha` towers; `count` operations at levels
    low..towers (low = 0: all at `towers`)."""
    return {"name": name, "kind": kind, "logn": logn, "towers": towers, "bits": bits, "alpha": alpha,
            "special": special, "count": count, "low": low or towers, "n1": n1, "n2": n2, "depth": depth}


def listed():
    return [
        # one product on the smallest chain in use (N = 2^15, 4 + 2 towers): latency and launches
        _case("product_one", "product", 15, 4, 2, 2, 1),
        # a handful of products at the deepest levels of the 12-tower chain: a program with a few ciphertexts in hand
        _case("product_few", "product", 16, 12, 3, 3, 5, low=9),
        # the batched throughput form: 128 independent products of uneven level
        _case("product_batch", "product", 16, 12, 3, 3, 128, low=4),
        # one serving-like step: products, rotations, keyswitches and rescales of uneven level, wide digits
        _case("mixed_step", "mixed", 14, 24, 8, 8, 13, low=4),
        # slot rotations of independent ciphertexts, a key per index
        _case("rotate_batch", "rotate", 16, 10, 3, 3, 48),
        # sixteen rotations of each of three ciphertexts sharing one ModUp
        _case("rotate_hoisted", "hoisted", 16, 10, 3, 3, 48),
        # baby-step giant-step linear transform on a bootstrapping-like chain (55-bit primes, digits of two)
        _case("linear_transform", "lintrans", 13, 15, 2, 2, 1, bits=55, n1=4, n2=4),
        # plaintext embedding: batched forward transforms into every tower
        _case("embed_batch", "embed", 16, 12, 3, 3, 64),
        # eval-form products back to coefficients: batched inverse transforms
        _case("inverse_batch", "inverse", 16, 12, 3, 3, 64),
        # ModRaise of a few ciphertexts, the first step of bootstrapping: inverse then forward transforms
        _case("modraise_few", "modraise", 16, 10, 3, 3, 7),
        # sums, differences, plaintext and integer products of a batch, uneven levels
        _case("pointwise_batch", "pointwise", 16, 10, 3, 3, 96, low=5),
        # a burst of encrypted requests through the server: chains of products and rotations from host buffers
        _case("serve_burst", "serve", 15, 24, 8, 8, 14, low=6, depth=3),
    ]


# Most work and memory of a drawn case, as tower transforms of N log N and bytes: those of product_batch.
def _budget():
    big = next(c for c in listed() if c["name"] == "product_batch")
    return _transform_points(big), _words(big) * 8


KINDS = ("product", "product", "mixed", "rotate", "hoisted", "lintrans", "embed", "inverse", "modraise", "pointwise",
         "serve")


def draw(rng):
    most, room = _budget()
    kind = rng.choice(KINDS)
    logn = rng.randint(13, 15) if kind in ("lintrans", "serve") else rng.randint(12, 16)
    towers = rng.randint(3, 24)
    alpha = rng.randint(2, min(8, towers))
    special = max(1, alpha - rng.randint(0, 1))
    bits = 55 if kind == "lintrans" or rng.random() < 0.15 else 50
    c = _case("", kind, logn, towers, alpha, special, 1, bits=bits, low=rng.randint(2, towers))
    if kind == "lintrans":
        c["n1"], c["n2"], c["low"] = rng.randint(2, 6), rng.randint(2, 5), towers
    if kind == "serve":
        c["depth"] = rng.randint(1, 4)
        c["low"] = max(c["low"], min(towers, c["depth"] + 1))
    if kind in ("embed", "inverse", "modraise"):
        c["low"] = towers
    top = 128 if kind in ("product", "rotate", "hoisted", "embed", "inverse", "pointwise") else 32
    fits = [k for k in range(1, top + 1)
            if k == 1 or (_transform_points({**c, "count": k}) <= 0.9 * most and _words({**c, "count": k}) * 8 <= 0.9 * room)]
    c["count"] = 1 if kind == "lintrans" else min(max(fits), max(1, round(math.exp(rng.uniform(0, math.log(max(fits) + 0.5))))))
    del c["name"]
    return c


def _levels(case):
    """Level of each operation: spread over low..towers, the same for every
    seed; hoisted rotations come in groups of 16 that share one ciphertext."""
    span = case["towers"] - case["low"] + 1
    group = 16 if case["kind"] == "hoisted" else 1
    return [case["low"] + (7 * (i // group) + 3) % span for i in range(case["count"])]


def _modes(case):
    """Operation of each plan entry."""
    kind, cycle = case["kind"], (G.EVALMULT_RESCALE, G.ROTATE, G.EVALMULT_RESCALE, G.KEYSWITCH, G.RESCALE)
    one = {"product": G.EVALMULT_RESCALE, "rotate": G.ROTATE, "hoisted": G.ROTATE_HOISTED}
    return [one.get(kind, cycle[i % len(cycle)]) for i in range(case["count"])]


def _galois(step, n):
    return pow(5, step, 2 * n) if step >= 0 else pow(pow(5, -step, 2 * n), -1, 2 * n)


def _chain_ops(case):
    """The server's request chains: (start level, [(mode, galois)])."""
    n, reqs = 1 << case["logn"], []
    for i, level in enumerate(_levels(case)):
        ops = []
        for d in range(min(case["depth"], level - 1)):
            ops.append((G.EVALMULT_RESCALE, 0))
            if (i + d) % 2:
                ops.append((G.ROTATE, _galois(ROT_STEPS[(i + d) % len(ROT_STEPS)], n)))
        reqs.append((level, ops))
    return reqs


# ------------------------------------------------------------------ what a pass cannot do without
def _op_cost(mode, level, alpha, special):
    """(input towers, output towers, tower transforms, products of towers) of one operation."""
    parts = -(-level // alpha)
    up = parts * (level + special) - level
    conv = up * min(alpha, level) + 2 * special * level
    if mode == G.RESCALE:
        return level, level - 1, level, 2 * level
    if mode == G.EVALMULT_RESCALE:
        return 4 * level, 2 * (level - 1), level + up + 2 * (special + 1) + 2 * (level - 1), \
            conv + 2 * parts * (level + special) + 8 * level
    return (level if mode == G.KEYSWITCH else 2 * level), 2 * level, level + up + 2 * special + 2 * level, \
        conv + 2 * parts * (level + special) + 2 * level


def _cost(case):
    """(words read and written, tower transforms, tower products) of one pass."""
    n, kind, a, k = 1 << case["logn"], case["kind"], case["alpha"], case["special"]
    T, cnt = case["towers"], case["count"]
    key = 2 * -(-T // a) * (T + k)                                  # towers of one eval key
    if kind in ("product", "mixed", "rotate", "hoisted"):
        tot = np.zeros(4)
        for i, (lv, md) in enumerate(zip(_levels(case), _modes(case))):
            c = np.array(_op_cost(md, lv, a, k), float)
            if md == G.ROTATE_HOISTED and i % 16:                   # ModUp and c1 shared by up to 16 rotations
                c[0] -= lv
                c[2] -= -(-lv // a) * (lv + k)
            tot += c
        keys = len({_op_key(case, i) for i in range(cnt)} - {None})
        return (tot[0] + tot[1] + keys * key) * n, tot[2], tot[3]
    if kind == "lintrans":
        rot = case["n1"] + case["n2"] - 2
        c = _op_cost(G.ROTATE, T, a, k)
        d = case["n1"] * case["n2"]
        return (4 * T + d * T + rot * key) * n, rot * c[2], rot * c[3] + 2 * d * T
    if kind == "embed":
        return cnt * (1 + T) * n, cnt * T, 0
    if kind == "inverse":
        return 3 * cnt * T * n, cnt * T, cnt * T
    if kind == "modraise":
        return cnt * (2 + 2 * T) * n, cnt * (2 + 2 * T), 0
    if kind == "pointwise":
        words, prod = 0, 0
        for i, lv in enumerate(_levels(case)):
            kd = _pw_kind(i)
            words += lv * (4 + {G.PW_ADD: 2, G.PW_SUB: 2, G.PW_MUL_INT: 0}.get(kd, 1))
            prod += 2 * lv if kd in (G.PW_MUL_PT, G.PW_MUL_INT) else 0
        return words * n, 0, prod
    words, tr, prod = 0, 0, 0                                       # serve
    used = set()
    for level, ops in _chain_ops(case):
        words += 2 * level
        for md, gal in ops:
            c = _op_cost(md, level, a, k)
            tr, prod = tr + c[2], prod + c[3]
            used.add(gal)
            level -= md == G.EVALMULT_RESCALE
        words += 2 * level
    return (words + len(used) * key) * n, tr, prod


def _transform_points(case):
    _, tr, prod = _cost(case)
    return (1 << case["logn"]) * (tr * case["logn"] / 2 + prod)


def _words(case):
    """Device words of a state: operands, results and workspace."""
    n, a, k, T = 1 << case["logn"], case["alpha"], case["special"], case["towers"]
    per = sum(6 * lv + -(-lv // a) * (lv + k) + 5 * lv + 2 + 2 * k for lv in _levels(case))
    if case["kind"] == "lintrans":
        per *= 2 * case["n1"] + case["n2"]
    return per * n


def work(case):
    """Inputs and keys read once and outputs written once. Arithmetic: ten
    FP64 operations for an exact butterfly (a six-operation modular product, a
    sum, a difference and the share of the reductions) and eight for a product."""
    words, tr, prod = _cost(case)
    n = 1 << case["logn"]
    return {"bytes": 8.0 * words, "flops": float(n * (10 * tr * case["logn"] / 2 + 8 * prod))}


def tolerance(case):
    return "exact"                                                   # residues: whole numbers


# ------------------------------------------------------------------ contexts and keys
_CONTEXTS = collections.OrderedDict()


def _primes(case):
    n = 1 << case["logn"]
    Q = [int(q) for q in G.native_primes(1, 60, n)]
    if case["towers"] > 1:
        Q += [int(q) for q in G.native_primes(case["towers"] - 1, case["bits"], n, avoid=Q)]
    return Q, [int(p) for p in G.native_primes(case["special"], 60, n, avoid=Q)]


def _root(n, q):
    """The smallest-base primitive 2n-th root of unity mod q."""
    g = 2
    while pow(c := pow(g, (q - 1) // (2 * n), q), n, q) != q - 1:
        g += 1
    return c


def _key_tensors(case, key_id):
    """A key's two halves [dnum][towers + special][n], seeded residues."""
    Q, P = _primes(case)
    n, dnum = 1 << case["logn"], -(-case["towers"] // case["alpha"])
    g = torch.Generator(device="cuda").manual_seed(20_000 + key_id)
    return [torch.stack([torch.stack([torch.randint(0, q, (n,), dtype=torch.int64, device="cuda", generator=g)
                                      for q in Q + P]) for _ in range(dnum)]) for _ in range(2)]


def _context(case, key_ids):
    at = tuple(case[k] for k in ("logn", "towers", "bits", "alpha", "special"))
    if at not in _CONTEXTS:
        Q, P = _primes(case)
        n = 1 << case["logn"]
        _CONTEXTS[at] = (G.Context(n, Q, P, case["alpha"], roots=[_root(n, q) for q in Q + P]), set())
        while len(_CONTEXTS) > 6:
            _CONTEXTS.popitem(last=False)
    _CONTEXTS.move_to_end(at)
    ctx, have = _CONTEXTS[at]
    for k in sorted(set(key_ids) - have):
        av, bv = _key_tensors(case, k)
        torch.cuda.synchronize()
        G.check(G.lib().gpufhe_ctx_set_key_device(ctx.h, k, av.data_ptr(), bv.data_ptr()))
        torch.cuda.synchronize()
        have.add(k)
    return ctx


def _op_key(case, i):
    """Key id of plan entry i: 0, or the Galois element of a rotation; None without a key."""
    md = _modes(case)[i]
    if md == G.RESCALE:
        return None
    if md in (G.ROTATE, G.ROTATE_HOISTED):
        return _galois(ROT_STEPS[i % len(ROT_STEPS)], 1 << case["logn"])
    return 0


def _residues(gen, moduli, n):
    return torch.stack([torch.randint(0, q, (n,), dtype=torch.int64, device="cuda", generator=gen) for q in moduli])


def _fill(gen, moduli, n, count):
    """[count][towers][n] seeded residues, drawn tower by tower."""
    x = torch.empty((count, len(moduli), n), dtype=torch.int64, device="cuda")
    for t, q in enumerate(moduli):
        x[:, t].copy_(torch.randint(0, q, (count, n), dtype=torch.int64, device="cuda", generator=gen))
    return x


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _pointers(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def _carve(flat, counts, n):
    """Views [towers][n] of a flat buffer, one per count."""
    out, at = [], 0
    for c in counts:
        out.append(flat[at:at + c * n].view(c, n))
        at += c * n
    return out


def _pw_kind(i):
    return (G.PW_MUL_PT, G.PW_ADD, G.PW_MUL_PT, G.PW_SUB, G.PW_ADD_PT, G.PW_MUL_INT)[i % 6]


# ------------------------------------------------------------------ states
def prepare(case, seed):
    n, kind, T, cnt = 1 << case["logn"], case["kind"], case["towers"], case["count"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    Q, _ = _primes(case)
    s = {"kind": kind, "case": dict(case)}
    if kind in ("product", "mixed", "rotate", "hoisted"):
        ctx = _context(case, {_op_key(case, i) for i in range(cnt)} - {None})
        levels, modes = _levels(case), _modes(case)
        nin = {G.EVALMULT_RESCALE: 4, G.KEYSWITCH: 1, G.RESCALE: 1}
        drop = (G.EVALMULT_RESCALE, G.RESCALE)
        s["in"], specs = [], []
        out_towers = []
        for lv, md in zip(levels, modes):
            out_towers += [lv - (md in drop)] * (1 if md == G.RESCALE else 2)
        s["out"] = torch.zeros(sum(out_towers) * n, dtype=torch.int64, device="cuda")
        outs = iter(_carve(s["out"], out_towers, n))
        for i, (lv, md) in enumerate(zip(levels, modes)):
            if md == G.ROTATE_HOISTED and i % 16:
                x = s["in"][-1]
            else:
                x = list(_fill(gen, Q[:lv], n, nin.get(md, 2)))
            s["in"].append(x)
            key = _op_key(case, i)
            specs.append(dict(level=lv, mode=md, key_id=key or 0, galois=key or 0, inp=[t.data_ptr() for t in x],
                              out=[next(outs).data_ptr() for _ in range(1 if md == G.RESCALE else 2)]))
        wsb = sum(ctx.workspace_bytes(sp["level"]) for sp in specs)
        s["ws"] = torch.empty(wsb // 8, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        s["plan"] = G.Plan(ctx, specs, s["ws"].data_ptr(), wsb)
    elif kind == "lintrans":
        n1, n2 = case["n1"], case["n2"]
        gal = {_galois(r, n) for r in list(range(1, n1)) + [g * n1 for g in range(1, n2)]}
        ctx = _context(case, gal)
        s["in"] = _fill(gen, Q, n, 2 + n1 * n2)
        s["out"] = torch.zeros((2, T, n), dtype=torch.int64, device="cuda")
        diag = _pointers(list(s["in"][2:]))
        h = ctypes.c_void_p()
        torch.cuda.synchronize()
        G.check(G.lib().gpufhe_lintrans_plan_create(ctx.h, T, s["in"][0].data_ptr(), s["in"][1].data_ptr(), n1, n2,
                                                    ctypes.cast(diag, ctypes.c_void_p), 0, s["out"][0].data_ptr(),
                                                    s["out"][1].data_ptr(), ctypes.byref(h)))
        s["plan"] = _LinearTransform(ctx, h)
    elif kind == "embed":
        s["ctx"] = _context(case, ())
        s["in"] = torch.randint(-(1 << 40), 1 << 40, (cnt, n), dtype=torch.int64, device="cuda", generator=gen)
        s["out"] = torch.zeros((cnt, T, n), dtype=torch.int64, device="cuda")
        s["outs"] = _pointers(list(s["out"]))
    elif kind == "inverse":
        s["ctx"] = ctx = _context(case, ())
        s["in"] = [_fill(gen, Q, n, cnt) for _ in range(2)]
        s["out"] = torch.zeros((cnt, T, n), dtype=torch.int64, device="cuda")
        s["jobs"] = torch.zeros(cnt * T * int(G.lib().gpufhe_ntt_job_bytes()) // 8 + 2, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()                                     # the job list of the output buffer, kept
        G.check(G.lib().gpufhe_ntt_batch(ctx.h, s["out"].data_ptr(), cnt, T, 0, 1, s["jobs"].data_ptr(), _stream()))
    elif kind == "modraise":
        s["ctx"] = _context(case, ())
        s["in"] = _fill(gen, Q[:1], n, 2 * cnt)
        s["out"] = torch.zeros((2 * cnt, T, n), dtype=torch.int64, device="cuda")
        s["ptrs"] = [_pointers(list(t)) for t in (s["in"][:cnt], s["in"][cnt:], s["out"][:cnt], s["out"][cnt:])]
    elif kind == "pointwise":
        s["ctx"] = _context(case, ())
        levels = _levels(case)
        s["out"] = torch.zeros(2 * sum(levels) * n, dtype=torch.int64, device="cuda")
        outs = iter(_carve(s["out"], [lv for lv in levels for _ in range(2)], n))
        s["in"], s["ops"] = [], []
        for i, lv in enumerate(levels):
            kd, x = _pw_kind(i), _fill(gen, Q[:lv], n, 4)
            s["in"].append(x)
            p = [t.data_ptr() for t in x]
            s["ops"].append(dict(kind=kd, towers=lv, a=(p[0], p[1]), b=(p[2], p[3]), scalar=3 + i % 5,
                                 o=(next(outs).data_ptr(), next(outs).data_ptr())))
    elif kind == "serve":
        reqs = _chain_ops(case)
        ctx = _context(case, {0} | {g for _, ops in reqs for _, g in ops})
        s["in"], s["out"], s["reqs"] = [], [], reqs
        arena = 1 << 20
        for level, ops in reqs:
            last = level - sum(md == G.EVALMULT_RESCALE for md, _ in ops)
            s["in"].append(_fill(gen, Q[:level], n, 2).cpu().pin_memory().numpy().view(np.uint64))
            s["out"].append(torch.zeros((2, last, n), dtype=torch.int64).pin_memory().numpy().view(np.uint64))
            arena += 4 * level * n * 8 + ctx.workspace_bytes(level) + 4096
        s["server"] = G.Server([ctx], ctx.resident_bytes() + arena)
        s["server"].tune(16)
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


class _LinearTransform:
    def __init__(self, ctx, h):
        self.ctx, self.h = ctx, h

    def launch(self, stream):
        G.check(G.lib().gpufhe_lintrans_plan_launch(self.h, stream))

    def __del__(self):
        G.lib().gpufhe_lintrans_plan_destroy(self.h)


def run(s):
    kind, case, lib = s["kind"], s["case"], G.lib()
    if "plan" in s:
        s["plan"].launch(_stream())
    elif kind == "embed":
        G.check(lib.gpufhe_pt_to_eval_batch(s["ctx"].h, case["count"], case["towers"], s["in"].data_ptr(), s["outs"],
                                            _stream()))
    elif kind == "inverse":
        a, b = s["in"]
        G.check(lib.gpufhe_rns_mult_batch(s["ctx"].h, a.data_ptr(), b.data_ptr(), s["out"].data_ptr(), case["count"],
                                          case["towers"], 0, _stream()))
        G.check(lib.gpufhe_ntt_run_jobs(s["ctx"].h, s["jobs"].data_ptr(), case["count"] * case["towers"], 1, _stream()))
    elif kind == "modraise":
        G.check(lib.gpufhe_modraise_batch(s["ctx"].h, case["count"], case["towers"], *s["ptrs"], _stream()))
    elif kind == "pointwise":
        G.pointwise(s["ctx"], s["ops"], _stream())
    else:
        srv = s["server"]
        srv.start()
        for (level, ops), x, y in zip(s["reqs"], s["in"], s["out"]):
            srv.submit(0, level, ops, h_in=x, h_out=y)
        srv.drain(60.0)
        return [y.view(np.int64) for y in s["out"]]
    return s["out"]


# ------------------------------------------------------------------ the definitions, in 64-bit integers
class _Ring:
    """Residue arithmetic of one chain from its definitions: negacyclic
    transforms in bit-reversed order, approximate basis conversion, the Hybrid
    keyswitch, ModDown and rescale."""

    def __init__(self, case):
        self.n, self.logn, self.alpha = 1 << case["logn"], case["logn"], case["alpha"]
        self.Q, self.P = _primes(case)
        self.mods = self.Q + self.P
        brv = torch.zeros(self.n, dtype=torch.int64)
        for b in range(self.logn):
            brv |= ((torch.arange(self.n) >> b) & 1) << (self.logn - 1 - b)
        self.brv = brv.cuda()
        m = self._col(self.mods)
        roots = [_root(self.n, q) for q in self.mods]
        self.tw = self._powers(roots, m)[:, self.brv]
        self.itw = self._powers([pow(r, -1, q) for r, q in zip(roots, self.mods)], m)[:, self.brv]

    @staticmethod
    def _col(v):
        return torch.tensor([int(x) for x in v], dtype=torch.int64, device="cuda")[:, None]

    def _powers(self, roots, m):
        p = torch.ones((len(roots), 1), dtype=torch.int64, device="cuda")
        while p.shape[1] < self.n:
            step = self._col([pow(r, p.shape[1], q) for r, q in zip(roots, self.mods)])
            p = torch.cat([p, self.mul(p, step, m)], 1)
        return p

    @staticmethod
    def _fix(r, q):
        r = torch.where(r < 0, r + q, r)
        return torch.where(r >= q, r - q, r)

    def _small(self, a, b, q):
        """a * b mod q for b below 2^31: the quotient's estimate is off by at most one."""
        k = (a.double() * b.double() / q.double()).long()
        return self._fix(a * b - k * q, q)

    def mul(self, a, b, q):
        hi = self._small(self._small(a, b >> 30, q), torch.full_like(q, 1 << 30), q)
        return self._fix(hi + self._small(a, b & ((1 << 30) - 1), q) - q, q)

    def add(self, a, b, q):
        return self._fix(a + b - q, q)

    def ntt(self, x, rows):
        """x [towers][n] coefficients -> eval form; rows: chain indices of the towers."""
        q, m = self._col([self.mods[r] for r in rows])[:, :, None], 1
        tw = self.tw[rows]
        while m < self.n:
            x = x.view(len(rows), m, 2, -1)
            u, v = x[:, :, 0], self.mul(x[:, :, 1], tw[:, m:2 * m, None], q)
            x = torch.stack([self.add(u, v, q), self._fix(u - v, q)], 2)
            m *= 2
        return x.reshape(len(rows), self.n)

    def intt(self, x, rows):
        q, m = self._col([self.mods[r] for r in rows])[:, :, None], self.n // 2
        tw = self.itw[rows]
        while m:
            x = x.view(len(rows), m, 2, -1)
            u, v = x[:, :, 0], x[:, :, 1]
            x = torch.stack([self.add(u, v, q), self.mul(self._fix(u - v, q), tw[:, m:2 * m, None], q)], 2)
            m //= 2
        return self.mul(x.reshape(len(rows), self.n), self._col([pow(self.n, -1, self.mods[r]) for r in rows]), q[:, 0])

    def rows(self, level):
        return list(range(level)) + [len(self.Q) + j for j in range(len(self.P))]

    def mod(self, x, q):
        return x % q

    def convert(self, x, src, dst):
        """sum_i [x_i * (S/s_i)^-1]_{s_i} * (S/s_i) mod each target: x [src towers][n] coefficients."""
        prod = math.prod(self.mods[r] for r in src)
        hat = [prod // self.mods[r] for r in src]
        y = self.mul(x, self._col([pow(h, -1, self.mods[r]) for h, r in zip(hat, src)]),
                     self._col([self.mods[r] for r in src]))
        q = self._col([self.mods[r] for r in dst])
        acc = torch.zeros((len(dst), self.n), dtype=torch.int64, device="cuda")
        for i, h in enumerate(hat):
            acc = self.add(acc, self.mul(self.mod(y[i][None], q), self._col([h % self.mods[r] for r in dst]), q), q)
        return acc

    def digits(self, a):
        """ModUp of a [level][n] (eval form): every digit over the level's Q towers and P."""
        level = a.shape[0]
        x, rows, out = self.intt(a, list(range(level))), self.rows(level), []
        for st in range(0, level, self.alpha):
            own = list(range(st, min(st + self.alpha, level)))
            d = torch.empty((len(rows), self.n), dtype=torch.int64, device="cuda")
            d[own] = a[own]
            other = [i for i in range(len(rows)) if i not in own]
            d[other] = self.ntt(self.convert(x[own], own, [rows[i] for i in other]), [rows[i] for i in other])
            out.append(d)
        return out

    def inner(self, digits, key):
        """Key inner product and ModDown: the two components over the level's Q towers."""
        level = digits[0].shape[0] - len(self.P)
        rows = self.rows(level)
        q = self._col([self.mods[r] for r in rows])
        p_rows, res = rows[level:], []
        for half in (key[1], key[0]):
            acc = torch.zeros_like(digits[0])
            for d, k in zip(digits, half):
                acc = self.add(acc, self.mul(d, k[rows], q), q)
            conv = self.convert(self.intt(acc[level:], p_rows), p_rows, list(range(level)))
            diff = self._fix(acc[:level] - self.ntt(conv, list(range(level))), q[:level])
            pinv = [pow(math.prod(self.P), -1, m) for m in self.Q[:level]]
            res.append(self.mul(diff, self._col(pinv), q[:level]))
        return res

    def rescale(self, t):
        last = t.shape[0] - 1
        ql, q = self.Q[last], self._col(self.Q[:last])
        r = self.intt(t[last:], [last])
        sw = self.mod(torch.where(r > ql // 2, r - ql, r), q)        # centred, into every tower
        s1 = self._col([pow(ql, -1, m) for m in self.Q[:last]])
        return self.mul(self._fix(t[:last] - self.ntt(sw, list(range(last))), q), s1, q)

    def permute(self, a, k):
        e = 2 * self.brv + 1
        return a[:, self.brv[(e * k % (2 * self.n) - 1) >> 1]]

    def product(self, x, key):
        a0, a1, b0, b1 = x
        q = self._col(self.Q[:a0.shape[0]])
        e0, e1 = self.inner(self.digits(self.mul(a1, b1, q)), key)
        t0 = self.add(self.mul(a0, b0, q), e0, q)
        t1 = self.add(self.add(self.mul(a0, b1, q), self.mul(a1, b0, q), q), e1, q)
        return [self.rescale(t0), self.rescale(t1)]

    def rotate(self, x, key, k):
        e0, e1 = self.inner(self.digits(self.permute(x[1], k)), key)
        return [self.add(self.permute(x[0], k), e0, self._col(self.Q[:x[0].shape[0]])), e1]


def exact(case, seed):
    if _transform_points(case) > 1.2 * _budget()[0]:
        return None                                                  # over twenty seconds
    s, R, kind, keys = prepare(case, seed), _Ring(case), case["kind"], {}

    def key(k):
        if k not in keys:
            keys[k] = _key_tensors(case, k)
        return keys[k]

    T, n, cnt = case["towers"], R.n, case["count"]
    q = R._col(R.Q)
    all_rows = list(range(T))
    if kind in ("product", "mixed", "rotate", "hoisted"):
        out, shared = [], None
        for i, (md, x) in enumerate(zip(_modes(case), s["in"])):
            k = _op_key(case, i)
            if md == G.EVALMULT_RESCALE:
                out += R.product(x, key(k))
            elif md == G.RESCALE:
                out.append(R.rescale(x[0]))
            elif md == G.KEYSWITCH:
                out += R.inner(R.digits(x[0]), key(k))
            elif md == G.ROTATE:
                out += R.rotate(x, key(k), k)
            else:
                if i % 16 == 0:
                    shared = R.digits(x[1])
                e0, e1 = R.inner([R.permute(d, k) for d in shared], key(k))
                out += [R.add(R.permute(x[0], k), e0, R._col(R.Q[:x[0].shape[0]])), e1]
        return torch.cat([o.reshape(-1) for o in out])
    if kind == "lintrans":
        n1, n2 = case["n1"], case["n2"]
        c0, c1, diag = s["in"][0], s["in"][1], s["in"][2:]
        baby = [[c0, c1]] + [R.rotate([c0, c1], key(_galois(r, n)), _galois(r, n)) for r in range(1, n1)]
        total = [torch.zeros_like(c0), torch.zeros_like(c1)]
        for g in range(n2):
            acc = [torch.zeros_like(c0), torch.zeros_like(c1)]
            for b in range(n1):
                acc = [R.add(a, R.mul(x, diag[g * n1 + b], q), q) for a, x in zip(acc, baby[b])]
            if g:
                acc = R.rotate(acc, key(_galois(g * n1, n)), _galois(g * n1, n))
            total = [R.add(t, a, q) for t, a in zip(total, acc)]
        return torch.stack(total)
    if kind == "embed":
        return torch.stack([R.ntt(R.mod(m[None], q), all_rows) for m in s["in"]])
    if kind == "inverse":
        return torch.stack([R.intt(R.mul(a, b, q), all_rows) for a, b in zip(*s["in"])])
    if kind == "modraise":
        out = []
        for x in s["in"]:
            r = R.intt(x, [0])
            out.append(R.ntt(R.mod(torch.where(r > R.Q[0] // 2, r - R.Q[0], r), q), all_rows))
        return torch.stack(out)
    if kind == "pointwise":
        out = []
        for i, (lv, x) in enumerate(zip(_levels(case), s["in"])):
            m, kd = q[:lv], _pw_kind(i)
            if kd == G.PW_ADD:
                r = [R.add(x[0], x[2], m), R.add(x[1], x[3], m)]
            elif kd == G.PW_SUB:
                r = [R._fix(x[0] - x[2], m), R._fix(x[1] - x[3], m)]
            elif kd == G.PW_MUL_PT:
                r = [R.mul(x[0], x[2], m), R.mul(x[1], x[2], m)]
            elif kd == G.PW_ADD_PT:
                r = [R.add(x[0], x[2], m), x[1]]
            else:
                f = torch.full_like(m, 3 + i % 5)
                r = [R.mul(x[0], f, m), R.mul(x[1], f, m)]
            out += r
        return torch.cat([o.reshape(-1) for o in out])
    out = []                                                         # serve
    for (level, ops), h in zip(_chain_ops(case), s["in"]):
        c = list(torch.from_numpy(h.view(np.int64)).cuda())
        for md, k in ops:
            c = R.product([c[0], c[1], c[0], c[1]], key(0)) if md == G.EVALMULT_RESCALE else R.rotate(c, key(k), k)
        out.append(torch.stack(c).cpu().numpy())
    return out
