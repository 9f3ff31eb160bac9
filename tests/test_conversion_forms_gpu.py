"""The pipeline's conversions at the edges of their forms: special primes and
digit widths on both sides of the bound that allows the FP64-quotient form
(conv_wrap_ok in csrc/conv_quot.hpp), tower widths from 30 to 60 bits, inputs at
0 and q - 1. Products, rotations, keyswitches and rescales equal the oracle
bit for bit in separate and in interleaved launches."""
import numpy as np
import pytest

import oracle as O
from gpu_util import dev, empty, host, ptr, sync

pytestmark = pytest.mark.gpu


def residues(rng, mods, n, edge):
    x = np.concatenate([rng.integers(0, int(q), n, dtype=np.uint64) for q in mods])
    if edge:   # runs of the smallest and largest residues
        for t, q in enumerate(mods):
            x[t * n:t * n + n // 4] = 0
            x[t * n + n // 4:t * n + n // 2] = int(q) - 1
    return x


@pytest.mark.parametrize("n,bits,K,alpha,pbits", [
    (1024, (60, 50, 50, 50, 50), 1, 1, 60),
    (2048, (60, 50, 50, 50, 50, 50, 50), 3, 3, 60),
    (1024, (60,) + (50,) * 9, 8, 8, 60),             # nine terms
    (1024, (60,) + (50,) * 5, 9, 5, 60),             # ten terms: the widest that fits at 60 bits
    (1024, (60,) + (50,) * 5, 10, 5, 60),            # eleven: the 128-bit form
    (1024, (60,) + (50,) * 5, 13, 6, 60),
    (1024, (60,) + (50,) * 5, 12, 6, 50),            # 50-bit special primes
    (1024, (50, 50, 50, 50), 2, 2, 60),
    (1024, (60, 30, 40, 30, 45, 49), 2, 3, 60),      # narrow towers
    (1024, (60, 55, 55, 50, 55), 2, 2, 60),
    (4096, (50, 60, 50, 60, 50), 4, 4, 55),
    (1024, (61,) + (50,) * 5, 6, 5, 61),             # seven terms: the widest that fits at 61 bits
    (1024, (61,) + (50,) * 5, 7, 5, 61),             # eight: the 128-bit form
    (1024, (61, 61, 50, 61), 2, 2, 61),              # the widest towers: 8q just below 2^64
])
def test_conversion_forms(n, bits, K, alpha, pbits):
    import gpufhe_b200 as G
    Q = []
    for b in bits:
        Q.append(int(O.native_primes(1, b, n, avoid=Q)[0]))
    P = [int(p) for p in O.native_primes(K, pbits, n, avoid=Q)]
    Q, P = np.array(Q, np.uint64), np.array(P, np.uint64)
    octx = O.Ctx(n, Q, P, alpha)
    g = G.Context(n, Q, P, alpha)
    rng = np.random.default_rng(len(bits) * 100 + K)
    QP, gal = np.concatenate([Q, P]), 5
    dnum = -(-len(Q) // alpha)
    for key in (0, gal):
        av, bv = (np.concatenate([residues(rng, QP, n, False) for _ in range(dnum)]) for _ in range(2))
        octx.set_key(key, av, bv)
        g.set_key(key, av, bv)
    keep, specs, want = [], [], []
    for j, L in enumerate((2, len(Q) - 1, len(Q), len(Q))):
        c = [residues(rng, Q[:L], n, j == 3) for _ in range(4)]
        d = [dev(x) for x in c]
        keep += d
        for mode, key, nin, tow, exp in (
                (G.EVALMULT_RESCALE, 0, 4, L - 1, lambda: octx.evalmult_rescale(L, *c)),
                (G.ROTATE, gal, 2, L, lambda: octx.rotate(L, gal, c[0], c[1], gal)),
                (G.KEYSWITCH, 0, 1, L, lambda: octx.keyswitch(L, c[0])),
                (G.RESCALE, 0, 1, L - 1, lambda: (octx.rescale(L, c[2]),))):
            e = exp()
            outs = [empty(tow * n) for _ in e]
            keep += outs
            specs.append(dict(level=L, mode=mode, key_id=key, galois=key, inp=[ptr(x) for x in (d[2:] if mode == G.RESCALE else d)[:nin]],
                              out=[ptr(x) for x in outs]))
            want.append((outs, e))
    for schedule in (0, 64 | 0x1ff << 8):
        plan = G.Plan(g, specs)
        plan.set_schedule(schedule)
        for outs, _ in want:
            for o in outs:
                o.fill_(-1)
        plan.launch()
        sync()
        for j, (outs, e) in enumerate(want):
            for o, x in zip(outs, e):
                assert np.array_equal(host(o), np.asarray(x)[:host(o).size]), (schedule, j)
