"""Batches whose operations write over an input of the batch: one run of such a
batch is right (inputs are last read by the key product, outputs written by the
last phase), a second one would read what the first wrote. So the first launch
must not time it, and equals the oracle."""
import numpy as np
import pytest

from ckks_setup import Setup
from gpu_util import dev, empty, host, ptr, sync

pytestmark = pytest.mark.gpu

N, L = 1024, 4


@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("which", ["keyswitch", "product", "second output", "another input", "part of an input"])
def test_first_launch_of_an_aliased_batch(which, rescale):
    import gpufhe_b200 as G
    S = Setup(N, L, K=2, alpha=2)
    g = S.gpu_context()
    rng = np.random.default_rng(5)
    c = S.rand_ct(rng, L) + S.rand_ct(rng, L)
    k = S.rand_ct(rng, L)[0]
    d = [dev(x) for x in c]
    kb = empty((L + 1) * N)                     # the keyswitch input, with one tower of room behind it
    kb[:L * N] = dev(k)
    o = [empty(L * N) for _ in range(4)]
    pr, ks = [ptr(o[0]), ptr(o[1])], [ptr(o[2]), ptr(o[3])]
    if which == "keyswitch":
        ks[0] = ptr(kb)
    elif which == "product":
        pr = [ptr(d[0]), ptr(d[1])]
    elif which == "second output":
        ks[1] = ptr(kb)
    elif which == "another input":
        pr[0] = ptr(kb)
    else:
        ks[1] = ptr(kb) + 8 * N                 # starts at the input's second tower
    specs = [dict(level=L, inp=[ptr(t) for t in d], out=pr),
             dict(level=L, mode=G.KEYSWITCH, inp=[ptr(kb)], out=ks)]
    x, y = dev(c[2]), empty((L - 1) * N)
    if rescale:
        specs.append(dict(level=L, mode=G.RESCALE, inp=[ptr(x)], out=[ptr(y)]))
    at = {ptr(t): t for t in [*o, *d]}
    at.update({ptr(kb): kb[:L * N], ptr(kb) + 8 * N: kb[N:]})
    plan = G.Plan(g, specs)
    plan.launch()
    sync()
    for p, e in zip(pr + ks, (*S.octx.evalmult_rescale(L, *c), *S.octx.keyswitch(L, k))):
        assert np.array_equal(host(at[p])[:e.size], e)
    if rescale:
        assert np.array_equal(host(y), S.octx.rescale(L, c[2]))
    assert not plan.schedule()["tuned"]
