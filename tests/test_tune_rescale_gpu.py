"""The autotuner on batches with rescales: out of place it measures (and the
inputs stay as they were, the outputs equal the oracle's), in place or onto
another operation's input it keeps the default schedule, since a second run
would read what the first one wrote."""
import numpy as np
import pytest

import oracle as O
from ckks_setup import Setup
from gpu_util import dev, empty, host, ptr, sync

pytestmark = pytest.mark.gpu

N, L = 1024, 4


@pytest.mark.parametrize("where", ["apart", "in place", "onto another input"])
def test_tuning_with_rescale(where):
    import gpufhe_b200 as G
    S = Setup(N, L, K=2, alpha=2)
    g = S.gpu_context()
    rng = np.random.default_rng(3)
    c = S.rand_ct(rng, L) + S.rand_ct(rng, L)
    d = [dev(x) for x in c]
    o0, o1, r = empty((L - 1) * N), empty((L - 1) * N), empty(L * N)
    x = dev(c[0])
    out = {"apart": r, "in place": x, "onto another input": d[3]}[where]
    specs = [dict(level=L, mode=G.RESCALE, inp=[ptr(x)], out=[ptr(out)])]
    if where != "onto another input":
        specs.append(dict(level=L, inp=[ptr(t) for t in d], out=[ptr(o0), ptr(o1)]))
    else:
        k0, k1 = empty(L * N), empty(L * N)
        specs.append(dict(level=L, mode=G.KEYSWITCH, inp=[ptr(d[3])], out=[ptr(k0), ptr(k1)]))
    plan = G.Plan(g, specs)
    plan.launch()
    sync()
    assert plan.schedule()["tuned"] == (where == "apart")
    assert np.array_equal(host(out)[:(L - 1) * N], S.octx.rescale(L, c[0]))
    if where == "onto another input":
        return
    e0, e1 = S.octx.evalmult_rescale(L, *c)
    assert np.array_equal(host(o0), e0) and np.array_equal(host(o1), e1)
    if where == "apart":
        assert np.array_equal(host(x), c[0])
