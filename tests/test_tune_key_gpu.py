"""What one batch's tuning leaves for others: a batch with rescales, or of
rotations alone, keeps its own entry and never sets the schedule of a batch of
products; where it cannot be timed itself it still takes the products' entry.
Captured launches never time, so they show what the cache holds."""
import numpy as np
import pytest

from ckks_setup import Setup
from gpu_util import dev, empty, ptr, sync

pytestmark = pytest.mark.gpu

N, L, GAL = 1024, 4, 5
TUNED = 32                                      # bit of gpufhe_plan_schedule: the plan's own entry was used


def make(G, g, S, products=0, rescales=0, keyswitches=0, rotations=0):
    rng = np.random.default_rng(1)
    keep = [dev(x) for x in S.rand_ct(rng, L) + S.rand_ct(rng, L)]
    specs = []
    for mode, cnt, nin in ((G.EVALMULT_RESCALE, products, 4), (G.RESCALE, rescales, 1), (G.KEYSWITCH, keyswitches, 1),
                           (G.ROTATE, rotations, 2)):
        gal = GAL if mode == G.ROTATE else 0
        for _ in range(cnt):
            o = [empty(L * N) for _ in range(1 if mode == G.RESCALE else 2)]
            keep += o
            specs.append(dict(level=L, mode=mode, key_id=gal, galois=gal, inp=[ptr(t) for t in keep[:nin]],
                              out=[ptr(t) for t in o]))
    return G.Plan(g, specs), keep


def captured(G, g, S, **kw):
    """Schedule word that a plan's first launch takes when it is captured."""
    import torch
    plan, keep = make(G, g, S, **kw)
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        plan.launch(st.cuda_stream)
    sync()
    return int(G.lib().gpufhe_plan_schedule(plan.h))


def launched(G, g, S, **kw):
    """Schedule word after a plain first launch, which times the batch."""
    plan, keep = make(G, g, S, **kw)
    plan.launch()
    sync()
    return int(G.lib().gpufhe_plan_schedule(plan.h))


@pytest.mark.parametrize("first", [dict(keyswitches=1, rescales=14), dict(products=13, rescales=2), dict(rotations=13)])
def test_other_batches_leave_products_alone(first):
    import gpufhe_b200 as G
    S = Setup(N, L, K=2, alpha=2, rot_ks=(GAL,))
    g = S.gpu_context()
    default = captured(G, g, S, products=13)
    assert not default & TUNED
    own = launched(G, g, S, **first)
    assert own & TUNED
    assert captured(G, g, S, **first) == own
    assert captured(G, g, S, products=13) == default
    products = launched(G, g, S, products=13)
    assert products & TUNED
    assert captured(G, g, S, products=13) == products
    assert captured(G, g, S, **first) == own


def test_batches_not_timed_take_the_products_entry():
    import gpufhe_b200 as G
    S = Setup(N, L, K=2, alpha=2, rot_ks=(GAL,))
    g = S.gpu_context()
    products = launched(G, g, S, products=13)
    for kw in (dict(products=12, rescales=3), dict(rotations=13), dict(rotations=9, rescales=1)):
        assert captured(G, g, S, **kw) | TUNED == products
