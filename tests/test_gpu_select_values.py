"""The selects' own square roots and quotients against the oracles on values that networks and long searches can produce --
zeros, values far from one, counts of millions, NaN -- and on every number of edges or actions where the split over the lanes
changes."""
import copy

import numpy as np
import pytest

from mcts_numba_cuda_b200 import duct, puct
from oracle import duct_oracle as do
from oracle import puct_oracle as po
from oracle import puct_v2_oracle as p2

pytestmark = pytest.mark.gpu


def odd_values(n, w, prior, seed):
    """Overwrites a share of the counts, value sums and priors (in place)."""
    rng = np.random.default_rng(seed)

    def some(a, share):
        return rng.random(a.shape) < share

    n[some(n, 0.2)] = 0
    big = some(n, 0.05)
    n[big] = rng.integers(1 << 21, 1 << 25, size=int(big.sum()))
    w[n == 0] = 0
    w[some(w, 0.05)] = 0
    tiny = some(w, 0.05)
    w[tiny] *= np.float32(1e-30)
    prior[some(prior, 0.05)] = 0
    small = some(prior, 0.05)
    prior[small] *= np.float32(1e-38)     # below the normal range
    w[some(w, 0.01)] = np.nan


@pytest.mark.parametrize("edges", [1, 2, 31, 32, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("c_pw", [0.0, 0.02])
def test_puct_selects_match_the_oracles_on_odd_values(edges, c_pw):
    import torch
    case = po.layered_case(12, edges, 3, 1, seed=edges, nodes_per_level=min(edges, 16))
    odd_values(case["edge_n"], case["edge_w"], case["edge_prior"], seed=edges)
    kw = dict(cpuct=1.5, c_pw=c_pw)
    with np.errstate(all="ignore"):
        want = po.select(copy.deepcopy(case), **kw)
    d = puct.to_device(case)
    puct.launch_select(d, **kw)
    torch.cuda.synchronize()
    got = puct.to_host(d)
    for k in ("out_selected", "out_len", "edge_inflight", "node_expand_inflight"):
        assert np.array_equal(got[k], want[k]), k
    for variant in (puct.V2_PRECLAIM, puct.V2_COUNTER_CAS):
        case2 = p2.from_v3_case(copy.deepcopy(case))
        with np.errstate(all="ignore"):
            want = p2.select(copy.deepcopy(case2), variant=variant, **kw)
        d = puct.to_device(case2)
        puct.launch_select_v2(d, variant=variant, **kw)
        torch.cuda.synchronize()
        got = puct.to_host(d)
        for k in ("out_selected", "out_len", "node_inflight", "node_expand_inflight"):
            assert np.array_equal(got[k], want[k]), (variant, k)


@pytest.mark.parametrize("actions", [2, 3, 4, 5, 8, 9, 16])
def test_duct_select_matches_the_oracle_on_odd_values(actions):
    import torch
    case = do.make_case(15, actions=actions, depth=4, seed=actions)
    odd_values(case["node_n"], case["node_w"], case["node_prior"], seed=actions)
    case["node_w"][np.isnan(case["node_w"])] = 1e-20      # a NaN has no place in the order the specification gives
    want = do.copy_case(case)
    with np.errstate(all="ignore"):
        do.select(want, cpuct=1.5, virtual_loss=2)
    d = puct.to_device(case)
    duct.launch_select(d, cpuct=1.5, virtual_loss=2)
    torch.cuda.synchronize()
    got = puct.to_host(d)
    for k in ("out_selected", "out_len", "node_inflight", "child"):
        assert np.array_equal(got[k], want[k]), k
