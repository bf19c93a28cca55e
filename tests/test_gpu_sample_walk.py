"""Hard samples bit for bit against the oracle for every number of warps per sample, leaves that a lane or a warp decides,
nodes of more edges than a warp holds, one parameter set and one per sample, and parameters without bounds."""
import numpy as np
import pytest

from lvd_pg_b200 import structures as st
from tests.helpers import random_hclt
from tests.test_gpu_kld_sample import _cuda, _param_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v,k,c,S,per_sample", [
    (12, 16, 2, 1, False), (40, 20, 8, 800, False), (30, 17, 9, 1500, False), (9, 70, 70, 2400, False), (5, 150, 3, 300, False),
    (7, 64, 300, 40, False), (12, 33, 4, 50, True)])
@pytest.mark.parametrize("extreme", [False, True])
def test_samples_equal_the_oracle(oracle, v, k, c, S, per_sample, extreme):
    torch, api = _cuda()
    fc = random_hclt(v, k, c, v + k)
    m = api.CuMetaBitsProbCircuit(fc)
    p = _param_sets(oracle, fc, S if per_sample else 1, 1)
    rng = np.random.default_rng(k)
    shp = api.noise_shapes(m, S)
    u_sum, u_leaf = rng.random(shp[0], dtype=np.float32), rng.random(shp[1], dtype=np.float32)
    if extreme:   # certain and impossible edges, tiny and huge weights, noise at both ends and ties
        p.reshape(-1)[::7] = -np.inf
        p.reshape(-1)[::11] = -100.0
        p.reshape(-1)[::13] = 80.0
        for u in (u_sum, u_leaf):
            u.reshape(-1)[::5] = 1 - 2.0 ** -24
            u.reshape(-1)[::6] = 0.0
            u.reshape(-1)[::3] = 0.5
    x = api.sample(m, p if per_sample else p[0], u_sum, u_leaf).cpu().numpy()
    assert np.array_equal(x, oracle.sample_hard(fc, p if per_sample else p[0], u_sum, u_leaf, S))


@pytest.mark.parametrize("v,k,c,S", [(12, 16, 2, 300), (9, 70, 70, 900), (20, 17, 9, 2400)])
@pytest.mark.parametrize("lo,hi,impossible", [(-95.0, -85.0, False), (-89.0, -88.0, True), (-300.0, -80.0, True)])
def test_low_log_weights(oracle, v, k, c, S, lo, hi, impossible):
    """Sets that are not normalised: every log-weight of a node lies where its exponential, or the race time, leaves the
    fp32 range; with and without impossible entries beside them.  Both walks."""
    torch, api = _cuda()
    fc = random_hclt(v, k, c, v + k)
    m = api.CuMetaBitsProbCircuit(fc)
    rng = np.random.default_rng(k)
    p = rng.uniform(lo, hi, fc.num_parameters).astype(np.float32)
    if impossible:
        p[::3] = -np.inf
    shp = api.noise_shapes(m, S)
    u_sum, u_leaf = rng.random(shp[0], dtype=np.float32), rng.random(shp[1], dtype=np.float32)
    for u in (u_sum, u_leaf):   # next to one: the smallest race times
        u.reshape(-1)[::5] = 1 - rng.random(u.reshape(-1)[::5].size).astype(np.float32) * 1e-2
    want = oracle.sample_hard(fc, p, u_sum, u_leaf, S)
    assert np.array_equal(api.sample(m, p, u_sum, u_leaf).cpu().numpy(), want)
    n = min(S, 100)
    x = torch.empty(v, n, dtype=torch.int32, device="cuda").t()
    api.sample_static(m, torch.from_numpy(p).cuda()[:, None], torch.from_numpy(u_sum[:n]).cuda(), torch.from_numpy(u_leaf[:n]).cuda(), x)
    assert np.array_equal(x.cpu().numpy(), want[:n])


@pytest.mark.parametrize("kind,v,k,c,S", [("chain", 60, 16, 3, 40), ("chain", 40, 70, 9, 700), ("star", 50, 20, 2, 300), ("chain", 30, 8, 4, 1300),
                                          ("chain", 3300, 2, 2, 1500), ("random", 4000, 2, 3, 2300)])
def test_deep_wide_and_large_trees(oracle, kind, v, k, c, S):
    """Hundreds of rounds of one node, one round of many, and lists that leave few samples on an SM: every number of
    warps per sample, products of many factors, children of edges past the first 64."""
    torch, api = _cuda()
    rng = np.random.default_rng(v)
    parent = {"chain": np.array([-1] + list(range(v - 1))), "star": np.array([-1, 0] + [1] * (v - 2))}.get(kind)
    if parent is None:
        parent = st.root_tree_at_center(v, st.random_spanning_tree(v, rng))
    fc = st.hclt_flat(parent.astype(np.int64), c, k, seed=v)
    m = api.CuMetaBitsProbCircuit(fc)
    p = oracle.vectorize(fc)
    shp = api.noise_shapes(m, S)
    u_sum, u_leaf = rng.random(shp[0], dtype=np.float32), rng.random(shp[1], dtype=np.float32)
    x = api.sample(m, p, u_sum, u_leaf).cpu().numpy()
    keep = np.arange(0, S, max(1, S // 100))     # the oracle on every so many samples
    assert np.array_equal(x[keep], oracle.sample_hard(fc, p[None], u_sum[keep], u_leaf[keep], len(keep)))
