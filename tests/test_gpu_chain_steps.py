"""The kernels that take a whole step of a pass (blocks, the products under them, single nodes) against the oracle, and
the tensor-core path over the same steps (PCB_CHAIN=0), at the edges of tiles, batches and the choice between the two."""
import numpy as np
import pytest

from lvd_pg_b200 import structures as st
from tests.helpers import random_data, rel_err
from tests.test_gpu_em import TOL, _cuda

pytestmark = pytest.mark.gpu


def _tree(kind, v):
    if kind == "star":      # one product over many blocks: more sources than are fetched together
        return np.array([-1] + [0] * (v // 2) + list(range(1, v - v // 2)), np.int64)
    if kind == "chain":     # no products at all
        return np.array([-1] + list(range(v - 1)), np.int64)
    rng = np.random.default_rng(v)
    return st.root_tree_at_center(v, st.random_spanning_tree(v, rng))


def _check(oracle, fc, data, miss=None, tol=TOL):
    torch, api = _cuda()
    ref, m = fc.copy(), api.CuMetaBitsProbCircuit(fc)
    mars_ref = oracle.forward(ref, data, miss=miss)
    ws, B = api.forward(m, api.DeviceData(data, m.device, miss))
    assert np.abs(m.mars(ws, B) - mars_ref).max() <= tol * max(1.0, np.abs(mars_ref).max())
    flows_ref, aggr_ref = oracle.backward(ref, mars_ref)
    m.lib.pcb_clear_flows(m.handle, 0.0, None)
    api.backward(m, ws)
    assert rel_err(m.flows(ws, B), flows_ref) <= tol
    sums = ref.edge_is_sum[ref.down2up.astype(np.int64) - 1]
    assert rel_err(m.edge_aggr()[sums], aggr_ref[sums]) <= tol
    return m


# (tree, variables, latents, rows): one, two and several batches of rows per thread, latents that are no multiple of
# eight or four, one row more than a tile, two row chunks, more rows than one wave of CTAs keeps, one example
@pytest.mark.parametrize("macs", ["0", "1000000000000"], ids=["rule", "always"])
@pytest.mark.parametrize("kind,v,k,rows", [
    ("random", 12, 16, 1), ("random", 14, 17, 33), ("star", 17, 33, 70), ("chain", 6, 65, 64), ("random", 9, 72, 300),
    ("star", 11, 130, 31), ("random", 6, 272, 40), ("random", 24, 32, 1300), ("star", 60, 16, 40)])
def test_steps_against_oracle(oracle, monkeypatch, kind, v, k, rows, macs):
    monkeypatch.setenv("PCB_CHAIN_MACS", macs)
    _check(oracle, st.hclt_flat(_tree(kind, v), 3, k, seed=v + k), random_data(rows, v, 3, 5)[0])


@pytest.mark.parametrize("kind,v,k,rows", [("random", 14, 17, 33), ("star", 17, 64, 130), ("chain", 6, 128, 260), ("random", 6, 272, 70)])
def test_tensor_core_steps_against_oracle(oracle, monkeypatch, kind, v, k, rows):
    monkeypatch.setenv("PCB_CHAIN", "0")
    data, miss = random_data(rows, v, 3, 5, 0.1)
    _check(oracle, st.hclt_flat(_tree(kind, v), 3, k, seed=v + k), data, miss)


def test_impossible_children(oracle):
    """Leaves with zero probability for the observed category: blocks whose maximum is -inf for some examples, which
    get the value -inf and leave the other examples of their tile alone."""
    torch, api = _cuda()
    fc = st.hclt_flat(_tree("random", 10), 3, 32, seed=3)
    heap = fc.heap.copy()
    for n in fc.input_node_ids[:64].astype(np.int64) - 1:       # two variables never take category 0
        heap[fc.node_heap_start[n] - 1] = -np.inf
    fc.heap = heap
    data, _ = random_data(97, 10, 3, 9)
    ref, m = fc.copy(), api.CuMetaBitsProbCircuit(fc)
    mars_ref = oracle.forward(ref, data)
    ws, B = api.forward(m, api.DeviceData(data, m.device))
    mars = m.mars(ws, B)
    assert np.array_equal(np.isneginf(mars), np.isneginf(mars_ref)) and not np.isnan(mars).any()
    ok = np.isfinite(mars_ref)
    assert np.abs(mars[ok] - mars_ref[ok]).max() <= TOL * np.abs(mars_ref[ok]).max()
    possible = np.isfinite(mars_ref[:, -1])
    assert 0 < possible.sum() < len(possible)
    api.backward(m, ws)
    flows_ref, _ = oracle.backward(ref, mars_ref)
    assert rel_err(m.flows(ws, B)[possible], flows_ref[possible]) <= TOL


@pytest.mark.parametrize("impl", [{}, {"PCB_CHAIN": "0"}, {"PCB_TC_IMPL": "km"}, {"PCB_DENSE_IMPL": "simt"}],
                         ids=["rule", "tensor", "km", "simt"])
@pytest.mark.parametrize("k,rows", [(32, 97), (72, 40)])
def test_dead_state(oracle, monkeypatch, impl, k, rows):
    """A latent state that cannot have produced some rows, and one that is e^100 less likely than its neighbours, in
    blocks that are possible otherwise: their value lies far below the block's maximum, their flow is 0, and neither the
    flows of the children nor the statistics see them.  The oracle takes -1e4 for -inf (0 * exp(-inf + inf) has no value)."""
    for key, val in impl.items():
        monkeypatch.setenv(key, val)
    torch, api = _cuda()
    fcs = []
    for zero in (-np.inf, -1e4):
        fc = st.hclt_flat(_tree("random", 9), 3, k, seed=5)
        start = fc.node_heap_start.astype(np.int64) - 1
        sums = np.nonzero(np.bincount(fc.up_parent[fc.edge_is_sum].astype(np.int64), minlength=fc.num_nodes + 1) == k)[0]
        blocks = sums[sums != fc.num_nodes].reshape(-1, k)      # consecutive states of one variable
        assert np.all(np.diff(blocks, axis=1) == 1)
        for rows_of in blocks:
            for state, value in ((3, zero), (7, -100.0)):       # all weight on one child, whose leaf never takes category 0
                e = np.nonzero(fc.up_parent == rows_of[state])[0]
                fc.up_logp[e] = zero
                fc.up_logp[e[5 + state]] = 0.0
                fc.heap[start[int(fc.up_sub[e[5 + state]]) - 1]] = value
        fcs.append(fc)
    data, _ = random_data(rows, 9, 3, 9)
    ref, m = fcs[1], api.CuMetaBitsProbCircuit(fcs[0])
    mars_ref = oracle.forward(ref, data)
    flows_ref, aggr_ref = oracle.backward(ref, mars_ref)
    ws, B = api.forward(m, api.DeviceData(data, m.device))
    m.lib.pcb_clear_flows(m.handle, 0.0, None)
    api.backward(m, ws)
    dead = mars_ref < mars_ref.max(1, keepdims=True) - 5000.0
    assert dead.any() and np.isfinite(mars_ref[:, -1]).all() and not dead[:, -1].any()
    assert rel_err(m.mars(ws, B)[:, -1], mars_ref[:, -1]) <= TOL
    assert rel_err(m.flows(ws, B), flows_ref) <= TOL
    sum_edges = ref.edge_is_sum[ref.down2up.astype(np.int64) - 1]
    assert rel_err(m.edge_aggr()[sum_edges], aggr_ref[sum_edges]) <= TOL


@pytest.mark.parametrize("weight", [-np.inf, -200.0, -110.0])
def test_root_of_unlikely_states(oracle, weight):
    """The root's most likely child has (almost) no weight: the others, e^150 below it, make up the likelihood."""
    torch, api = _cuda()
    k = 32
    fc = st.hclt_flat(_tree("random", 8), 3, k, seed=5)
    start = fc.node_heap_start.astype(np.int64) - 1
    e = np.nonzero(fc.up_parent == fc.num_nodes)[0]
    leaves = start[fc.up_sub[e].astype(np.int64) - 1]
    fc.heap[leaves[1:]] = -150.0          # category 0 of the root's variable is next to impossible but in state 0
    fc.up_logp[e[0]] = weight
    data, _ = random_data(70, 8, 3, 9)
    m = api.CuMetaBitsProbCircuit(fc)
    mars_ref = oracle.forward(fc, data)
    ws, B = api.forward(m, api.DeviceData(data, m.device))
    assert rel_err(m.mars(ws, B)[:, -1], mars_ref[:, -1]) <= TOL
    flows_ref, _ = oracle.backward(fc, mars_ref)
    api.backward(m, ws)
    assert rel_err(m.flows(ws, B), flows_ref) <= TOL
