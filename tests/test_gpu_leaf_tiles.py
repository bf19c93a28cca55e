"""Leaf statistics with one leaf per lane: categories from two to the largest the kernel takes, slices of one example,
a full one and one more, leaves that do not fill a block, missing values, weights and values no leaf has."""
import numpy as np
import pytest

from tests.helpers import random_data, random_hclt, rel_err
from tests.test_gpu_em import TOL, _cuda

pytestmark = pytest.mark.gpu


# the sums of B flows in another order: TOL is a thousand times their rounding
@pytest.mark.parametrize("k,c,rows,missing,weighted", [
    (17, 2, 1, 0.0, False), (40, 2, 256, 0.2, True), (33, 3, 257, 0.0, True), (70, 10, 31, 0.3, False),
    (17, 100, 1100, 0.1, False), (40, 256, 520, 0.0, True), (5, 500, 64, 0.1, False), (40, 256, 1100, 0.1, False)])
def test_against_oracle(oracle, k, c, rows, missing, weighted):
    torch, api = _cuda()
    fc = random_hclt(5, k, c, 3)
    data, miss = random_data(rows, 5, min(c, 256), 11, missing)
    w = np.random.default_rng(1).random(rows).astype(np.float32) if weighted else None
    ref, m = fc.copy(), api.CuMetaBitsProbCircuit(fc)
    flows_ref, _ = oracle.backward(ref, oracle.forward(ref, data, miss=miss))
    oracle.input_flows(ref, flows_ref, data, miss=miss, weights=w)
    dd, wd = api.DeviceData(data, m.device, miss), None if w is None else torch.from_numpy(w).cuda()
    for _ in range(2):   # the second pass adds to what the first left
        ws, B = api.forward(m, dd)
        api.backward(m, ws, wd)
    heap = m.heap()
    flow = np.concatenate([np.arange(h - 1 + c, h + 2 * c) for h in fc.node_heap_start[fc.input_node_ids.astype(np.int64) - 1].astype(np.int64)])
    assert rel_err(heap[flow], 2.0 * ref.heap[flow]) <= TOL


@pytest.mark.parametrize("k,c,rows", [(5, 2, 20000), (16, 3, 37000), (33, 100, 30111)])
def test_few_leaves_and_many_examples(oracle, k, c, rows):
    """The slices of a batch dealt out over blocks: as many as blocks, one more, several per block."""
    test_against_oracle(oracle, k, c, rows, 0.1, True)


@pytest.mark.parametrize("impl", ["", "sorted", "atomic"])
def test_values_that_no_leaf_has(monkeypatch, impl):
    """A value one past the extra slot is no missing value: it is dropped, as every larger one."""
    monkeypatch.setenv("PCB_LEAF_FLOW_IMPL", impl)
    torch, api = _cuda()
    fc = random_hclt(5, 17, 3, 3)
    data, _ = random_data(300, 5, 3, 11)
    var = int(fc.node_var[fc.input_node_ids[0] - 1]) - 1     # its leaves are not the last: their tables are followed by others
    data[::7, var] = 4
    m = api.CuMetaBitsProbCircuit(fc)
    ws, B = api.forward(m, api.DeviceData(data, m.device))
    m.lib.pcb_clear_flows(m.handle, 0.0, None)
    api.backward(m, ws)
    flows, heap = m.flows(ws, B), m.heap()
    for n in np.nonzero((fc.node_kind == 0) & (fc.node_var == var + 1))[0]:
        h = int(fc.node_heap_start[n]) - 1 + 3
        want = [flows[data[:, var] == x, n].sum() for x in range(3)] + [0.0]
        np.testing.assert_allclose(heap[h:h + 4], want, rtol=1e-4, atol=1e-6)
