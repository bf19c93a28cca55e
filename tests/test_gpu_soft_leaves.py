"""Leaves under soft evidence, one variable at a time: category counts at the edges of the register tiles and past the
largest the kernels take, batches that end inside a tile, more leaves than a group, and the values whose sum leaves the
range of the fast form."""
import numpy as np
import pytest

from tests.helpers import random_hclt, rel_err
from tests.test_gpu_em import TOL, _cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,c,rows,weighted,spread", [
    (5, 2, 1, False, 1.0), (17, 8, 33, True, 1.0), (70, 9, 64, False, 1.0), (16, 40, 45, True, 1.0), (33, 41, 31, False, 1.0),
    (16, 64, 100, True, 1.0), (16, 65, 40, False, 1.0), (17, 12, 70, True, 60.0), (17, 33, 70, False, 60.0)])
def test_against_oracle(oracle, k, c, rows, weighted, spread):
    """`spread` 60: the likely categories of a leaf often have weights e^-100 below the example's best one, where the
    sum underflows and the exact form takes over for that leaf and example."""
    torch, api = _cuda()
    rng = np.random.default_rng(k + c)
    fc = random_hclt(6, k, c, 3)
    if spread > 1.0:   # leaves that know one category
        heap = fc.heap.copy()
        for n in fc.input_node_ids.astype(np.int64) - 1:
            s = int(fc.node_heap_start[n]) - 1
            heap[s:s + c] = -200.0
            heap[s + rng.integers(c)] = 0.0
        fc.heap = heap
    soft = (rng.normal(0, spread, (rows, 6, c))).astype(np.float32)
    w = rng.random(rows).astype(np.float32) if weighted else None
    ref, m = fc.copy(), api.CuMetaBitsProbCircuit(fc)
    dsoft, wd = api.colmajor(soft, m.device), None if w is None else torch.from_numpy(w).cuda()
    mars_ref = oracle.forward_ex(ref, soft=soft)
    ws, B = api.forward_ex(m, soft=dsoft)
    assert np.abs(m.mars(ws, B) - mars_ref).max() <= TOL * max(1.0, np.abs(mars_ref).max())
    flows_ref, _ = oracle.backward(ref, mars_ref)
    oracle.input_flows_ex(ref, flows_ref, soft=soft, weights=w)
    m.lib.pcb_clear_flows(m.handle, 0.0, None)
    api.backward(m, ws, wd)
    heap = m.heap()
    flow = np.concatenate([np.arange(h - 1 + c, h + 2 * c) for h in fc.node_heap_start[fc.input_node_ids.astype(np.int64) - 1].astype(np.int64)])
    # flows of extreme evidence are exponentials of float32 differences of a few hundred (spacing 3e-5, a few of them)
    assert rel_err(heap[flow], ref.heap[flow], 1e-4) <= (TOL if spread == 1.0 else 5 * TOL)
