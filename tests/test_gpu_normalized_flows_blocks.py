"""The block kernel of the normalised flows at the edges of its tiles."""
import numpy as np
import pytest

from lvd_pg_b200 import structures as st
from tests.helpers import random_data, random_hclt, under_one_root, without_root
from tests.test_gpu_normalized_flows import _compare

pytestmark = pytest.mark.gpu


# (variables, latents, rows): one parent more than a chunk and an odd one, two tiles of examples with a ragged and a
# whole end, a block too wide for shared memory, a root with more edges than its threads keep
@pytest.mark.parametrize("v,k,rows", [(6, 17, 131), (5, 33, 128), (5, 65, 36), (4, 144, 132), (3, 336, 12)])
def test_against_oracle(oracle, v, k, rows):
    from lvd_pg_b200 import api
    fc = random_hclt(v, k, 3, v + k)
    data, _ = random_data(rows, v, 3, 4)
    m = api.CuMetaBitsProbCircuit(fc)
    want = oracle.per_sample_normalized_flows(fc, data)
    _compare(api.per_sample_normalized_flows(m, data, batch_size=rows).cpu().numpy(), want)
    _compare(api.per_sample_normalized_flows(m, data, batch_size=rows // 2 + 1).cpu().numpy(), want)


@pytest.mark.parametrize("rows", [90, 132])
def test_impossible_part(oracle, rows):
    """A root over the latent states of two circuits, one of which cannot produce some rows: its blocks have the maximum
    -inf there, no flow reaches them and their edges keep log(1e-8).  The oracle takes -1e4 for -inf
    (0 * exp(-inf + inf) has no value there)."""
    from lvd_pg_b200 import api
    k, parent = 32, np.array([-1, 0, 1, 2, 2], np.int64)
    data, _ = random_data(rows, 5, 3, 4)
    fcs = []
    for zero in (-np.inf, -1e4):
        parts, children = [], []
        for i in (0, 1):
            fc = st.hclt_flat(parent, 3, k, seed=i)
            if i:
                leaf = (fc.node_kind == 0) & (fc.node_var == 4)     # variable 3: no leaf takes category 0
                fc.heap[fc.node_heap_start[leaf].astype(np.int64) - 1] = zero
            parts.append(without_root(fc))
            children += [(i, int(n)) for n in fc.up_prime[fc.up_parent == fc.num_nodes]]
        fcs.append(under_one_root(parts, children))
    m = api.CuMetaBitsProbCircuit(fcs[0])
    assert m.info.num_dense_blocks == 4 and 0 < (data[:, 3] == 0).sum() < rows
    want = oracle.per_sample_normalized_flows(fcs[1], data)
    ni, ok = m.num_inner_params, ~np.isnan(want)
    assert ok[:, :ni].all()
    for batch in (rows, rows // 2 + 1):
        got = api.per_sample_normalized_flows(m, data, batch_size=batch).cpu().numpy()
        assert np.array_equal(np.isnan(got), ~ok)   # leaves without flow: 0 / 0, as in the reference
        _compare(got[:, :ni], want[:, :ni])
        assert np.array_equal(got[:, ni:][ok[:, ni:]], want[:, ni:][ok[:, ni:]])
