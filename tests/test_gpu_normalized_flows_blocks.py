"""The block kernel of the normalised flows at the edges of its tiles."""
import pytest

from tests.helpers import random_data, random_hclt
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
