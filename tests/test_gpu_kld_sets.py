"""KLD of several parameter sets: the layer kernels at the edges of their tiles, and the transposition of the sets."""
import numpy as np
import pytest

from tests.helpers import random_hclt, rel_err
from tests.test_gpu_kld_sample import TOL, _cuda, _param_sets

pytestmark = pytest.mark.gpu

# (variables, latents, categories, sets): sets that do not divide the block, one set more than a tile, a child list
# longer than the staged values (272 x 32 > 2048) with more steps per thread than are parked, single-child chains
SHAPES = [(9, 17, 3, 3), (12, 64, 2, 24), (6, 272, 2, 33), (7, 72, 5, 32), (5, 130, 2, 5), (6, 16, 2, 65)]


@pytest.mark.parametrize("v,k,c,S", SHAPES)
def test_layer_kernels_against_oracle(oracle, v, k, c, S):
    torch, api = _cuda()
    fc = random_hclt(v, k, c, 3 + v)
    p1, p2 = _param_sets(oracle, fc, S, 1), _param_sets(oracle, fc, S, 2)
    m = api.CuMetaBitsProbCircuit(fc)
    out, reuse = api.kld(m, torch.from_numpy(p1).cuda(), torch.from_numpy(p2).cuda())   # row-major on the device
    klds_ref, ek_ref = oracle.kld(fc, p1, p2)
    assert rel_err(out.cpu().numpy(), klds_ref[:, -1]) <= TOL
    assert rel_err(api.kld_matrices(m, reuse)[0], klds_ref) <= TOL
    g1, g2 = api.kld_backward(m, reuse=reuse)
    ref = oracle.kld_backward(fc, p1, p2, klds_ref, ek_ref)
    assert rel_err(g1.cpu().numpy(), ref["param_grads1"], 1e-2) <= TOL
    assert rel_err(g2.cpu().numpy(), ref["param_grads2"]) <= TOL


@pytest.mark.parametrize("S,P", [(2, 2), (3, 129), (31, 128), (33, 1000), (70, 257)])
def test_param_columns(S, P):
    torch, api = _cuda()
    m = api.CuMetaBitsProbCircuit(random_hclt(4, 8, 2, 1))
    x = torch.randn(S, P, device="cuda")
    y = api._columns(m, x)
    assert y.is_contiguous() and torch.equal(y, x.t())
    assert torch.equal(api._columns(m, x[:, ::2]), x[:, ::2].t())    # not row-major: the general path
