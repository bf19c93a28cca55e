"""KLD of several parameter sets: the layer kernels at the edges of their tiles, and the transposition of the sets."""
import numpy as np
import pytest

from tests.helpers import random_hclt, rel_err
from tests.test_gpu_kld_sample import TOL, _cuda, _param_sets

pytestmark = pytest.mark.gpu

# (variables, latents, categories, sets): sets that do not divide the block, one set more than a tile, a child list
# longer than the staged values (272 x 32 > 2048) with more steps per thread than are parked, single-child chains, few
# sets on either side of the line between warps and tiles, no dense blocks
SHAPES = [(9, 17, 3, 3), (20, 130, 2, 3), (60, 40, 2, 8), (20, 130, 2, 5), (40, 70, 2, 4), (30, 64, 2, 8), (9, 8, 3, 8), (9, 8, 3, 9), (12, 64, 2, 24), (6, 272, 2, 33), (7, 72, 5, 32), (5, 130, 2, 5), (6, 16, 2, 65)]


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


@pytest.mark.parametrize("S,P", [(2, 2), (3, 129), (31, 128), (33, 1000), (70, 257), (13, 310001)])
def test_param_columns(S, P):
    torch, api = _cuda()
    m = api.CuMetaBitsProbCircuit(random_hclt(4, 8, 2, 1))
    x = torch.randn(S, P, device="cuda")
    y = api._columns(m, x)
    assert y.is_contiguous() and torch.equal(y, x.t())
    assert torch.equal(api._param_columns(m, x), x.t())
    assert torch.equal(api._columns(m, x[:, ::2]), x[:, ::2].t())    # not row-major: the general path


def test_adam_steps_around_more_sets(oracle):
    """A KLD of several sets grows the buffers that the captured single-set step was recorded with."""
    torch, api = _cuda()
    fc = random_hclt(8, 17, 3, 4)
    sets = _param_sets(oracle, fc, 40, 1)
    p, q0 = torch.from_numpy(sets[0]).cuda(), torch.from_numpy(sets[1])
    got = []
    for others in (False, True):
        m = api.CuMetaBitsProbCircuit(fc)
        opt = api.KldAdam(m, q0.cuda().clone(), p)
        klds = []
        for step in range(9):
            if others and step in (4, 7):
                S = 12 if step == 4 else 40
                api.kld(m, torch.from_numpy(sets[:S]).cuda(), torch.from_numpy(sets[:S][::-1].copy()).cuda())
            klds.append(opt.step().item())
        got.append((klds, opt.q.cpu().numpy()))
    # the sums of the node gradients are atomics: their order differs from run to run
    np.testing.assert_allclose(got[1][0], got[0][0], rtol=1e-5)
    np.testing.assert_allclose(got[1][1], got[0][1], rtol=1e-4, atol=1e-4)
