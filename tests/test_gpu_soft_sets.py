"""Relaxed sampling at the edges of its tiles, and its table logarithm / exponential next to their range's ends."""
import numpy as np
import pytest

from tests.helpers import random_hclt, rel_err
from tests.test_gpu_kld_sample import TOL, _cuda, _param_sets

pytestmark = pytest.mark.gpu

# sets that do not divide the block, more sets than a tile, nodes with more than eight edges per thread (272 edges over
# eight groups), more rows per thread than are parked (272 rows over four groups)
SHAPES = [(9, 17, 3, 3), (12, 64, 2, 24), (6, 272, 2, 33), (5, 130, 2, 1)]


@pytest.mark.parametrize("noise", [True, False])
@pytest.mark.parametrize("v,k,c,S", SHAPES)
def test_relaxed_samples_against_oracle(oracle, v, k, c, S, noise):
    torch, api = _cuda()
    fc = random_hclt(v, k, c, 3 + v)
    m = api.CuMetaBitsProbCircuit(fc)
    p = _param_sets(oracle, fc, S, 1)
    u = np.random.default_rng(2).random((S, m.num_inner_params), dtype=np.float32) if noise else None
    out = api.gumbel_sample(m, torch.from_numpy(p).cuda(), v, c, 0.7, no_gumbel=not noise,
                            u=torch.from_numpy(u).cuda() if noise else None)
    assert rel_err(out.cpu().numpy(), oracle.sample_soft(fc, p, u, 0.7, S, c)[0]) <= TOL


@pytest.mark.parametrize("temperature", [0.25, 0.7, 20.0])
def test_relaxed_samples_extreme_noise(oracle, temperature):
    """Uniforms of 0, next to 0 and next to 1, parameters of -inf: the ends of the tables' ranges and the values
    beyond them, which the CUDA functions take.  fp32 rounds the weights once on either side: TOL covers it."""
    torch, api = _cuda()
    fc = random_hclt(5, 16, 2, 1)
    m = api.CuMetaBitsProbCircuit(fc)
    S = 6
    p = _param_sets(oracle, fc, S, 1)
    u = np.random.default_rng(2).random((S, m.num_inner_params), dtype=np.float32)
    ends = np.array([0.0, 1e-38, 1e-7, 0.3678, 0.36788, 0.5, 1 - 2.0 ** -24, 1 - 2.0 ** -10], np.float32)
    u[:, ::3] = ends[np.arange(u[:, ::3].size) % ends.size].reshape(u[:, ::3].shape)
    p[:, 1:m.num_inner_params:5] = -np.inf
    out = api.gumbel_sample(m, p, 5, 2, temperature, u=u).cpu().numpy()
    ref = oracle.sample_soft(fc, p, u, temperature, S, 2)[0]
    assert np.isfinite(ref).all() and rel_err(out, ref) <= TOL


@pytest.mark.parametrize("v,k,c,S", [(7, 31, 5, 2), (5, 65, 2, 33), (4, 256, 2, 40)])
def test_relaxed_samples_of_row_major_sets(oracle, v, k, c, S):
    """Row-major device matrices are read as they are (a remainder of lanes, of warps and of a tile of sets; the widest
    node the tile takes); the same values from the host, and uniforms with unused columns, go through the columns."""
    torch, api = _cuda()
    fc = random_hclt(v, k, c, 3 + v)
    m = api.CuMetaBitsProbCircuit(fc)
    p = _param_sets(oracle, fc, S, 1)
    u = np.random.default_rng(2).random((S, m.num_inner_params), dtype=np.float32)
    u[:, ::7], u[:, 1::7] = 0.0, 1 - 2.0 ** -24
    ref = oracle.sample_soft(fc, p, u, 0.7, S, c)[0]
    wide = torch.from_numpy(np.concatenate([u, u[:, :3]], 1)).cuda()
    for pp, uu in ((torch.from_numpy(p).cuda(), torch.from_numpy(u).cuda()), (p, u), (torch.from_numpy(p).cuda(), wide)):
        assert rel_err(api.gumbel_sample(m, pp, v, c, 0.7, u=uu).cpu().numpy(), ref) <= TOL


@pytest.mark.parametrize("temperature", [0.7, 1.0 / 300, 1e-6])
@pytest.mark.parametrize("rows", [True, False])
def test_relaxed_weights_at_low_temperatures(temperature, rows):
    """Edges whose log-weight and noise nearly cancel, so that the temperature divides small sums: against 64 bits.  The
    inputs are exact, the weights and their sums are rounded a few times."""
    torch, api = _cuda()
    v, k, S = 2, 64, 8
    fc = random_hclt(v, k, k, 1)      # one sum node; leaf i always takes category i
    m = api.CuMetaBitsProbCircuit(fc)
    u = np.random.default_rng(1).uniform(0.01, 0.99, (S, k)).astype(np.float32)
    gumbel = lambda: -np.log(-np.log(u.astype(np.float64) * (1.0 - 1e-6) + 1e-6))
    p = np.full((S, fc.num_parameters), -np.inf, np.float32)
    p[:, :k] = (np.random.default_rng(2).uniform(-3, 3, (S, k)) * temperature - gumbel()).astype(np.float32)
    leaves = p[:, k:].reshape(S, v, k, k)
    leaves[:, :, np.arange(k), np.arange(k)] = 0.0
    z = (p[:, :k].astype(np.float64) + gumbel()) / temperature
    want = np.exp(z - z.max(1, keepdims=True))
    want /= want.sum(1, keepdims=True)
    dp, du = torch.from_numpy(p).cuda(), torch.from_numpy(u).cuda()
    if not rows:
        dp, du = dp.t().contiguous().t(), du.t().contiguous().t()
    got = api.gumbel_sample(m, dp, v, k, temperature, u=du).cpu().numpy()
    assert np.abs(got - want[:, None, :]).max() <= 5e-7 * want.max()
