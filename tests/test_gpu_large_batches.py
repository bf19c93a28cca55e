"""Batches beyond 65535 tiles of a kernel's second grid dimension."""
import numpy as np
import pytest

from tests.helpers import random_hclt, rel_err
from tests.test_gpu_em import TOL, _cuda

pytestmark = pytest.mark.gpu


def test_soft_evidence():
    torch, api = _cuda()
    fc = random_hclt(2, 16, 2, 1)
    m = api.CuMetaBitsProbCircuit(fc)
    B = 65535 * 32 + 40
    soft = torch.randn(2, 2, B, device="cuda").permute(2, 1, 0)     # [B, variables, categories], column-major
    out = torch.empty(B, device="cuda")
    ws, _ = api.forward_ex(m, soft=soft, B=B, ll_out=out)
    tail = torch.empty(100, device="cuda")
    small = api.CuMetaBitsProbCircuit(fc)
    api.forward_ex(small, soft=soft, row_start=B - 99, B=100, ll_out=tail)
    assert torch.equal(out[-100:], tail)
    m.lib.pcb_clear_flows(m.handle, 0.0, None)
    api.backward(m, ws)
    # one learnable leaf per (variable, state): the flow of a variable's leaves is one per example
    stats = m.heap().reshape(32, 5)[:, 2:].astype(np.float64)
    assert abs(stats.sum() - 2.0 * B) <= 1e-3 * B


def test_normalised_flows():
    torch, api = _cuda()
    fc = random_hclt(2, 16, 2, 1)
    B = 65535 * 32 + 40
    data = torch.randint(0, 2, (2, B), device="cuda", dtype=torch.uint8)
    full = api.per_sample_normalized_flows(api.CuMetaBitsProbCircuit(fc), api.DeviceData.from_colmajor(data), batch_size=B)
    tail = api.per_sample_normalized_flows(api.CuMetaBitsProbCircuit(fc), api.DeviceData.from_colmajor(data[:, -128:].contiguous()),
                                           batch_size=128)
    assert torch.equal(full[-128:], tail)


def test_leaf_statistics():
    torch, api = _cuda()
    fc = random_hclt(2, 16, 2, 1)
    m = api.CuMetaBitsProbCircuit(fc)
    half = 65535 * 128 + 300
    data = api.DeviceData.from_colmajor(torch.randint(0, 2, (2, 2 * half), device="cuda", dtype=torch.uint8))
    heaps = []
    for parts in (1, 2):
        m.free_workspaces()
        m.lib.pcb_clear_flows(m.handle, 0.0, None)
        for i in range(parts):
            n = 2 * half // parts
            ws, _ = api.forward(m, data, row_start=1 + i * n, B=n)
            api.backward(m, ws)
        heaps.append(m.heap())
    assert rel_err(heaps[0], heaps[1]) <= TOL
