"""Random circuits that are no latent trees: products over permuted, shared and consecutive runs of nodes, sums with and
without a second child, blocks whose children have other readers, thin and odd blocks.  What the tables of the steps make
of them (blocks, fused products, single nodes) agrees with the oracle on every pass that goes by them."""
import numpy as np
import pytest

from lvd_pg_b200.circuit import PCB_INPUT, PCB_PRODUCT, PCB_SUM, TAG_FIRST, TAG_LAST, finish_flat
from tests.helpers import random_data, rel_err
from tests.test_gpu_em import TOL, _cuda

pytestmark = pytest.mark.gpu


def _random_circuit(seed):
    """(circuit, variables, categories): blocks of K nodes are multiplied and mixed until two cover every variable."""
    rng = np.random.default_rng(seed)
    V, K, C = int(rng.integers(3, 9)), int(rng.choice([4, 16, 17, 20, 32, 40, 72])), int(rng.choice([2, 3, 5]))
    kind, var, layer, edges, blocks = [], [], [], {}, []

    def new(k, n, v=0):
        kind.extend([k] * n)
        var.extend([v] * n)
        layer.extend([0] * n)
        return len(kind) - n + 1

    def add(node, es):
        edges[node] = es
        layer[node - 1] = 1 + max(layer[c - 1] for p, s, _ in es for c in (p, s) if c)

    def block(base, n, parts):
        for b in parts:
            b["readers"] += 1
        blocks.append(dict(base=base, n=n, scope=frozenset().union(*[b["scope"] for b in parts]), readers=0))

    for v in rng.permutation(V):
        for _ in range(int(rng.integers(1, 3))):
            blocks.append(dict(base=new(PCB_INPUT, K, int(v) + 1), n=K, scope=frozenset([int(v)]), readers=0))
    for step in range(200):
        if step > 8 and sum(len(b["scope"]) == V for b in blocks) >= 2:
            break
        usable = [b for b in blocks if b["n"] == K and (not b["readers"] or rng.random() < 0.15)] or [b for b in blocks if b["n"] == K]
        parts = [usable[rng.integers(len(usable))]]
        others = [b for b in usable if not b["scope"] & parts[0]["scope"]]
        if rng.random() < 0.55 and others:      # a block of products
            for i in rng.permutation(len(others)):
                if len(parts) < 5 and rng.random() < 0.8 and not any(others[i]["scope"] & p["scope"] for p in parts):
                    parts.append(others[i])
            if len(parts) > 1:
                order = [np.arange(K) if rng.random() < 0.85 else rng.permutation(K) for _ in parts]
                base = new(PCB_PRODUCT, K)
                for j in range(K):
                    c = [p["base"] + int(o[j]) for p, o in zip(parts, order)] + [0]
                    add(base + j, [(c[i], c[i + 1], 0.0) for i in range(0, len(parts), 2)])
                block(base, K, parts)
        elif rng.random() < 0.9:                # a block of sums, over pairs of children or single ones
            if others and rng.random() < 0.5:
                parts.append(others[rng.integers(len(others))])
            R = K if rng.random() < 0.8 else int(rng.choice([1, 5, 16, 33]))
            base = new(PCB_SUM, R)
            for r in range(R):
                w = np.log(rng.dirichlet(np.ones(K)) + 1e-12)
                add(base + r, [(parts[0]["base"] + j, parts[1]["base"] + j if len(parts) > 1 else 0, w[j]) for j in range(K)])
            block(base, R, parts)
    tops = [b["base"] + j for b in blocks if len(b["scope"]) == V for j in range(b["n"])]
    root = new(PCB_SUM, 1)
    add(root, [(c, 0, w) for c, w in zip(tops, np.log(rng.dirichlet(np.ones(len(tops))) + 1e-12))])
    up, ends = [], []
    for lay in range(1, max(layer) + 1):
        for n in [n for n in range(1, root + 1) if layer[n - 1] == lay]:
            es = edges[n]
            up += [(n, p, s, w, (i == 0) * TAG_FIRST | (i == len(es) - 1) * TAG_LAST) for i, (p, s, w) in enumerate(es)]
        ends.append(len(up))
    up = [np.array(x) for x in zip(*up)]
    kind = np.array(kind, np.uint8)
    leaf = np.nonzero(kind == PCB_INPUT)[0]
    heap = np.zeros((len(leaf), 2 * C + 1), np.float32)
    heap[:, :C] = np.log(rng.dirichlet(np.ones(C), len(leaf)) + 1e-9)
    start = np.zeros(root, np.int64)
    start[leaf] = np.arange(len(leaf)) * (2 * C + 1) + 1
    return finish_flat(kind, var, np.where(kind == PCB_INPUT, C, 0), start, np.zeros(root), *up[:3], up[3].astype(np.float32), up[4], ends,
                       leaf + 1, heap.reshape(-1), V), V, C


@pytest.mark.parametrize("chain", ["1", "0"])
@pytest.mark.parametrize("seed", range(16))
def test_every_pass_against_the_oracle(oracle, monkeypatch, seed, chain):
    monkeypatch.setenv("PCB_CHAIN", chain)
    torch, api = _cuda()
    fc, V, C = _random_circuit(seed)
    rng = np.random.default_rng(seed)
    data, miss = random_data(int(rng.choice([1, 33, 70, 300])), V, C, seed, 0.1)
    ref, m = fc.copy(), api.CuMetaBitsProbCircuit(fc)
    mars_ref = oracle.forward(ref, data, miss=miss)
    flows_ref, aggr_ref = oracle.backward(ref, mars_ref)
    oracle.input_flows(ref, flows_ref, data, miss=miss)
    ws, B = api.forward(m, api.DeviceData(data, m.device, miss))
    m.lib.pcb_clear_flows(m.handle, 0.0, None)
    api.backward(m, ws)
    assert rel_err(m.mars(ws, B), mars_ref, 1e-2) <= TOL
    assert rel_err(m.flows(ws, B), flows_ref) <= TOL
    sums = ref.edge_is_sum[ref.down2up.astype(np.int64) - 1]
    assert rel_err(m.edge_aggr()[sums], aggr_ref[sums]) <= TOL
    assert rel_err(m.heap(), ref.heap) <= TOL
    # parameter sets: KLD and its gradients by warps and by tiles, relaxed samples
    for S in (1, 3, 20):
        p1, p2 = (oracle.normalize_params(fc, oracle.vectorize(fc) + rng.normal(0, 0.3, (S, fc.num_parameters)).astype(np.float32))
                  for _ in range(2))
        out, reuse = api.kld(m, torch.from_numpy(p1).cuda(), torch.from_numpy(p2).cuda())
        klds_ref, ek_ref = oracle.kld(fc, p1, p2)
        assert rel_err(api.kld_matrices(m, reuse)[0], klds_ref, 1e-2) <= TOL
        grads = oracle.kld_backward(fc, p1, p2, klds_ref, ek_ref)
        g1, g2 = api.kld_backward(m, reuse=reuse)
        assert rel_err(g1.cpu().numpy(), grads["param_grads1"], 1e-2) <= TOL
        assert rel_err(g2.cpu().numpy(), grads["param_grads2"], 1e-4) <= TOL
        u = rng.random((S, fc.num_inner_params), dtype=np.float32)
        got = api.gumbel_sample(m, torch.from_numpy(p1).cuda(), V, C, 0.7, u=torch.from_numpy(u).cuda()).cpu().numpy()
        assert rel_err(got, oracle.sample_soft(fc, p1, u, 0.7, S, C)[0], 1e-4) <= TOL
