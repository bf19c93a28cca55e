"""Shared builders and comparison rules for the test-suite."""
import numpy as np

from lvd_pg_b200 import structures as st
from lvd_pg_b200.circuit import compile_circuit


def rel_err(a, ref, floor_frac=1e-6):
    """|a - ref| / max(|ref|, floor_frac * max|ref|): the parity metric for flows and parameters
    (values can be exactly 0)."""
    a = np.asarray(a, np.float64)
    ref = np.asarray(ref, np.float64)
    scale = np.maximum(np.abs(ref), floor_frac * max(np.abs(ref).max(), 1e-30))
    return float((np.abs(a - ref) / scale).max()) if ref.size else 0.0


def random_hclt(v, k, c, seed, tree_seed=None):
    rng = np.random.default_rng(seed if tree_seed is None else tree_seed)
    parent = st.root_tree_at_center(v, st.random_spanning_tree(v, rng))
    return st.hclt_flat(parent, c, k, seed=seed)


def random_data(rows, v, c, seed, missing_frac=0.0):
    rng = np.random.default_rng(seed)
    data = rng.integers(0, c, (rows, v)).astype(np.uint8)
    miss = None
    if missing_frac > 0:
        miss = (rng.random((rows, v)) < missing_frac).astype(np.uint8)
    return data, miss


def simple3(fixed=False, num_cats=5, seed=0):
    rng = np.random.default_rng(seed)
    return compile_circuit(st.simple_3vars_circuit(num_cats=num_cats, fixed=fixed, rng=rng))


# ---- golden fixtures (tests/golden/make_golden.py) -------------------------------------------
import os

GOLDEN_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
GOLDEN_CASES = ["simple3", "hclt_v6_k3_c4", "hclt_chain5_k2_c2"]


def load_golden(name):
    """Returns (golden arrays, FlatCircuit with the golden's parameters)."""
    from oracle import oracle as orc
    g = np.load(os.path.join(GOLDEN_DIR, name + ".npz"))
    if name == "simple3":
        fc = compile_circuit(st.simple_3vars_circuit(num_cats=5, fixed=False, rng=None))
    else:
        fc = compile_circuit(st.hclt_graph(g["parent"], int(g["num_cats"]), int(g["k"]), None))
    orc.update_parameters(fc, g["theta"].astype(np.float32))
    return g, fc


def flat_stats(fc, edge_aggr_down, heap, edge2param):
    """Sufficient statistics in flat parameter order: edge flows of sum edges, then the C flow
    slots of every learnable leaf."""
    out = np.zeros(fc.num_parameters, np.float64)
    up = fc.down2up.astype(np.int64) - 1
    pid = edge2param[up].astype(np.int64)
    ok = pid > 0
    out[pid[ok] - 1] = edge_aggr_down[ok]
    pos = fc.num_inner_params
    for nid in fc.input_node_ids.astype(np.int64):
        if fc.node_fixed[nid - 1]:
            continue
        c = int(fc.node_num_cats[nid - 1])
        hs = int(fc.node_heap_start[nid - 1]) - 1
        out[pos:pos + c] = heap[hs + c:hs + 2 * c]
        pos += c
    return out


def under_one_root(fcs, children, user_tag=False):
    """One circuit over the nodes and variables of `fcs` with a new root sum on top: `children` are (circuit, 1-based
    node id) pairs, equally weighted; `user_tag` makes it the fake root of a multi-head circuit.  Runs of consecutive
    nodes stay consecutive."""
    from lvd_pg_b200.circuit import PCB_SUM, TAG_FIRST, TAG_LAST, TAG_USER, finish_flat
    node0 = np.concatenate([[0], np.cumsum([f.num_nodes for f in fcs])])
    heap0 = np.concatenate([[0], np.cumsum([len(f.heap) for f in fcs])])
    cat = lambda xs: np.concatenate([np.asarray(x, np.int64) for x in xs])
    up = {"up_parent": [], "up_prime": [], "up_sub": [], "up_logp": [], "up_tag": []}
    ends, total = [], 0
    for lay in range(max(len(f.up_layer_ends) for f in fcs)):
        for f, n0 in zip(fcs, node0):
            if lay >= len(f.up_layer_ends):
                continue
            sl = slice(int(f.up_layer_ends[lay - 1]) if lay else 0, int(f.up_layer_ends[lay]))
            for name in up:
                x = getattr(f, name)[sl]
                if name in ("up_parent", "up_prime", "up_sub"):
                    x = np.where(x > 0, x.astype(np.int64) + n0, 0)
                up[name].append(x)
            total += sl.stop - sl.start
        ends.append(total)
    h = len(children)
    root = int(node0[-1]) + 1
    up["up_parent"].append(np.full(h, root))
    up["up_prime"].append(np.array([node0[i] + n for i, n in children]))
    up["up_sub"].append(np.zeros(h, np.int64))
    up["up_logp"].append(np.full(h, -np.log(h), np.float32))
    tag = np.full(h, TAG_USER if user_tag else 0, np.uint8)
    tag[0] |= TAG_FIRST
    tag[-1] |= TAG_LAST
    up["up_tag"].append(tag)
    ends.append(total + h)
    kind = np.concatenate([f.node_kind for f in fcs] + [[PCB_SUM]])
    hstart = cat([np.where(f.node_num_cats > 0, f.node_heap_start.astype(np.int64) + o, 0) for f, o in zip(fcs, heap0)] + [[0]])
    return finish_flat(kind, cat([f.node_var for f in fcs] + [[0]]), cat([f.node_num_cats for f in fcs] + [[0]]), hstart,
                       cat([f.node_fixed for f in fcs] + [[0]]), cat(up["up_parent"]), cat(up["up_prime"]), cat(up["up_sub"]),
                       np.concatenate(up["up_logp"]), np.concatenate(up["up_tag"]), ends,
                       cat([f.input_node_ids.astype(np.int64) + n for f, n in zip(fcs, node0)]),
                       np.concatenate([f.heap for f in fcs]), max(f.num_vars for f in fcs))


def without_root(fc):
    """`fc` without its last node and that node's edges: nodes for `under_one_root`, no circuit of its own."""
    out = fc.copy()
    keep = fc.up_parent != fc.num_nodes
    for name in ("up_parent", "up_prime", "up_sub", "up_logp", "up_tag"):
        setattr(out, name, getattr(fc, name)[keep])
    out.up_layer_ends = np.unique(np.cumsum(keep)[fc.up_layer_ends.astype(np.int64) - 1])
    for name in ("node_kind", "node_var", "node_num_cats", "node_heap_start", "node_fixed"):
        setattr(out, name, getattr(fc, name)[:-1])
    return out
