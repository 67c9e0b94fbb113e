"""The work this framework does for its users, as cases that can be timed one by one.

Kinds of work, each through the public entry points a program calls:

  train    one training step of the GCN on one rank, as dist_train.train runs it: forward through the DistGCNLayers
           (stage loop + dense transform), loss over the local train rows, backward, optimiser step
  infer    the forward pass alone, no gradients (evaluation between epochs, serving)
  stages   one rank's share of a distributed SpMM: the products of its P stage blocks, accumulated in stage order
  spmm     one local product on a plan that the program holds (SpmmPlan.spmm), plain or with the fused epilogue
  dropin   the nine-argument spmm_cusparse call, with fresh int32 copies of the ids as the reference's binding passes them
  setup    a block that was not seen before: its plan is built, it is multiplied once, and both are dropped

Graphs are the seeded R-MAT graphs of coo_graph.synthetic (self loops added, symmetrically normalised), features N(0, 1).
"""
import math
import os
import socket
import sys
import tempfile

import torch

PACKAGE = os.path.abspath('dist-gnn_b200')
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

# node and edge counts, widths and depths of coo_graph.synthetic.CONFIGS
PLUMBING = dict(nodes=10_000, edges=200_000, feat=128, classes=10, hidden=64, layers=2)
DENSE = dict(nodes=232_965, edges=114_615_892, feat=602, classes=41, hidden=256, layers=2)
SPARSE = dict(nodes=2_449_029, edges=123_718_280, feat=100, classes=47, hidden=256, layers=3)
BLOCK_PARTS = 8                             # row blocks of the 8-GPU partition


def listed():
    return [
        # the smallest training job: launches and host work count
        dict(name='train_plumbing', kind='train', **PLUMBING),
        # an ordinary one: the default model (3 layers, hidden 256) on a ragged mid-sized graph that fits the L2 in parts
        dict(name='train_mid', kind='train', nodes=150_001, edges=2_400_000, feat=100, classes=47, hidden=256, layers=3),
        # few nodes with very long rows, wide odd features (602) and odd class count (41)
        dict(name='train_dense', kind='train', **DENSE),
        # the headline job: 2.4 M nodes, 124 M edges on one GPU
        dict(name='train_sparse', kind='train', **SPARSE),
        # evaluation on an eighth of the headline graph
        dict(name='infer_eighth', kind='infer', nodes=306_128, edges=15_464_784, feat=100, classes=47, hidden=256, layers=3),
        # what one of 8 GPUs multiplies in one 256-wide distributed SpMM: eight blocks with about six entries per row
        dict(name='stages_of_8', kind='stages', nodes=SPARSE['nodes'], edges=SPARSE['edges'], parts=BLOCK_PARTS, width=256),
        # points of the SpMM sweep: short rows and a narrow operand; long rows, an operand far larger than the L2
        dict(name='spmm_1m_16_f64', kind='spmm', nodes=1_000_000, edges=16_000_000, width=64, epilogue=False),
        dict(name='spmm_4m_64_f256', kind='spmm', nodes=4_000_000, edges=256_000_000, width=256, epilogue=False),
        # a class-wide operand with odd rows (41 floats) and the fused epilogue: D^-1/2 kept out of the values, bias, ReLU
        dict(name='spmm_200k_50_f41', kind='spmm', nodes=200_003, edges=10_000_000, width=41, epilogue=True),
        # the drop-in call: a block of the two-rank plumbing graph, and a stage block of the headline graph
        dict(name='dropin_small', kind='dropin', nodes=10_000, edges=200_000, parts=2, width=128),
        dict(name='dropin_block', kind='dropin', nodes=SPARSE['nodes'], edges=SPARSE['edges'], parts=BLOCK_PARTS, width=256),
        # a loader's block on its way into the job: plan construction and the first product
        dict(name='setup_300k', kind='setup', nodes=300_007, edges=15_000_000, width=100),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _graph(rng, low, high, most_edges):
    """Node and (even) directed edge count: average degree 4 to 500, density of at most 1 %."""
    nodes = _log(rng, low, high)
    degree = _log(rng, 4, max(5, min(500, nodes // 100)))
    return nodes, max(2, min(nodes * degree, int(most_edges)) // 2 * 2)


def draw(rng):
    kind = rng.choice(['train', 'train', 'train', 'train', 'infer', 'stages', 'spmm', 'spmm', 'spmm', 'dropin', 'dropin', 'setup'])
    if kind in ('train', 'infer'):
        feat, hidden, classes, layers = _log(rng, 16, 602), _log(rng, 16, 256), rng.randint(2, 47), rng.randint(2, 4)
        widths = 2 * (feat + hidden * (2 * layers - 3) + classes)
        nodes, edges = _graph(rng, 2_000, SPARSE['nodes'], min(SPARSE['edges'], 1.2e11 / widths))
        return dict(kind=kind, nodes=nodes, edges=edges, feat=feat, classes=classes, hidden=hidden, layers=layers)
    if kind == 'setup':
        nodes, edges = _graph(rng, 2_000, 1_000_000, 40_000_000)
        return dict(kind=kind, nodes=nodes, edges=edges, width=_log(rng, 4, 256))
    width = _log(rng, 1, 512)
    if rng.random() < 0.5:                  # half of the widths are whole 16-byte pieces, as models have them
        width += (-width) % 4
    if kind == 'spmm':
        nodes, edges = _graph(rng, 1_000, 4_000_000, min(128_000_000, 6e10 / width))
        return dict(kind=kind, nodes=nodes, edges=edges, width=width, epilogue=rng.random() < 0.3)
    nodes, edges = _graph(rng, 10_000, SPARSE['nodes'], SPARSE['edges'])
    return dict(kind=kind, nodes=nodes, edges=edges, parts=rng.choice([2, 4, 8]), width=width)


# ---- inputs ------------------------------------------------------------------------------------------------------------
_env = None


def _environment():
    """The one-rank environment of a training program, made once per process."""
    global _env
    if _env is None:
        from dist_utils import DistEnv
        with socket.socket() as s:
            s.bind(('127.0.0.1', 0))
            port = s.getsockname()[1]
        os.environ.update(MASTER_ADDR='127.0.0.1', MASTER_PORT=str(port))
        os.environ.setdefault('DIST_GNN_LOG_ROOT', os.path.join(tempfile.gettempdir(), 'dist_gnn_cases_logs'))
        _env = DistEnv(0, 1, 'nccl')
    return _env


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device='cuda', dtype=torch.float32)


def _adjacency(case, seed):
    from coo_graph import graph_utils, synthetic
    edge_index = synthetic.rmat_edge_index(case['nodes'], case['edges'], seed, device='cuda')
    return graph_utils.sym_normalization(edge_index, case['nodes'])


def _row_block(case, seed):
    """Rank 0's blocks of the P-way partition."""
    from coo_graph import graph_utils
    n = -(-case['nodes'] // case['parts'])
    adj = _adjacency(case, seed)
    idx, val = adj.indices(), adj.values()
    rows = int(torch.searchsorted(idx[0].contiguous(), n))
    block = torch.sparse_coo_tensor(idx[:, :rows].clone(), val[:rows].clone(), (n, n * case['parts']), is_coalesced=True, check_invariants=False)
    return n, graph_utils.sparse_2d_split(block, n, split_dim=1)


def prepare(case, seed):
    kind, gen = case['kind'], torch.Generator(device='cuda').manual_seed(seed)
    state = {'kind': kind}
    if kind in ('train', 'infer'):
        from coo_graph import COO_Graph, Parted_COO_Graph, synthetic
        from models import GCN
        env = _environment()
        full = COO_Graph.from_dict('cases', synthetic.make_dataset(
            num_nodes=case['nodes'], directed_edges=case['edges'], feat_dim=case['feat'], num_classes=case['classes'],
            split=(0.6, 0.2, 0.2), seed=seed, device='cuda', features_on_device=True), device='cuda')
        g = Parted_COO_Graph.from_full(full, 0, 1)
        dims = [case['feat']] + [case['hidden']] * (case['layers'] - 1) + [case['classes']]
        model = GCN(g, env, hidden_dim=case['hidden'], num_layers=case['layers'], weights=synthetic.glorot_weights(dims, seed))
        g.plan(0)
        # Plain SGD: its update is a smooth function of the gradient, so that rounding differences stay what they are
        # (Adam's first steps turn the sign of a gradient that is zero up to rounding into a full-sized step).
        state.update(g=g, model=model, optimizer=torch.optim.SGD(model.parameters(), lr=0.01), loss_func=torch.nn.CrossEntropyLoss())
    elif kind == 'stages':
        import spmm_cpp
        n, parts = _row_block(case, seed)
        state.update(plans=[spmm_cpp.SpmmPlan.from_coo(p) for p in parts], x=[_randn(gen, n, case['width']) for _ in parts],
                     z=torch.empty(n, case['width'], device='cuda'))
    elif kind == 'spmm':
        import spmm_cpp
        n, width = case['nodes'], case['width']
        state.update(plan=spmm_cpp.SpmmPlan.from_coo(_adjacency(case, seed)), b=_randn(gen, n, width), c=torch.empty(n, width, device='cuda'), options={})
        if case['epilogue']:
            state['options'] = dict(row_scale=torch.rand(n, generator=gen, device='cuda') + 0.5, bias=_randn(gen, width), relu=True)
    elif kind == 'dropin':
        n, parts = _row_block(case, seed)
        state.update(a=parts[1], b=_randn(gen, n, case['width']), c=_randn(gen, n, case['width']))
    else:
        state.update(a=_adjacency(case, seed), b=_randn(gen, case['nodes'], case['width']))
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(state):
    kind = state['kind']
    if kind == 'train':
        from dist_train import local_loss
        g, model = state['g'], state['model']
        outputs = model(g.features)
        state['optimizer'].zero_grad()
        loss = local_loss(g, outputs, state['loss_func'])
        loss.backward()
        state['optimizer'].step()
        weights = model.weights()
        return {'loss': loss.detach(), 'outputs': outputs.detach(), 'grads': [w.grad for w in weights], 'weights': [w.detach() for w in weights]}
    if kind == 'infer':
        with torch.no_grad():
            return state['model'](state['g'].features)
    if kind == 'stages':
        for s, (plan, x) in enumerate(zip(state['plans'], state['x'])):
            plan.spmm(x, state['z'], 1.0, 0.0 if s == 0 else 1.0)
        return state['z']
    if kind == 'spmm':
        return state['plan'].spmm(state['b'], state['c'], 1.0, 0.0, **state['options'])
    import spmm_cpp
    a = state['a']
    if kind == 'dropin':
        idx = a.indices()
        spmm_cpp.spmm_cusparse(idx[0].int(), idx[1].int(), a.values(), a.size(0), a.size(1), state['b'], state['c'], 1.0, 1.0)
        return state['c']
    c = torch.empty(a.size(0), state['b'].size(1), device='cuda')
    return spmm_cpp.SpmmPlan.from_coo(a).spmm(state['b'], c, 1.0, 0.0)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------
def work(case):
    """Bytes: the sparse block once per product (column id and value of every entry, row offsets), every dense operand read
    once, every result written once (and read first where it is added to).  Flops: 2 per entry and column, 2 per
    multiply-add of the dense transforms."""
    kind, n = case['kind'], case['nodes']
    nnz = case['edges'] + n                                                # with the self loops
    if kind in ('train', 'infer'):
        dims = [case['feat']] + [case['hidden']] * (case['layers'] - 1) + [case['classes']]
        total_bytes = total_flops = 0
        for l, (d_in, d_out) in enumerate(zip(dims[:-1], dims[1:])):
            total_bytes += 8 * nnz + 4 * n + 4 * n * (d_in + d_out)        # forward: input in, activation out
            total_flops += 2 * nnz * min(d_in, d_out) + 2 * n * d_in * d_out
            if kind == 'train':                                            # backward: gradient and input in, next gradient out
                total_bytes += 8 * nnz + 4 * n + 4 * n * (d_in + d_out + (d_in if l else 0))
                total_flops += 2 * nnz * d_out + 2 * n * d_in * d_out * (2 if l else 1)
        return {'bytes': total_bytes, 'flops': total_flops}
    width = case['width']
    if kind == 'stages':
        rows = -(-n // case['parts'])
        return {'bytes': 8 * nnz / case['parts'] + 4 * rows * case['parts'] + 4 * width * (min(n, nnz / case['parts']) + rows),
                'flops': 2 * nnz / case['parts'] * width}
    if kind == 'dropin':                                                   # ids come as int64, the block is added to C
        rows, entries = -(-n // case['parts']), nnz / case['parts'] ** 2
        return {'bytes': 20 * entries + 4 * width * (min(rows, entries) + 2 * rows), 'flops': 2 * entries * width}
    per_entry = 20 if kind == 'setup' else 8                               # setup reads the int64 ids of the loader's block
    return {'bytes': per_entry * nnz + 4 * n + 8 * n * width, 'flops': 2 * nnz * width}


def tolerance(case):
    """fp32 sums in another order: 1e-5.  A training step or forward pass chains up to eight products and as many dense
    transforms, each within that order of magnitude."""
    return {'rel': 3e-5 if case['kind'] in ('train', 'infer') else 1e-5}
