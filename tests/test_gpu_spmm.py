"""Parity of the CUDA SpMM (through the C ABI) with the reference's outputs and with the CPU oracle.  Needs a GPU."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import assert_close
from oracle import ref_gcn, ref_graph

pytestmark = pytest.mark.gpu
TOL = 1e-5   # fp32 parity tolerance of the path (max-abs and Frobenius relative error); the sum order differs


def dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.to('cuda', dtype=dtype) if dtype else t.cuda()


def make_plan(A, **kw):
    import spmm_cpp
    return spmm_cpp.SpmmPlan(dev(A.row, torch.int32), dev(A.col, torch.int32), dev(A.val), A.shape[0], A.shape[1], **kw)


def random_coo(rng, m, k, nnz, heavy=None):
    flat = rng.choice(m * k, size=min(nnz, m * k), replace=False)
    row, col = flat // k, flat % k
    if heavy:   # (row id, entries) pairs forced to be dense-ish rows
        for r, cnt in heavy:
            keep = row != r
            row, col = row[keep], col[keep]
            row = np.concatenate((row, np.full(cnt, r)))
            col = np.concatenate((col, rng.choice(k, cnt, replace=False)))
    val = rng.standard_normal(row.size, dtype=np.float32)
    return ref_graph.fast_coalesce_sorted(row.astype(np.int64), col.astype(np.int64), val, (m, k))


def test_library_exports_and_version():
    import spmm_cpp
    assert spmm_cpp.lib().dg_version() >= 100


def test_golden_cases_through_the_drop_in_signature(golden):
    """spmm_cusparse(row, col, val, A_row, A_col, B, C, alpha, beta) against the reference's C.addmm_(A, B)."""
    import spmm_cpp
    z = golden('spmm_cases')
    for name in z['names']:
        g = lambda key: z[f'{name}/{key}']
        m, k, F = (int(v) for v in g('dims'))
        alpha, beta = (float(v) for v in g('ab'))
        C = dev(g('C0'))
        spmm_cpp.spmm_cusparse(dev(g('row')), dev(g('col')), dev(g('val')), m, k, dev(g('B')), C, alpha, beta)
        assert_close(C.cpu().numpy(), g('C'), TOL, name)


def test_drop_in_route_keeps_plans_only_for_the_same_matrix():
    """spmm_cusparse recognises a block by the address of its values and re-checks the ids it is given: the same block
    again reuses the plan (fresh int32 copies of the ids, as the reference's binding passes them), other ids at the same
    values address build a new one, and the transient-plan route (cache off) gives the same numbers."""
    import spmm_cpp
    rng = np.random.Generator(np.random.PCG64(91))
    A = random_coo(rng, 200, 150, 3000, heavy=[(9, 140)])
    B = rng.standard_normal((150, 36), dtype=np.float32)
    C0 = rng.standard_normal((200, 36), dtype=np.float32)
    want = ref_gcn.spmm_coo(A, B, C0.copy(), 1.0, 1.0)
    row, col, val = dev(A.row, torch.int32), dev(A.col, torch.int32), dev(A.val)
    spmm_cpp._dropin_plans.clear()
    for _ in range(3):
        C = dev(C0)
        spmm_cpp.spmm_cusparse(row.clone(), col.clone(), val, 200, 150, dev(B), C, 1, 1)
        assert_close(C.cpu().numpy(), want, TOL, 'drop-in, cached plan')
    assert len(spmm_cpp._dropin_plans) == 1
    first_plan = next(iter(spmm_cpp._dropin_plans.values()))[0]
    # another matrix whose values live at the same address: same nnz and shape, rows reversed
    A2 = ref_graph.fast_coalesce_sorted((199 - A.row).astype(np.int64), A.col.astype(np.int64), A.val, (200, 150))
    val.copy_(dev(A2.val))
    C = dev(C0)
    spmm_cpp.spmm_cusparse(dev(A2.row, torch.int32), dev(A2.col, torch.int32), val, 200, 150, dev(B), C, 1, 1)
    assert_close(C.cpu().numpy(), ref_gcn.spmm_coo(A2, B, C0.copy(), 1.0, 1.0), TOL, 'drop-in after the matrix changed')
    assert len(spmm_cpp._dropin_plans) == 1 and next(iter(spmm_cpp._dropin_plans.values()))[0] is not first_plan
    keep = spmm_cpp.DROPIN_PLAN_CACHE
    try:
        spmm_cpp.DROPIN_PLAN_CACHE = 0
        C = dev(C0)
        spmm_cpp.spmm_cusparse(dev(A2.row, torch.int32), dev(A2.col, torch.int32), val, 200, 150, dev(B), C, 1, 1)
        assert_close(C.cpu().numpy(), ref_gcn.spmm_coo(A2, B, C0.copy(), 1.0, 1.0), TOL, 'drop-in, transient plan')
    finally:
        spmm_cpp.DROPIN_PLAN_CACHE = keep
        spmm_cpp._dropin_plans.clear()


@pytest.mark.parametrize('F', [1, 2, 3, 4, 6, 8, 10, 16, 20, 32, 41, 47, 64, 100, 128, 130, 256, 300, 512, 602, 1024])
def test_widths_against_oracle(F):
    rng = np.random.Generator(np.random.PCG64(F))
    A = random_coo(rng, 257, 193, 4000, heavy=[(5, 150), (256, 193)])
    B = rng.standard_normal((193, F), dtype=np.float32)
    C0 = rng.standard_normal((257, F), dtype=np.float32)
    want = ref_gcn.spmm_coo(A, B, C0.copy(), 0.75, -1.25)
    for kw in ({}, {'heavy_threshold': 16, 'chunk': 7}):     # default bins, and bins that force the split-row path
        plan = make_plan(A, **kw)
        C = dev(C0)
        plan.spmm(dev(B), C, 0.75, -1.25)
        assert_close(C.cpu().numpy(), want, TOL, f'F={F} {kw}')


def test_beta_zero_ignores_garbage_in_c():
    rng = np.random.Generator(np.random.PCG64(11))
    A = random_coo(rng, 100, 80, 900, heavy=[(7, 60)])
    B = rng.standard_normal((80, 48), dtype=np.float32)
    want = ref_gcn.spmm_coo(A, B, np.zeros((100, 48), dtype=np.float32), 2.0, 0.0)
    for kw in ({}, {'heavy_threshold': 8, 'chunk': 8}):
        C = torch.full((100, 48), float('nan'), device='cuda')
        make_plan(A, **kw).spmm(dev(B), C, 2.0, 0.0)
        assert_close(C.cpu().numpy(), want, TOL, 'beta=0')


def test_empty_shapes():
    import spmm_cpp
    empty = ref_graph.Coo(np.zeros(0, np.int64), np.zeros(0, np.int64), np.zeros(0, np.float32), (6, 5))
    plan = make_plan(empty)
    C = torch.ones(6, 4, device='cuda')
    plan.spmm(torch.ones(5, 4, device='cuda'), C, 1.0, 1.0)
    assert torch.equal(C.cpu(), torch.ones(6, 4))
    plan.spmm(torch.ones(5, 4, device='cuda'), C, 1.0, 0.0)
    assert torch.equal(C.cpu(), torch.zeros(6, 4))
    assert plan.rowptr().tolist() == [0] * 7
    zero_rows = ref_graph.Coo(np.zeros(0, np.int64), np.zeros(0, np.int64), np.zeros(0, np.float32), (0, 5))
    make_plan(zero_rows).spmm(torch.ones(5, 4, device='cuda'), torch.ones(0, 4, device='cuda'))
    spmm_cpp.spmm_cusparse(torch.zeros(0, dtype=torch.int32, device='cuda'), torch.zeros(0, dtype=torch.int32, device='cuda'),
                           torch.zeros(0, device='cuda'), 3, 2, torch.ones(2, 0, device='cuda'), torch.ones(3, 0, device='cuda'), 1, 1)


def test_row_strided_operands_and_unaligned_views():
    rng = np.random.Generator(np.random.PCG64(12))
    A = random_coo(rng, 90, 70, 1200)
    for F, ld, off in ((32, 40, 0), (32, 35, 1), (6, 9, 3)):     # aligned stride, odd stride, odd offset
        Bbig = rng.standard_normal((70, ld + off), dtype=np.float32)
        Cbig = rng.standard_normal((90, ld + off), dtype=np.float32)
        want = ref_gcn.spmm_coo(A, np.ascontiguousarray(Bbig[:, off:off + F]), np.ascontiguousarray(Cbig[:, off:off + F]), 1.0, 1.0)
        Bd, Cd = dev(Bbig), dev(Cbig)
        make_plan(A).spmm(Bd[:, off:off + F], Cd[:, off:off + F])
        got = Cd.cpu().numpy()
        assert_close(got[:, off:off + F], want, TOL, f'F={F} ld={ld + off}')
        untouched = np.ones(Cbig.shape, dtype=bool)
        untouched[:, off:off + F] = False
        assert np.array_equal(got[untouched], Cbig[untouched])


@pytest.mark.parametrize('F', [20, 47, 256])
def test_fused_epilogue(F):
    rng = np.random.Generator(np.random.PCG64(13))
    A = random_coo(rng, 120, 110, 2500, heavy=[(3, 100)])
    B = rng.standard_normal((110, F), dtype=np.float32)
    C0 = rng.standard_normal((120, F), dtype=np.float32)
    scale = rng.uniform(0.1, 2.0, 120).astype(np.float32)
    bias = rng.standard_normal(F, dtype=np.float32)
    want = ref_gcn.spmm_epilogue(A, B, C0, 1.0, 0.5, row_scale=scale, bias=bias, relu=True)
    for kw in ({}, {'heavy_threshold': 8, 'chunk': 16}):
        C = dev(C0)
        make_plan(A, **kw).spmm(dev(B), C, 1.0, 0.5, row_scale=dev(scale), bias=dev(bias), relu=True)
        assert_close(C.cpu().numpy(), want, TOL, f'epilogue F={F}')
        assert (C >= 0).all()


def test_results_are_bit_reproducible():
    rng = np.random.Generator(np.random.PCG64(14))
    A = random_coo(rng, 500, 400, 30000, heavy=[(0, 400), (499, 333)])
    B = dev(rng.standard_normal((400, 100), dtype=np.float32))
    plan = make_plan(A, heavy_threshold=64, chunk=50)
    outs = []
    for _ in range(3):
        C = torch.zeros(500, 100, device='cuda')
        plan.spmm(B, C, 1.0, 0.0)
        outs.append(C.cpu())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


def test_csr_indexing_is_bit_exact_on_the_reference_partition(golden):
    """Row offsets of every adj_parts block of the reference's own partition (P=2,3), and the plan census."""
    z = golden('graph_small')
    for P in (2, 3):
        for r in range(P):
            pre = f'P{P}/r{r}/'
            nnz, idx, val, shapes = z[pre + 'parts_nnz'], z[pre + 'parts_idx'], z[pre + 'parts_val'], z[pre + 'parts_shape']
            start = 0
            for s in range(P):
                sl = slice(start, start + int(nnz[s]))
                A = ref_graph.Coo(idx[0, sl], idx[1, sl], val[sl], tuple(int(v) for v in shapes[s]))
                start += int(nnz[s])
                plan = make_plan(A)
                assert np.array_equal(plan.rowptr().numpy(), ref_graph.rowptr_of(A))
                st = plan.stats()
                assert st['nnz'] == A.nnz and (st['m'], st['k']) == A.shape
                assert st['touched_columns'] == np.unique(A.col).size
                assert st['max_row_nnz'] == np.bincount(A.row, minlength=A.shape[0]).max()
                assert torch.equal(plan.col.cpu(), torch.from_numpy(A.col.astype(np.int32)))


def test_plan_census_of_heavy_rows():
    rng = np.random.Generator(np.random.PCG64(15))
    A = random_coo(rng, 60, 500, 800, heavy=[(4, 300), (40, 101)])
    st = make_plan(A, heavy_threshold=100, chunk=64).stats()
    deg = np.bincount(A.row, minlength=60)
    assert st['heavy_rows'] == int((deg > 100).sum()) == 2
    assert st['heavy_chunks'] == sum(-(-int(d) // 64) for d in deg if d > 100)
    assert st['heavy_nnz'] == int(deg[deg > 100].sum())


def test_bad_input_is_rejected_before_any_product():
    import spmm_cpp
    row = torch.tensor([0, 2, 1], dtype=torch.int32, device='cuda')      # not ascending
    col = torch.tensor([0, 1, 1], dtype=torch.int32, device='cuda')
    val = torch.ones(3, device='cuda')
    with pytest.raises(RuntimeError, match='row-sorted'):
        spmm_cpp.SpmmPlan(row, col, val, 3, 2)
    with pytest.raises(RuntimeError, match='row-sorted'):                 # column id outside the matrix
        spmm_cpp.SpmmPlan(torch.tensor([0, 1, 2], dtype=torch.int32, device='cuda'), torch.tensor([0, 5, 1], dtype=torch.int32, device='cuda'), val, 3, 2)
    with pytest.raises(RuntimeError, match='CUDA tensor'):
        spmm_cpp.spmm_cusparse(row.cpu(), col.cpu(), val.cpu(), 3, 2, torch.ones(2, 4), torch.ones(3, 4), 1, 1)
    plan = spmm_cpp.SpmmPlan(torch.tensor([0, 1, 2], dtype=torch.int32, device='cuda'), col, val, 3, 2)
    with pytest.raises(RuntimeError):
        plan.spmm(torch.ones(3, 4, device='cuda'), torch.ones(3, 4, device='cuda'))     # B has the wrong row count
    L = spmm_cpp.lib()
    assert L.dg_spmm_csr(None, None, None, 4, None, 4, 4, 1.0, 1.0, 0, None, None, None) == -1
    assert L.dg_spmm_csr(plan.handle, val.data_ptr(), val.data_ptr(), 2, val.data_ptr(), 4, 4, 1.0, 1.0, 0, None, None, None) == -2
    assert L.dg_spmm_csr(plan.handle, val.data_ptr(), val.data_ptr(), 4, val.data_ptr(), 4, 4, 1.0, 1.0, 64, None, None, None) == -4
    assert b'NULL' in L.dg_strerror(-1)
    # after all those refusals the context still computes
    C = torch.zeros(3, 1, device='cuda')
    plan.spmm(torch.ones(2, 1, device='cuda'), C, 1.0, 0.0)
    assert C.cpu().flatten().tolist() == [1.0, 1.0, 1.0]


def _emulated_bcast(parted):
    """One distributed SpMM for P ranks emulated on one GPU: rank r adds plan(A[r][s]) @ X_s for s = 0..P-1 in order."""
    plans = [[make_plan(a) for a in p['adj_parts']] for p in parted]

    def bcast(blocks):
        xs = [dev(np.ascontiguousarray(b)) for b in blocks]
        out = []
        for r in range(len(parted)):
            z = torch.empty_like(xs[r])
            for s, x in enumerate(xs):
                plans[r][s].spmm(x, z, 1.0, 0.0 if s == 0 else 1.0)
            out.append(z.cpu().numpy())
        return out
    return bcast


def test_stage_loop_values_match_reference_run_over_gloo(golden):
    """Every broadcast-SpMM result of the reference's epoch 0 at P=2 (3 forward, 3 backward), with the CUDA kernels
    doing the sparse products and the oracle doing the dense algebra around them; then losses over 3 epochs."""
    from test_oracle_golden import _parted_from_fixture
    z, t = golden('graph_small'), golden('gcn_small')
    parted = _parted_from_fixture(z, 2)
    model = ref_gcn.GcnOracle(_emulated_bcast(parted), [t[f'r0/w0_{i}'] for i in range(3)], [[0, 1]])
    feats = [p['features'] for p in parted]
    for epoch in range(3):
        losses, outputs, trace, btrace = model.epoch(feats, [p['local_labels'] for p in parted], [p['local_train_mask'] for p in parted])
        for r in range(2):
            assert abs(losses[r] - t[f'r{r}/losses'][epoch]) <= 2e-5 * max(1.0, abs(t[f'r{r}/losses'][epoch]))
        if epoch == 0:
            for r in range(2):
                got = [trace[l]['z'][r] for l in range(3)] + [btrace[l]['ag'][r] for l in (2, 1, 0)]
                for i, g in enumerate(got):
                    assert_close(g, t[f'r{r}/bcast_{i}'], TOL, f'rank {r} bcast {i}')
                for l in range(3):
                    assert_close(btrace[l]['dw'][r], t[f'r{r}/dw_{l}'], TOL, f'dW{l}')


@pytest.mark.parametrize('P,c', [(4, 2), (8, 2), (9, 3)])
def test_15d_schedule_with_cuda_products_equals_1d_and_full_product(golden, P, c):
    """1.5D(P, c) == 1D(P/c) == single full product, the identity that pins the 1.5D schedule."""
    from dist_utils import schedule
    z = golden('graph_small')
    n_nodes = int(z['in/meta'][0])
    A = ref_graph.Coo(z['full/adj_idx'][0], z['full/adj_idx'][1], z['full/adj_val'], (n_nodes, n_nodes))
    R = P // c
    parts = [ref_graph.parted_graph(p) for p in ref_graph.partition(A, z['full/features'], z['in/labels'].astype(np.int64), z['in/masks'], R)]
    plans = [[make_plan(a) for a in p['adj_parts']] for p in parts]
    X = [dev(p['features']) for p in parts]
    rows_grp = schedule.row_groups(P, c)
    partial = []
    for rank in range(P):
        b = rank // c
        zr = torch.zeros_like(X[b])
        for st in schedule.stages_15d(rank, P, c):
            assert st.root_global // c == st.part and schedule.col_groups(P, c)[rank % c][st.root_in_group] == st.root_global
            plans[b][st.part].spmm(X[st.part], zr, 1.0, 1.0)
        partial.append(zr)
    full = ref_gcn.spmm_coo(A, np.ascontiguousarray(z['full/features']), np.zeros_like(z['full/features']), 1.0, 0.0)
    pad = parts[0]['adj'].shape[0] * R - n_nodes
    full = np.concatenate((full, np.zeros((pad, full.shape[1]), dtype=np.float32)))
    oracle_15d = ref_gcn.broadcast_15d([p['adj_parts'] for p in parts], [p['features'] for p in parts], P, c)
    n = parts[0]['adj'].shape[0]
    for grp in rows_grp:
        total = partial[grp[0]].clone()
        for r in grp[1:]:
            total += partial[r]
        b = grp[0] // c
        assert_close(total.cpu().numpy(), full[b * n:(b + 1) * n], TOL, f'block {b} vs full product')
        assert_close(total.cpu().numpy(), oracle_15d[grp[0]], TOL, f'block {b} vs 1.5D oracle')


@pytest.mark.parametrize('F', [64, 100, 128, 256, 300, 512, 1024])
@pytest.mark.parametrize('task', [5, 32, 100, 0])
def test_streaming_kernel_against_oracle(F, task):
    """Widths whose rows are 16-byte aligned take the bulk-copy streaming kernel; small task sizes cut rows at many task
    boundaries (carry rows + fix-up), 0 keeps the default.  Includes empty leading/trailing rows and a row spanning
    dozens of tasks."""
    rng = np.random.Generator(np.random.PCG64(1000 + F + task))
    A = random_coo(rng, 261, 190, 3500, heavy=[(7, 150), (200, 190)])
    keep = (A.row >= 3) & (A.row < 255) & (A.row != 100) & (A.row != 101)       # rows 0-2, 100-101, 255-260 are empty
    A = ref_graph.Coo(A.row[keep], A.col[keep], A.val[keep], A.shape)
    B = rng.standard_normal((190, F), dtype=np.float32)
    C0 = rng.standard_normal((261, F), dtype=np.float32)
    import spmm_cpp
    plan = make_plan(A).set_task_size(task)
    spmm_cpp.select_kernel('stream')
    try:
        for alpha, beta in ((1.0, 0.0), (0.75, -1.25)):
            want = ref_gcn.spmm_coo(A, B, C0.copy(), alpha, beta)
            C = dev(C0) if beta != 0 else torch.full((261, F), float('nan'), device='cuda')
            plan.spmm(dev(B), C, alpha, beta)
            assert_close(C.cpu().numpy(), want, TOL, f'F={F} task={task} beta={beta}')
    finally:
        spmm_cpp.select_kernel('auto')
    assert plan.device_status() == 0


def test_streaming_kernel_epilogue_and_reproducibility():
    rng = np.random.Generator(np.random.PCG64(77))
    A = random_coo(rng, 400, 300, 20000, heavy=[(0, 300), (399, 250)])
    B = rng.standard_normal((300, 256), dtype=np.float32)
    C0 = rng.standard_normal((400, 256), dtype=np.float32)
    scale = rng.uniform(0.1, 2.0, 400).astype(np.float32)
    bias = rng.standard_normal(256, dtype=np.float32)
    want = ref_gcn.spmm_epilogue(A, B, C0, 1.0, 0.5, row_scale=scale, bias=bias, relu=True)
    import spmm_cpp
    plan = make_plan(A).set_task_size(64)
    outs = []
    spmm_cpp.select_kernel('stream')
    try:
        for _ in range(3):
            C = dev(C0)
            plan.spmm(dev(B), C, 1.0, 0.5, row_scale=dev(scale), bias=dev(bias), relu=True)
            outs.append(C.cpu())
    finally:
        spmm_cpp.select_kernel('auto')
    assert_close(outs[0].numpy(), want, TOL, 'streaming epilogue')
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert plan.device_status() == 0


@pytest.mark.parametrize('m,k,nnz', [(1, 1, 1), (300, 190, 5000), (4099, 257, 1024), (5000, 100003, 70001)])
def test_plan_from_int64_ids_equals_the_int32_plan(m, k, nnz):
    """The loader's int64 block narrowed while the plan is built: same offsets, columns and census as from int32 arrays
    (with empty first and last rows, split rows, and entry counts around a CTA's share), ids beyond int32 are refused, and a
    plan built in the blocks an earlier one left behind is none the wiser."""
    import spmm_cpp
    rng = np.random.Generator(np.random.PCG64(m + k))
    A = random_coo(rng, m, k, min(nnz, m * k)) if m * k < 10**8 else ref_graph.Coo(
        np.sort(rng.integers(0, m // 50, nnz)), rng.integers(0, k, nnz), np.ones(nnz, np.float32), (m, k))
    if m > 1:
        keep = (A.row > 2) & (A.row < m - 2)
        A = ref_graph.Coo(A.row[keep], A.col[keep], A.val[keep], A.shape)
    t = torch.sparse_coo_tensor(torch.from_numpy(np.stack((A.row, A.col))), torch.from_numpy(A.val), A.shape, is_coalesced=True).cuda()
    for _ in range(2):
        wide, narrow = spmm_cpp.SpmmPlan.from_coo(t, 40, 16), make_plan(A, heavy_threshold=40, chunk=16)
        assert torch.equal(wide.col, narrow.col) and torch.equal(wide.rowptr(), narrow.rowptr()) and wide.stats() == narrow.stats()
        assert np.array_equal(wide.rowptr().numpy(), ref_graph.rowptr_of(A))
        deg = np.bincount(A.row, minlength=m)
        st = wide.stats()
        assert st['heavy_rows'] == int((deg > 40).sum()) and st['heavy_chunks'] == sum(-(-int(d) // 16) for d in deg if d > 40)
        assert st['touched_columns'] == np.unique(A.col).size and st['max_row_nnz'] == deg.max()
        B, C, D = torch.randn(k, 20, device='cuda'), torch.zeros(m, 20, device='cuda'), torch.zeros(m, 20, device='cuda')
        assert torch.equal(wide.spmm(B, C, 1.0, 0.0), narrow.spmm(B, D, 1.0, 0.0))
        del wide, narrow
    row, col = torch.zeros(1, dtype=torch.int64, device='cuda'), torch.tensor([2**32], dtype=torch.int64, device='cuda')
    out, narrowed = ctypes.c_void_p(), torch.empty(1, dtype=torch.int32, device='cuda')
    assert spmm_cpp.lib().dg_plan_create_i64(row.data_ptr(), col.data_ptr(), 1, m, k, 0, 0, narrowed.data_ptr(), None, ctypes.byref(out)) == -3
    spmm_cpp.empty_cache()


@pytest.mark.parametrize('F', [32, 41, 64, 100, 256, 260, 604])
def test_tensor_core_tiles_against_float64(F):
    """A block with a dense corner (rows of 40 to 3,000 entries, columns as skewed) whose tiles run on the tensor cores: all
    widths' panels, odd rows through the padded copy, accumulation into C, the epilogue, and the same bits every time.  The
    values span six orders of magnitude; the error is held to a tenth of the parity tolerance."""
    import spmm_cpp
    rng = np.random.Generator(np.random.PCG64(4000 + F))
    m, k = 3001, 2600
    deg = np.minimum((40 * (m / (1 + np.arange(m))) ** 0.7).astype(np.int64) + 1, 2400)
    p = 1.0 / (1 + np.arange(k)) ** 0.8
    p /= p.sum()
    row = np.repeat(rng.permutation(m), deg)
    col = np.concatenate([rng.choice(k, d, replace=False, p=p) for d in deg])
    col = rng.permutation(k)[col]
    val = (rng.standard_normal(row.size) * 10.0 ** rng.uniform(-3, 3, row.size)).astype(np.float32)
    A = ref_graph.fast_coalesce_sorted(row.astype(np.int64), col.astype(np.int64), val, (m, k))
    plan = make_plan(A)
    keep = spmm_cpp.TILE_NNZ
    try:
        spmm_cpp.TILE_NNZ = 0
        plan.tile()
    finally:
        spmm_cpp.TILE_NNZ = keep
    assert plan.tiled_entries() > A.nnz // 8
    B = torch.randn(k, F, device='cuda', generator=torch.Generator(device='cuda').manual_seed(F))
    C0 = torch.randn(m, F, device='cuda', generator=torch.Generator(device='cuda').manual_seed(F + 1))
    dense = torch.zeros(m, k, dtype=torch.float64, device='cuda')
    dense[torch.from_numpy(A.row).cuda(), torch.from_numpy(A.col).cuda()] = dev(A.val).double()
    want = (dense @ B.double()).cpu().numpy()
    C = plan.spmm(B, torch.full((m, F), float('nan'), device='cuda'), 1.0, 0.0)
    assert plan.device_status() == 0
    assert_close(C.cpu().numpy(), want, TOL / 10, 'tiles, beta = 0')
    plain = make_plan(A).spmm(B, torch.empty_like(C), 1.0, 0.0)
    err = lambda t: np.linalg.norm(t.cpu().numpy() - want) / np.linalg.norm(want)
    assert err(C) <= 4 * err(plain) + 1e-7                         # no worse than gathering beyond rounding
    assert torch.equal(C, plan.spmm(B, torch.empty_like(C), 1.0, 0.0))
    scale = torch.rand(m, device='cuda')
    got = plan.spmm(B, C0.clone(), 0.5, -2.0, row_scale=scale, relu=True)
    full = ((0.5 * dense @ B.double() - 2.0 * C0.double()) * scale.double()[:, None]).clamp(min=0)
    assert_close(got.cpu().numpy(), full.cpu().numpy(), TOL, 'tiles with the epilogue')
    acc = plan.spmm(B, C0.clone(), 1.0, 1.0)
    assert_close(acc.cpu().numpy(), (dense @ B.double() + C0.double()).cpu().numpy(), TOL / 10, 'tiles, beta = 1')
    # other values, or the same changed in place, are gathered
    other = plan.values * 2
    assert_close(plan.spmm(B, torch.empty_like(C), 1.0, 0.0, values=other).cpu().numpy(), 2 * want, TOL / 10, 'other values')
    plan.values.mul_(3.0)
    assert_close(plan.spmm(B, torch.empty_like(C), 1.0, 0.0).cpu().numpy(), 3 * want, TOL / 10, 'values changed in place')
    assert plan.tiled_entries() == 0


@pytest.mark.parametrize('alpha,beta,epilogue', [(1.0, 1.0, False), (1.0, 1.0, True), (0.5, 1.0, False), (1.0, -2.0, False), (1.0, 0.0, False)])
@pytest.mark.parametrize('F', [3, 41, 48, 256])
def test_empty_rows(F, alpha, beta, epilogue):
    """Rows without entries, windows without any row that has one: left alone where the product adds to C, else scaled, finished or cleared."""
    rng = np.random.Generator(np.random.PCG64(F))
    A = random_coo(rng, 1001, 700, 300, heavy=[(5, 600), (999, 1)])
    keep = (A.row < 256) | (A.row > 700)
    A = ref_graph.fast_coalesce_sorted(A.row[keep], A.col[keep], A.val[keep], A.shape)
    B, C0 = rng.standard_normal((700, F), dtype=np.float32), rng.standard_normal((1001, F), dtype=np.float32)
    want = ref_gcn.spmm_coo(A, B, C0.copy(), alpha, beta)
    options = {}
    if epilogue:
        scale, bias = rng.random(1001, dtype=np.float32), rng.standard_normal(F, dtype=np.float32)
        want = np.maximum(want * scale[:, None] + bias, 0)
        options = dict(row_scale=dev(scale), bias=dev(bias), relu=True)
    got = make_plan(A).spmm(dev(B), dev(C0), alpha, beta, **options).cpu().numpy()
    assert_close(got, want, TOL, f'F={F}')
    if (alpha, beta, epilogue) == (1.0, 1.0, False):
        empty = np.setdiff1d(np.arange(1001), A.row)
        assert np.array_equal(got[empty], C0[empty])


@pytest.mark.parametrize('where', [0, -1])
@pytest.mark.parametrize('F', [1, 41, 100, 256])
def test_checked_product_writes_nothing_for_other_ids(F, where):
    """The product behind the id check, through the C ABI: the plan's own ids, then lists that differ in one entry - C untouched -
    and the plan still works afterwards."""
    import spmm_cpp
    rng = np.random.Generator(np.random.PCG64(700 + F))
    A = random_coo(rng, 500, 333, 4000, heavy=[(17, 300), (499, 90)])
    plan = make_plan(A)
    row, col, val = dev(A.row, torch.int32), dev(A.col, torch.int32), plan.values
    other = col.clone()
    other[where] += 1
    B, C0 = rng.standard_normal((333, F), dtype=np.float32), rng.standard_normal((500, F), dtype=np.float32)
    want = ref_gcn.spmm_coo(A, B, C0.copy(), 1.0, 1.0)
    b, same = dev(B), ctypes.c_int(-1)
    for ids, equal in ((col, 1), (other, 0), (col, 1)):
        C = dev(C0)
        spmm_cpp.check(spmm_cpp.lib().dg_spmm_csr_checked(plan.handle, row.data_ptr(), col.data_ptr(), row.data_ptr(), ids.data_ptr(), val.data_ptr(), b.data_ptr(),
                                                          F, C.data_ptr(), F, F, 1.0, 1.0, ctypes.byref(same), torch.cuda.current_stream().cuda_stream))
        assert same.value == equal
        got = C.cpu().numpy()
        if equal:
            assert_close(got, want, TOL, f'F={F}')
        else:
            assert np.array_equal(got, C0)


def skewed_block(seed, m=3001, k=2600):
    """Rows of 40 to 2,400 entries, columns as skewed: a block with a dense corner."""
    rng = np.random.Generator(np.random.PCG64(seed))
    deg = np.minimum((40 * (m / (1 + np.arange(m))) ** 0.7).astype(np.int64) + 1, 2400)
    p = 1.0 / (1 + np.arange(k)) ** 0.8
    row = np.repeat(rng.permutation(m), deg)
    col = np.concatenate([rng.choice(k, d, replace=False, p=p / p.sum()) for d in deg])
    val = rng.standard_normal(row.size, dtype=np.float32)
    return ref_graph.fast_coalesce_sorted(row.astype(np.int64), rng.permutation(k)[col].astype(np.int64), val, (m, k))


def tiled_plan(A):
    import spmm_cpp
    keep = spmm_cpp.TILE_NNZ
    try:
        spmm_cpp.TILE_NNZ = 0
        return make_plan(A).tile()
    finally:
        spmm_cpp.TILE_NNZ = keep


def leave_free(mib):
    """Takes all but about `mib` MiB of the device's free memory."""
    import spmm_cpp
    spmm_cpp.empty_cache()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - (mib << 20), dtype=torch.uint8, device='cuda')


def test_plan_and_scratch_beside_a_framework_that_keeps_the_whole_device():
    """PyTorch holds all but a few MiB as freed blocks: the plan, its tiles and its scratch get theirs all the same."""
    A = skewed_block(5)
    F = 1024
    B = np.random.Generator(np.random.PCG64(6)).standard_normal((2600, F), dtype=np.float32)
    b, C = dev(B), torch.empty(3001, F, device='cuda')
    held = leave_free(8)
    del held                                                       # kept by torch's cache
    assert torch.cuda.mem_get_info()[0] < 64 << 20
    plan = tiled_plan(A)
    assert plan.tiled_entries() > 0
    plan.spmm(b, C, 1.0, 0.0)
    assert plan.device_status() == 0
    assert_close(C.cpu().numpy(), ref_gcn.spmm_coo(A, B, np.zeros((3001, F), np.float32), 1.0, 0.0), TOL, 'beside a full cache')
    torch.cuda.empty_cache()


def test_product_without_memory_for_its_tiles():
    """The device is really full: the scratch of the tiles finds no room, the product gathers everything; later launches see no stale error."""
    A = skewed_block(7)
    F = 1024
    B = np.random.Generator(np.random.PCG64(8)).standard_normal((2600, F), dtype=np.float32)
    plan = tiled_plan(A)
    assert plan.tiled_entries() > 0
    b, C = dev(B), torch.empty(3001, F, device='cuda')
    partial = plan.stats()['heavy_chunks'] * F * 4 >> 20
    assert partial < 40                                            # the tiles' partial results and images take 100 MiB and more
    held = leave_free(partial + 24)
    plan.spmm(b, C, 1.0, 0.0)
    assert plan.tiled_entries() == 0
    b.add_(0)
    del held
    torch.cuda.empty_cache()
    assert_close(C.cpu().numpy(), ref_gcn.spmm_coo(A, B, np.zeros((3001, F), np.float32), 1.0, 0.0), TOL, 'without tiles')


@pytest.mark.parametrize('code', [2, -5])
def test_tile_search_that_fails_leaves_the_plan_without_tiles(monkeypatch, code):
    import spmm_cpp
    A = skewed_block(9)
    B = np.random.Generator(np.random.PCG64(10)).standard_normal((2600, 64), dtype=np.float32)
    monkeypatch.setattr(spmm_cpp.lib(), 'dg_plan_add_tiles', lambda *a: code)
    with pytest.warns(UserWarning, match='no tensor-core tiles'):
        plan = tiled_plan(A)
    assert plan.tiled_entries() == 0
    C = plan.spmm(dev(B), torch.empty(3001, 64, device='cuda'), 1.0, 0.0)
    assert_close(C.cpu().numpy(), ref_gcn.spmm_coo(A, B, np.zeros((3001, 64), np.float32), 1.0, 0.0), TOL, 'without tiles')


LARGEST = """
import sys, torch
sys.path.insert(0, sys.argv[1])
import spmm_cpp
from coo_graph import graph_utils, synthetic
n, F, seed = 4_000_000, 256, int(sys.argv[2])
A = graph_utils.sym_normalization(synthetic.rmat_edge_index(n, 256_000_000, seed, device='cuda'), n)
b = torch.randn(n, F, device='cuda', generator=torch.Generator(device='cuda').manual_seed(seed))
plan = spmm_cpp.SpmmPlan.from_coo(A)
C = plan.spmm(b, torch.empty(n, F, device='cuda'), 1.0, 0.0)
assert plan.device_status() == 0
first = plan.rowptr()
length = first[1:] - first[:-1]
rows = torch.cat((torch.topk(length, 128).indices, torch.randint(n, (256,), generator=torch.Generator().manual_seed(seed))))
col, val = A.indices()[1], A.values()
for r in rows.tolist():
    e = slice(int(first[r]), int(first[r + 1]))
    want = val[e].double() @ b[col[e]].double()
    err = float((C[r].double() - want).norm() / want.norm())
    assert err < 1e-5, (r, int(length[r]), err)
print('rows agree')
"""


@pytest.mark.parametrize('seed', [1, 2])
def test_largest_graph_in_a_fresh_process(seed):
    """4 M nodes, 260 M entries, operand and result of 4 GB: the longest rows and a sample against float64."""
    import subprocess
    import sys
    from conftest import PKG
    done = subprocess.run([sys.executable, '-c', LARGEST, PKG, str(seed)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and 'rows agree' in done.stdout, done.stdout + done.stderr[-2000:]


def test_tile_kernel_that_gives_up_is_noticed():
    """A tile kernel whose waits run out sets the word that training reads after every step; other plans' products are unharmed."""
    import spmm_cpp
    A = skewed_block(11)
    b = torch.randn(2600, 256, device='cuda')
    plan = tiled_plan(A)
    spmm_cpp.check_dense_status()
    spmm_cpp.check(spmm_cpp.lib().dg_tiles_wait_selftest(plan.handle, b.data_ptr(), 256, 256, torch.cuda.current_stream().cuda_stream))
    assert plan.device_status() != 0
    with pytest.raises(RuntimeError, match='gave up'):
        spmm_cpp.check_dense_status()
    spmm_cpp.check_dense_status()
    fresh, plain = tiled_plan(A), make_plan(A)
    C = fresh.spmm(b, torch.empty(3001, 256, device='cuda'), 1.0, 0.0)
    assert fresh.device_status() == 0
    assert_close(C.cpu().numpy(), plain.spmm(b, torch.empty_like(C), 1.0, 0.0).cpu().numpy(), TOL / 10, 'after a kernel that gave up')
    assert spmm_cpp.lib().dg_tiles_wait_selftest(plain.handle, b.data_ptr(), 256, 256, None) == -5


@pytest.mark.parametrize('bad', [float('inf'), float('-inf'), float('nan'), 3.4e38, 1e19])
@pytest.mark.parametrize('F', [41, 100, 256, 300])
def test_tiles_leave_rows_alone_that_have_no_entry_in_a_column(F, bad):
    """Infinities, NaN and numbers near the largest in the row of B of the most frequent column (and of the rarest): the bits of
    a plan without tiles, in every row; and tiles again for the next, ordinary operand."""
    A = skewed_block(13)
    plan, plain = tiled_plan(A), make_plan(A)
    assert plan.tiled_entries() > 0
    count = np.bincount(A.col, minlength=2600)
    b = torch.randn(2600, F, device='cuda', generator=torch.Generator(device='cuda').manual_seed(F))
    usual = plan.spmm(b, torch.empty(3001, F, device='cuda'), 1.0, 0.0)
    for column in (int(count.argmax()), int(count.argmin())):
        x = b.clone()
        x[column, F - 1] = bad
        for alpha, beta in ((1.0, 0.0), (1.0, 1.0)):
            C = torch.ones(3001, F, device='cuda')
            got, want = plan.spmm(x, C.clone(), alpha, beta).cpu().numpy(), plain.spmm(x, C.clone(), alpha, beta).cpu().numpy()
            if column == int(count.argmax()):
                assert np.array_equal(got, want, equal_nan=True)
            else:
                assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        if not np.isfinite(bad):
            touched = np.unique(A.row[A.col == column])
            assert np.isfinite(np.delete(got, touched, 0)).all() and not np.isfinite(got[touched, F - 1]).any()
        assert plan.device_status() == 0
    assert torch.equal(plan.spmm(b, torch.empty_like(usual), 1.0, 0.0), usual)


@pytest.mark.parametrize('bad', [float('inf'), float('nan'), 1e19])
def test_values_that_cannot_be_cut_get_no_tiles(bad):
    A = skewed_block(14)
    longest, widest = np.bincount(A.row).argmax(), np.bincount(A.col).argmax()
    A.val[np.flatnonzero((A.row == longest))[0]] = bad
    A.val[np.flatnonzero((A.col == widest))[:50]] = bad
    plan = tiled_plan(A)
    assert plan.tiled_entries() == 0
    b = torch.randn(2600, 64, device='cuda')
    assert torch.equal(plan.spmm(b, torch.zeros(3001, 64, device='cuda'), 1.0, 0.0).isnan(), make_plan(A).spmm(b, torch.zeros(3001, 64, device='cuda'), 1.0, 0.0).isnan())


@pytest.mark.parametrize('offset', [0, 1])
def test_values_changed_behind_the_plan(offset):
    """Values written through .data, one at a time and all of them, at every alignment: every product reads those in front of it."""
    import spmm_cpp
    A = skewed_block(15)
    values = torch.empty(A.nnz + 4, device='cuda')[offset:offset + A.nnz]
    values.copy_(dev(A.val))
    keep = spmm_cpp.TILE_NNZ
    try:
        spmm_cpp.TILE_NNZ = 0
        plan = spmm_cpp.SpmmPlan(dev(A.row, torch.int32), dev(A.col, torch.int32), values, *A.shape).tile()
    finally:
        spmm_cpp.TILE_NNZ = keep
    assert plan.tiled_entries() > 0
    b = torch.randn(2600, 256, device='cuda')
    product = lambda p, **kw: p.spmm(b, torch.zeros(3001, 256, device='cuda'), 1.0, 0.0, **kw)
    usual = product(plan)
    for at in (0, 1, A.nnz // 2, A.nnz - 2, A.nnz - 1):
        kept = float(values[at])
        plan.values.data[at] = kept + 1.0
        assert plan.tiled_entries() > 0
        assert torch.equal(product(plan), product(make_plan(A), values=plan.values.clone()))
        plan.values.data[at] = kept
        assert torch.equal(product(plan), usual)                   # the tiles' values again
    plan.values.data.mul_(2.0)
    assert torch.equal(product(plan), product(make_plan(A), values=plan.values.clone()))


@pytest.mark.parametrize('value_exponent,operand_exponent', [(0, -95), (0, -105), (0, -130), (-40, -55), (-50, -60), (-99, 0), (-105, 0), (60, -99)])
def test_tiles_of_small_numbers_are_as_exact_as_gathering(value_exponent, operand_exponent):
    """Whole operands and values down to the smallest normal numbers: the same error against float64 as without tiles."""
    A = skewed_block(16)
    A.val *= np.float32(2.0 ** value_exponent)
    plan, plain = tiled_plan(A), make_plan(A)
    assert (plan.tiled_entries() > 0) == (value_exponent > -100)
    b = torch.randn(2600, 64, device='cuda', generator=torch.Generator(device='cuda').manual_seed(1)) * 2.0 ** operand_exponent
    b[5] = 0.0
    dense = torch.zeros(3001, 2600, dtype=torch.float64, device='cuda')
    dense[dev(A.row), dev(A.col)] = dev(A.val).double()
    want = dense @ b.double()
    err = lambda p: float((p.spmm(b, torch.empty(3001, 64, device='cuda'), 1.0, 0.0).double() - want).norm() / want.norm())
    assert err(plan) <= 1.5 * err(plain)
    assert torch.equal(plan.spmm(torch.zeros_like(b), torch.ones_like(b[:1]).repeat(3001, 1), 1.0, 0.0), torch.zeros(3001, 64, device='cuda'))


def test_checked_products_from_several_threads():
    """Four host threads on one plan and one stream, two of them with ids that differ: their results stay as they are, every time."""
    import threading
    import spmm_cpp
    rng = np.random.Generator(np.random.PCG64(701))
    A = random_coo(rng, 500, 333, 4000, heavy=[(17, 300), (499, 90)])
    plan, F = make_plan(A), 64
    row, col = dev(A.row, torch.int32), dev(A.col, torch.int32)
    other = col.clone()
    other[-1] += 1
    b = torch.randn(333, F, device='cuda')
    want = plan.spmm(b, torch.zeros(500, F, device='cuda'), 1.0, 0.0)
    L, stream, wrong = spmm_cpp.lib(), torch.cuda.current_stream().cuda_stream, []
    results = [torch.full((500, F), 7.0, device='cuda') for _ in range(4)]
    plan.spmm(b, torch.empty_like(want), 1.0, 0.0)
    torch.cuda.synchronize()

    def work(i):
        ids, C, same = (other if i % 2 else col), results[i], ctypes.c_int(-1)
        for _ in range(300):
            rc = L.dg_spmm_csr_checked(plan.handle, row.data_ptr(), col.data_ptr(), row.data_ptr(), ids.data_ptr(), plan.values.data_ptr(), b.data_ptr(), F,
                                       C.data_ptr(), F, F, 1.0, 0.0, ctypes.byref(same), stream)
            if rc or same.value != (0 if i % 2 else 1):
                wrong.append((i, rc, same.value))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong
    for i in range(4):
        assert torch.equal(results[i], torch.full_like(want, 7.0) if i % 2 else want)


OUT_OF_HOST_MEMORY = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>
#include <cuda_runtime.h>
#include "dist_gnn_b200.h"
static long left = -1;                                   // allocations until one is refused; negative: never
void* operator new(std::size_t n)
{
    if (left >= 0 && left-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void* operator new(std::size_t n, const std::nothrow_t&) noexcept
{
    if (left >= 0 && left-- == 0) return nullptr;
    return std::malloc(n);
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
    const int m = 400, each = 300, F = 64;               // every row split, frequent columns: tiles
    std::vector<int> row, col;
    std::vector<float> val(m * each, 1.f), b(each * F, 1.f), c(m * F);
    for (int i = 0; i < m * each; ++i) row.push_back(i / each), col.push_back(i % each);
    int *d_row, *d_col;
    float *d_val, *d_b, *d_c;
    cudaMalloc(&d_row, row.size() * 4), cudaMalloc(&d_col, row.size() * 4), cudaMalloc(&d_val, row.size() * 4), cudaMalloc(&d_b, b.size() * 4), cudaMalloc(&d_c, c.size() * 4);
    cudaMemcpy(d_row, row.data(), row.size() * 4, cudaMemcpyHostToDevice), cudaMemcpy(d_col, col.data(), row.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d_val, val.data(), row.size() * 4, cudaMemcpyHostToDevice), cudaMemcpy(d_b, b.data(), b.size() * 4, cudaMemcpyHostToDevice);
    int refused = 0, tiled = 0;
    for (long after = 0; after < 60; ++after) {
        dg_plan* plan = nullptr;
        left = after;
        const int created = dg_plan_create(d_row, d_col, (int64_t)row.size(), m, each, nullptr, &plan);
        const int tiles = created == 0 ? dg_plan_add_tiles(plan, d_val, nullptr) : 0;
        const int began = dg_profile_begin();
        const int product = created == 0 ? dg_spmm_csr(plan, d_val, d_b, F, d_c, F, F, 1.f, 0.f, 0u, nullptr, nullptr, nullptr) : 0;
        const int mark = dg_mark_record(nullptr);
        left = -1;
        dg_profile out;
        const int ended = dg_profile_end(&out);
        for (int code : {created, tiles, began, product, ended})
            if (code == (int)cudaErrorMemoryAllocation) ++refused;
            else if (code != 0) return std::printf("code %d after %ld\n", code, after), 1;
        if (mark == (int)cudaErrorMemoryAllocation) ++refused;
        else if (mark < 0) return std::printf("mark %d after %ld\n", mark, after), 1;
        if (created != 0) continue;
        tiled += dg_plan_tiled_entries(plan) > 0;
        if (dg_spmm_csr(plan, d_val, d_b, F, d_c, F, F, 1.f, 0.f, 0u, nullptr, nullptr, nullptr) != 0) return std::printf("product\n"), 1;
        cudaMemcpy(c.data(), d_c, c.size() * 4, cudaMemcpyDeviceToHost);
        for (float x : c)
            if (x != (float)each) return std::printf("%f after %ld\n", x, after), 1;
        dg_plan_destroy(plan);
    }
    std::printf("refused %d tiled %d\n", refused, tiled);
    return refused > 3 && tiled > 0 ? 0 : 1;
}
"""


def test_host_allocations_that_fail_come_back_as_codes(tmp_path):
    """A program whose operator new refuses the n-th allocation, for every n that plan, tiles and product make: codes, no exception
    through the C ABI, and right products afterwards."""
    import os
    import subprocess
    from conftest import PKG, ROOT
    source, program, csrc = tmp_path / 'refuse.cpp', tmp_path / 'refuse', os.path.join(PKG, 'csrc')
    source.write_text(OUT_OF_HOST_MEMORY)
    subprocess.run(['g++', '-O1', '-std=c++17', '-I', os.path.join(ROOT, 'include'), '-I/usr/local/cuda/include', str(source), '-o', str(program), '-L', csrc,
                    '-l:libdist_gnn_b200.so', '-L/usr/local/cuda/lib64', '-lcudart', f'-Wl,-rpath,{csrc}', '-Wl,-rpath,/usr/local/cuda/lib64',
                    '-Wl,--allow-shlib-undefined'], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, (done.returncode, done.stdout, done.stderr)


@pytest.mark.parametrize('tiles,many', [(None, False), (False, False), (True, True)])
def test_caller_says_whether_a_block_is_multiplied_often(monkeypatch, tiles, many):
    """from_coo goes by the size unless its caller knows better; both ends of the size rule."""
    import spmm_cpp
    A = skewed_block(17)
    t = torch.sparse_coo_tensor(torch.from_numpy(np.stack((A.row, A.col))), torch.from_numpy(A.val), A.shape, is_coalesced=True).cuda()
    monkeypatch.setattr(spmm_cpp, 'TILE_NNZ', A.nnz)
    assert (spmm_cpp.SpmmPlan.from_coo(t, tiles=tiles).tiled_entries() > 0) == many
    monkeypatch.setattr(spmm_cpp, 'TILE_ALWAYS', A.nnz)
    assert (spmm_cpp.SpmmPlan.from_coo(t, tiles=tiles).tiled_entries() > 0) == (tiles is not False)
    monkeypatch.setattr(spmm_cpp, 'TILE_ALWAYS', A.nnz + 1)
    assert (spmm_cpp.SpmmPlan.from_coo(t, tiles=tiles).tiled_entries() > 0) == many
    monkeypatch.setattr(spmm_cpp, 'TILE_NNZ', A.nnz + 1)
    assert spmm_cpp.SpmmPlan.from_coo(t, tiles=tiles).tiled_entries() == 0


def tiled_entries_by_numpy(A, threshold):
    """How many entries lie in 128 x 32 tiles of 160 or more: rows longer than the threshold, longest first, by columns of at least six
    such entries, most frequent first; ties by id.  0 where they are fewer than an eighth of all."""
    deg = np.bincount(A.row, minlength=A.shape[0])
    long_rows = np.flatnonzero(deg > threshold)
    if long_rows.size < 128:
        return 0
    inside = deg[A.row] > threshold
    weight = np.bincount(A.col[inside], minlength=A.shape[1])
    columns = np.flatnonzero(weight >= 6)
    row_rank, col_rank = np.full(A.shape[0], -1), np.full(A.shape[1], -1)
    row_rank[long_rows[np.argsort(-deg[long_rows], kind='stable')]] = np.arange(long_rows.size)
    col_rank[columns[np.argsort(-weight[columns], kind='stable')]] = np.arange(columns.size)
    r, c = row_rank[A.row], col_rank[A.col]
    both = (r >= 0) & (c >= 0)
    tiles = np.bincount(r[both] // 128 * (columns.size // 32 + 1) + c[both] // 32)
    entries = int(tiles[tiles >= 160].sum())
    return entries if columns.size >= 32 and entries >= A.nnz // 8 else 0


@pytest.mark.parametrize('rows', [127, 128, 129, 2047, 2048, 2049, 4200])
@pytest.mark.parametrize('columns', [80, 96, 97, 700, 9001])
def test_tile_search_finds_what_numpy_finds(rows, columns):
    """Lists around the edges of a sort's block and of a tile, with many equal lengths and weights; product and its bits on a second plan."""
    rng = np.random.Generator(np.random.PCG64(rows * 10000 + columns))
    length = 65 + rng.integers(0, 12, rows)
    p = 1.0 / (1 + np.arange(columns)) ** 0.9
    col = np.concatenate([np.sort(rng.choice(columns, n, replace=False, p=p / p.sum())) for n in length])
    A = ref_graph.Coo(np.repeat(np.arange(rows), length), col, rng.standard_normal(length.sum(), dtype=np.float32), (rows, columns))
    plan = tiled_plan(A)
    assert plan.stats()['heavy_threshold'] == 64 and plan.tiled_entries() == tiled_entries_by_numpy(A, 64)
    B = rng.standard_normal((columns, 72), dtype=np.float32)
    C = plan.spmm(dev(B), torch.empty(rows, 72, device='cuda'), 1.0, 0.0)
    want = np.zeros((rows, 72))
    np.add.at(want, A.row, A.val[:, None].astype(np.float64) * B[A.col])
    assert_close(C.cpu().numpy(), want, TOL / 10, f'{plan.tiled_entries()} tiled entries')
    assert torch.equal(C, tiled_plan(A).spmm(dev(B), torch.empty_like(C), 1.0, 0.0)) and plan.device_status() == 0


@pytest.mark.parametrize('where', [0, 63, 64, 200])
def test_entries_that_come_twice_are_both_multiplied(where):
    """A row-sorted block that was never coalesced, its repeated entry inside a chunk of a split row, across the border of two, and last;
    and one whose columns are in no order: no tiles, the product of a plan without them."""
    A = skewed_block(18)
    longest = np.bincount(A.row).argmax()
    at = np.flatnonzero(A.row == longest)[where if where < 200 else -2]
    twice = ref_graph.Coo(A.row, A.col.copy(), A.val, A.shape)
    twice.col[at + 1] = twice.col[at]
    mixed = ref_graph.Coo(A.row, A.col.copy(), A.val.copy(), A.shape)
    mixed.col[[at, at + 1]], mixed.val[[at, at + 1]] = A.col[[at + 1, at]], A.val[[at + 1, at]]
    B = np.random.Generator(np.random.PCG64(19)).standard_normal((2600, 64), dtype=np.float32)
    assert tiled_plan(A).tiled_entries() > 0
    for block in (twice, mixed):
        plan = tiled_plan(block)
        assert plan.tiled_entries() == 0
        got = plan.spmm(dev(B), torch.empty(3001, 64, device='cuda'), 1.0, 0.0).cpu().numpy()
        assert_close(got, ref_gcn.spmm_coo(block, B, np.zeros((3001, 64), np.float32), 1.0, 0.0), TOL, 'not coalesced')


def lengths_block(lengths, k, seed):
    """Rows of the given lengths with random columns, on the device: row ids, column ids, values."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    lengths = torch.as_tensor(lengths, device='cuda')
    row = torch.repeat_interleave(torch.arange(lengths.numel(), device='cuda'), lengths).to(torch.int32)
    col = torch.randint(0, k, (row.numel(),), device='cuda', generator=g, dtype=torch.int32)
    return row, col, torch.randn(row.numel(), device='cuda', generator=g)


class Exact:
    """Products of a block in float64, and the bound on a product's error: 128 roundings of the sum of the magnitudes, and of one."""

    def __init__(self, row, col, val, m, k):
        self.m, self.k = m, k
        self.sparse = torch.sparse_coo_tensor(torch.stack((row, col)).long(), val.double(), (m, k)).to_sparse_csr()
        self.magnitudes = torch.sparse_csr_tensor(self.sparse.crow_indices(), self.sparse.col_indices(), self.sparse.values().abs(), (m, k))

    def check(self, plan, b, g):
        """The product alone, added to C, and with the fused epilogue; returns the first."""
        F = b.size(1)
        c0 = torch.randn(self.m, F, device='cuda', generator=g)
        scale, bias = torch.rand(self.m, device='cuda', generator=g) + 0.5, torch.randn(F, device='cuda', generator=g)
        want, bound = torch.sparse.mm(self.sparse, b.double()), torch.sparse.mm(self.magnitudes, b.double().abs()) + c0.abs()
        close = lambda got, exact: bool(((got.double() - exact).abs() <= 128 * 2.0 ** -24 * (bound + 1)).all())
        out = plan.spmm(b, torch.empty_like(c0), 1.0, 0.0)
        assert close(out, want), (self.m, F)
        assert close(plan.spmm(b, c0.clone(), 1.0, 1.0), want + c0), (self.m, F)
        assert close(plan.spmm(b, c0.clone(), 0.5, -1.0, row_scale=scale, bias=bias, relu=True), ((0.5 * want - c0) * scale[:, None] + bias).clamp(min=0)), (self.m, F)
        return out


@pytest.mark.parametrize('nnz', [200_000, 1_100_000, 4_300_000])
def test_forms_by_size_and_width(nnz):
    """The forms that widths and the number of entries choose for an operand that the L2 holds: widths around 8 / 12 / 16 / 24 / 32 vectors and
    whole tiles, rows of 32-byte pieces read as such and the same operand one vector off them, odd widths through the padded copy, products
    added to C and the fused epilogue; rows with no entry, around the sets of 4 to 32 entries, and split ones."""
    import spmm_cpp
    edges = torch.tensor([0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 30, 31, 32, 33, 34, 35, 63, 64, 65, 66, 67, 127, 128, 129, 130, 300, 1025])
    k = 40_000
    lengths = edges.repeat(nnz // int(edges.sum()) + 1)
    row, col, val = lengths_block(lengths, k, nnz)
    m = lengths.numel()
    plan, exact = spmm_cpp.SpmmPlan(row, col, val, m, k), Exact(row, col, val, m, k)
    g = torch.Generator(device='cuda').manual_seed(7)
    for F in (33, 36, 41, 44, 48, 49, 52, 65, 68, 93, 96, 97, 100, 200, 256, 264, 320):
        b = torch.randn(k, F, device='cuda', generator=g)
        out = exact.check(plan, b, g)
        if F % 8 == 0:
            apart = torch.empty(k, F + 4, device='cuda')[:, 4:]            # rows 16 bytes off a 32-byte piece
            apart.copy_(b)
            assert torch.equal(plan.spmm(apart, torch.empty_like(out), 1.0, 0.0), out), (nnz, F)


@pytest.mark.parametrize('m,nnz,k,widths', [(100_000, 1_500_000, 40_000, (33, 36, 40, 48)), (150_000, 4_400_000, 300_000, (36, 41, 44, 48)),
                                            (150_000, 4_400_000, 750_000, (48,)), (600_000, 4_400_000, 2_000_000, (68, 93, 96)),
                                            (600_000, 4_900_000, 2_000_000, (68,))])
def test_forms_by_rows_and_operand(m, nnz, k, widths):
    """What the number of rows and the size of the operand add to that: medium matrices with many rows, operands on either side of what the
    L2 holds and of three eighths of it (rows that straddle sectors), short rows of an operand of more than four times the L2."""
    import spmm_cpp
    lengths = torch.arange(m) % (2 * nnz // m + 1)
    lengths[::1000] += 600                                        # split rows
    row, col, val = lengths_block(lengths, k, m + nnz)
    plan, exact = spmm_cpp.SpmmPlan(row, col, val, m, k), Exact(row, col, val, m, k)
    g = torch.Generator(device='cuda').manual_seed(8)
    for F in widths:
        exact.check(plan, torch.randn(k, F, device='cuda', generator=g), g)


@pytest.mark.parametrize('m', [200_000, 262_145])
@pytest.mark.parametrize('F', [72, 93, 96, 200, 256, 264, 320])
def test_tiles_beside_the_forms_of_large_matrices(F, m):
    """A block of more than 4.2 M entries with tiles, in windows of 64 and of 128 rows: whole, incomplete and several column tiles of rows of 32-byte
    pieces, thirds, the padded copy.  Then with a value that was changed without the version counter's notice, and with an operand
    element that the tiles cannot take: the launch behind the tiles gathers the split rows whole."""
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(F + m)
    k, dense_rows = 6000, 1200
    lengths = torch.full((m,), 6, device='cuda')
    mask = torch.rand(dense_rows, k, device='cuda', generator=g) < 0.45
    at = torch.randperm(m, device='cuda', generator=g)[:dense_rows].sort().values
    lengths[at] = mask.sum(1)
    row = torch.repeat_interleave(torch.arange(m, device='cuda'), lengths).to(torch.int32)
    first = lengths.cumsum(0) - lengths
    place = torch.arange(row.numel(), device='cuda') - first[row.long()]
    col = (place * 1000 + torch.randint(0, 1000, (row.numel(),), device='cuda', generator=g)).to(torch.int32)      # ascending, one of every thousand
    in_dense = torch.isin(row, at.to(torch.int32))
    col[in_dense] = mask.nonzero()[:, 1].to(torch.int32)
    val = torch.randn(row.numel(), device='cuda', generator=g)
    assert row.numel() > 4_200_000
    keep = spmm_cpp.TILE_NNZ
    try:
        spmm_cpp.TILE_NNZ = 0
        plan = spmm_cpp.SpmmPlan(row, col, val, m, k).tile()
    finally:
        spmm_cpp.TILE_NNZ = keep
    assert plan.tiled_entries() > row.numel() // 4
    b = torch.randn(k, F, device='cuda', generator=g)
    Exact(row, col, val, m, k).check(plan, b, g)
    assert plan.device_status() == 0
    b[17, F // 2] = 1e19
    Exact(row, col, val, m, k).check(plan, b, g)
    b[17, F // 2] = 1.0
    changed = int(first[at[5]]) + 1000
    val.data[changed] = 300.0
    Exact(row, col, val, m, k).check(plan, b, g)
    assert plan.device_status() == 0


def test_infinite_values_beside_short_batches():
    """Three gathers at a time do not divide a set of 32 entries: what the last step reads beyond it must not touch the row."""
    import spmm_cpp
    lengths = [31, 32, 33, 64] * 3
    row, col, val = lengths_block(lengths, 500, 3)
    first = torch.cat((torch.zeros(1, dtype=torch.long), torch.tensor(lengths).cumsum(0)[:-1])).cuda()
    val[first[4:8]] = float('inf')
    b = torch.rand(500, 256, device='cuda') + 0.5
    out = spmm_cpp.SpmmPlan(row, col, val, len(lengths), 500).spmm(b, torch.empty(len(lengths), 256, device='cuda'), 1.0, 0.0)
    assert bool(torch.isinf(out[4:8]).all()) and bool(torch.isfinite(out[:4]).all()) and bool(torch.isfinite(out[8:]).all())
