"""The distributed GCN layer and model with the surface of light_dist_gnn/models/gcn.py, running on the CUDA stage loop.

``broadcast(local_adj_parts, local_feature, tag)`` computes z = sum_s A[rank, s] @ X_s like gcn.py:16-30, but hands
the whole loop to the library (spmm_cpp.bcast_spmm): NCCL broadcasts on a side stream into two receive buffers,
hand-written SpMM kernels on the current stream, no host synchronisation.  With ``DistEnv(..., rep=c)`` the same call
runs the 1.5D schedule of 1D_CAGNET/dist_15d.py:61-106 (column-group broadcasts, then the sum of the partial z over
the replication group).  ``DistGCNLayer`` keeps the reference's forward/backward algebra (gcn.py:35-53), including
the reuse of the un-transposed row block of A in backward, which is exact only for a symmetric adjacency.

There is no CPU implementation: CPU tensors raise.
"""
import os
import weakref

import torch
import torch.nn as nn
import torch.nn.functional as F

import spmm_cpp
from dist_utils import DistEnv, schedule


def spmm(A, B, C):
    """C += A @ B in place for a sparse COO block A (the binding of gcn.py:9-13, on a cached plan)."""
    spmm_cpp.plan_for(A).spmm(B, C, 1.0, 1.0)
    return C


# How the dense transforms around the SpMM (torch.mm at gcn.py:41, :49-50) are computed:
#   'fp32'    plain fp32 library GEMM (CUDA cores), bit-for-bit what the reference's torch.mm does on a GPU
#   'tcgen05' the library's own tensor-core kernel (dg_dense_nt): three TF32 passes on head/tail splits, fp32 accumulator
#             in tensor memory, the tall operands split inside the kernel (dg_dense_nt for Z*W and AG*W^T, dg_dense_tn
#             for the weight gradient X^T*AG; results wider than 256 in panels, odd row strides on padded copies)
#   '3xtf32'  each fp32 operand is cut into a TF32-exact head and its residual, and the product is accumulated in fp32
#             from three tensor-core TF32 GEMMs  head*head + head*tail + tail*head  (the tail*tail term, 2^-22 relative,
#             is dropped).  About 5e-7 relative error per product - inside the 1e-5 parity bound - at a fraction of the
#             CUDA-core time, because these skinny GEMMs are then bound by reading the activations.
DENSE_MODE = os.environ.get('DIST_GNN_DENSE', 'tcgen05')
PAD_ODD_WIDTHS = os.environ.get('DIST_GNN_PAD_WIDTHS', '1') != '0'
FUSE_RELU = os.environ.get('DIST_GNN_FUSE_RELU', '1') != '0'


_padded_rows = {}


def _rows(t, keep=False):
    """t itself when its rows are dense and start on 16-byte boundaries (a column slice of a padded buffer is fine), else
    the first t.size(1) columns of a copy whose rows are padded to a multiple of 4 floats.  keep=True caches that copy for
    as long as t lives and is not modified in place (the input features: 602 floats per row -> 604); a stream that did not
    make it waits until it has been made (a captured one cannot: captures begin on an idle device)."""
    if t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 4 == 0 and t.stride(0) >= t.size(1) and t.data_ptr() % 16 == 0:
        return t
    if keep:
        hit = _padded_rows.get(id(t))
        if hit is not None and hit[0]() is t and hit[1] == t._version:
            _, _, view, stream, made = hit
            if made is not None and stream != spmm_cpp.current_stream(t) and not torch.cuda.is_current_stream_capturing():
                now = torch.cuda.current_stream(t.device)
                now.wait_event(made)
                view.record_stream(now)
            return view
    rows, cols = t.shape
    wide = torch.empty((rows, cols + (-cols) % 4), dtype=t.dtype, device=t.device)
    view = _pad_into(t, wide)[:, :cols]
    if keep and not (t.is_cuda and torch.cuda.is_current_stream_capturing()):      # a captured copy is not made before the graph runs
        key, stream, made = id(t), None, None
        if t.is_cuda:
            stream, made = spmm_cpp.current_stream(t), torch.cuda.Event()
            made.record(torch.cuda.current_stream(t.device))
        _padded_rows[key] = (weakref.ref(t, lambda _r, key=key: _padded_rows.pop(key, None)), t._version, view, stream, made)
    return view


def _pad_into(t, wide):
    """wide's first columns become t, the rest zero: one launch for fp32 rows on a GPU."""
    if t.is_cuda and t.dtype == torch.float32 and wide.size(1) % 4 == 0:
        if t.size(1) > 1 and t.stride(1) != 1 or t.stride(0) < t.size(1):
            t = t.contiguous()
        return spmm_cpp.pad_rows(t, wide)
    wide[:, :t.size(1)] = t
    wide[:, t.size(1):] = 0
    return wide


def _tf32_split(x):
    head = (x.contiguous().view(torch.int32) & -8192).view(torch.float32)    # sign, exponent, top 10 mantissa bits
    return head, x - head


def dense_mm(a, b, ta=False, tb=False, relu=False, mask=None, weight_key=None, constant_a=False):
    """op(a) @ op(b) for fp32 CUDA matrices according to DENSE_MODE; ta / tb transpose the operand.
    relu applies max(x, 0) to the product; mask (same shape as the product) zeroes it where mask <= 0.  Both are fused
    into the tensor-core kernel's epilogue and are separate passes on the library paths.  weight_key: the weight object
    behind b, which lets the tensor-core path keep its transposed, split copy until the weight changes; constant_a: a is
    an input that never changes (its padded copy, if it needs one, is kept)."""
    if DENSE_MODE == 'tcgen05' and a.is_cuda and not ta:
        # hand-written tensor-core kernel: a [M x K] times a small matrix; shapes it does not take fall through
        out = spmm_cpp.dense_nt(_rows(a), b, transposed=not tb, relu=relu, mask=_rows(mask) if mask is not None else None,
                                cache_key=weight_key)
        if out is not None:
            return out
    if DENSE_MODE == 'tcgen05' and a.is_cuda and ta and not tb and not relu and mask is None:
        out = spmm_cpp.dense_tn(_rows(a, keep=constant_a), _rows(b))         # a^T @ b with the reduction over the shared rows
        if out is not None:
            return out
    out = _library_mm(a, b, ta, tb)
    if relu:
        out = out.relu_()
    if mask is not None:
        out = out.mul_(mask > 0)
    return out


def _library_mm(a, b, ta, tb):
    if DENSE_MODE != '3xtf32' or not a.is_cuda:
        return torch.mm(a.t() if ta else a, b.t() if tb else b)
    (ah, at), (bh, bt) = _tf32_split(a), _tf32_split(b)
    if ta:
        ah, at = ah.t(), at.t()
    if tb:
        bh, bt = bh.t(), bt.t()
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        out = torch.mm(ah, bh)
        out.addmm_(ah, bt)
        out.addmm_(at, bh)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = prev
    return out


def broadcast(local_adj_parts, local_feature, tag):
    return _distributed_spmm(local_adj_parts, local_feature)


def _distributed_spmm(local_adj_parts, local_feature, constant=False):
    """z = sum over the stages of A[rank, s] X_s.  constant: the operand is an input that never changes (where its rows
    have to be padded, the padded copy is kept)."""
    env = DistEnv.env
    if not local_feature.is_cuda:
        raise RuntimeError('the broadcast-SpMM stage loop runs on CUDA tensors only; there is no CPU path')
    if env.col_comm is None:
        return _local_products(env, local_adj_parts, local_feature, constant)
    x = local_feature.contiguous()
    true_width = x.size(1)
    if true_width % 4 and PAD_ODD_WIDTHS:
        # Rows that are not a whole number of 16-byte pieces (47 classes = 188 bytes) cannot be moved with 128-bit loads
        # and start at odd offsets.  The stage loop then runs on a copy whose rows are padded with zero columns to the
        # next multiple of 4; the caller gets the first true_width columns of the wider result.
        x = _pad_into(x, env.recv_buffers(x.size(0), true_width + (-true_width) % 4, nbuf=1, tag='padded')[0])
    z = torch.empty_like(x)
    _stage_loop(env, local_adj_parts, x, z, env.stages(), env.col_comm)
    return z if z.size(1) == true_width else z[:, :true_width]


def _product_operand(env, t, constant):
    """t [n x w] as an operand whose rows are whole 16-byte pieces, [n x pad4(w)]: t itself wherever it lies (any row stride
    of whole pieces; the columns beyond w are read and their results dropped), else a padded copy as above."""
    n, true_width = t.shape
    width = true_width + (-true_width) % 4 if PAD_ODD_WIDTHS else true_width
    if spmm_cpp.binding().readable_padded(t, width):
        return t if width == true_width else t.as_strided((n, width), (t.stride(0), 1))
    if width == true_width:
        return t.contiguous()
    if constant:
        kept = _rows(t, keep=True)
        return kept.as_strided((n, width), (kept.stride(0), 1))
    return _pad_into(t, torch.empty((n, width), dtype=torch.float32, device=t.device))


def _local_products(env, adj_parts, t, constant):
    """The stage loop of a rank without peers: its own products, straight on the operand.  No communicator, no buffers, no
    argument tables: on small graphs the host's share of a step is what a step costs."""
    x = _product_operand(env, t, constant)
    z = torch.empty(x.shape, dtype=torch.float32, device=t.device)
    with env.timer.timing_cuda('broadcast+spmm'):
        beta = 0.0
        for st in env.stages():
            spmm_cpp.plan_for(adj_parts[st.part]).spmm(x, z, 1.0, beta)
            beta = 1.0
    return z if x.size(1) == t.size(1) else z[:, :t.size(1)]


def _stage_loop(env, local_adj_parts, x, z, stages, comm, timed=False):
    """z <- sum over the stages of A[rank, s] @ X_s by the schedule env.stage_order names (timed: leave per-product event
    pairs behind for Comm.last_times)."""
    n, width = x.shape
    if comm is not None and env.stage_order == 'feature_chunks' and env.rep == 1:
        # 1D only: pipeline along the feature dimension (all-gather of column chunks, full-length rows per product)
        plan = group_plans(local_adj_parts, [st.part for st in stages], len(stages))[0]
        widths = spmm_cpp.chunk_widths(width, env.chunk_width)
        pack = env.recv_buffers(n, max(widths), nbuf=2, tag='pack')
        area = env.recv_buffers(n * comm.size, max(widths), nbuf=2, tag='area')
        with env.timer.timing_cuda('broadcast+spmm'):
            spmm_cpp.allgather_spmm(comm, plan, x, pack, area, z, widths, timed=timed)
        return z
    if comm is not None and env.stage_order == 'peer_gather' and env.rep == 1 and width % 4 == 0:
        ex = compact_exchange(env, local_adj_parts, stages, owner_packs=False)
        if env.ensure_peer_buffers(n * width):
            area = env.recv_buffers(max(ex['area_rows'], 1), width, nbuf=1, tag='compact')[0]
            landing = [None] * len(ex['own']) + [area[o:o + r] for o, r in zip(ex['area_offsets'], ex['stage_rows'])]
            products = [(spmm_cpp.plan_for(local_adj_parts[stages[i].part]), x, -1) for i in ex['own']]
            products += [(plan, area[o:o + r], len(ex['own']) + last)
                         for plan, (o, r), last in zip(ex['plans'], ex['plan_slices'], ex['plan_last'])]
            with env.timer.timing_cuda('broadcast+spmm'):
                spmm_cpp.peer_spmm_gather(comm, ex['roots'], [None] * len(ex['own']) + ex['lists'], [0] * len(ex['own']) + ex['stage_rows'],
                                          landing, products, x, z, timed=timed)
            return z
    if comm is not None and env.stage_order in ('peer_compact', 'peer_gather') and env.rep == 1:
        ex = compact_exchange(env, local_adj_parts, stages)
        if env.ensure_peer_buffers(ex['send_rows'] * width):
            area = env.recv_buffers(max(ex['area_rows'], 1), width, nbuf=1, tag='compact')[0]
            landing = [None] * len(ex['own']) + [area[o:o + r] for o, r in zip(ex['area_offsets'], ex['stage_rows'])]
            products = [(spmm_cpp.plan_for(local_adj_parts[stages[i].part]), x, -1) for i in ex['own']]
            products += [(plan, area[o:o + r], len(ex['own']) + last)
                         for plan, (o, r), last in zip(ex['plans'], ex['plan_slices'], ex['plan_last'])]
            zeros = [0] * len(ex['own'])
            with env.timer.timing_cuda('broadcast+spmm'):
                spmm_cpp.peer_spmm_packed(comm, ex['packs'], ex['roots'], zeros + ex['stage_offsets'], zeros + ex['stage_rows'], landing,
                                          products, x, z, timed=timed)
            return z
    if comm is not None and env.stage_order in ('peer_copy', 'peer_compact', 'peer_gather') and env.ensure_peer_buffers(n * width):
        with env.timer.timing_cuda('broadcast+spmm'):
            spmm_cpp.peer_spmm(comm, *ordered_products(env, local_adj_parts, stages, x, rotate=True), x, z, row_comm=env.row_comm,
                               timed=timed)
        return z
    if comm is not None and env.stage_order == 'local_first':
        with env.timer.timing_cuda('broadcast+spmm'):
            spmm_cpp.bcast_spmm_ordered(comm, *ordered_products(env, local_adj_parts, stages, x), x, z,
                                        row_comm=env.row_comm, bcast_group=env.group_k, timed=timed)
        return z
    group = min(env.group_k, len(stages)) if comm is not None else 1
    plans = group_plans(local_adj_parts, [st.part for st in stages], group)
    recv = env.recv_buffers(n * group, width) if comm is not None else None
    with env.timer.timing_cuda('broadcast+spmm'):
        spmm_cpp.bcast_spmm(comm, [st.root_in_group for st in stages], plans, x, recv, z, row_comm=env.row_comm, group=group,
                            timed=timed)
    return z


_compact_cache = {}


def group_sizes(count, spec):
    """How `count` remote arrivals are shared out over the products of a 'peer_compact' loop.  spec: an int k (groups of k,
    the last one takes what is left) or a sequence of sizes (used in order, the last size repeats)."""
    if isinstance(spec, int):
        spec = [spec]
    spec = [max(1, int(v)) for v in spec] or [1]
    sizes, i = [], 0
    while count > 0:
        take = min(count, spec[min(i, len(spec) - 1)])
        sizes.append(take)
        count -= take
        i += 1
    return sizes


def compact_exchange(env, adj_parts, stages, owner_packs=True):
    """One-off set-up of the stage orders that move only the operand rows a block touches (1D).  For every remote block:
    the sorted list of the columns it touches and the block with its column ids replaced by positions in that list.  The
    pulled rows land side by side in one area in pull order, and env.stage_group consecutive arrivals are multiplied by
    ONE product over their joined block (column id = position inside the group's slice of the area): fewer
    read-modify-write passes over the result and longer rows, at the price of waiting for the group's last arrival.

    owner_packs=True ('peer_compact'): the lists are exchanged once (an all-gather of host objects over the column
    communicator's ranks), every owner then packs, per distributed SpMM, each reader's rows into its send buffer and the
    reader pulls its list with one copy: this call also returns where this rank's rows start inside each owner's buffer
    and which rows this rank packs for every reader.
    owner_packs=False ('peer_gather'): nothing is exchanged; the reader gathers its rows out of the owner's whole block
    itself, so all it needs are its own lists (kept on the device)."""
    import torch.distributed as dist
    key = (id(adj_parts), tuple(group_sizes(len(stages), env.stage_group)), bool(owner_packs))
    hit = _compact_cache.get(key)
    if hit is not None and hit[0] is adj_parts:
        return hit[1]
    comm = env.col_comm
    me, size = comm.rank, comm.size
    own, remote = schedule.pull_order(stages, me, size)
    n = adj_parts[0].size(0)
    wanted, blocks, kept, lists = {}, [], [], []
    for i in remote:
        block = adj_parts[stages[i].part]
        idx = block.indices()
        if idx.size(1) == 0:
            continue                                                  # an empty block adds nothing: no list, no copy, no product
        touched = torch.unique(idx[1])                                # ascending
        blocks.append((idx[0], torch.searchsorted(touched, idx[1].contiguous()), block.values(), touched.numel()))
        if owner_packs:
            wanted[stages[i].root_in_group] = touched.to(torch.int32).cpu().numpy()
        else:
            lists.append(touched.to(torch.int32).contiguous())
        kept.append(i)
    if owner_packs:
        gathered = [None] * size
        dist.all_gather_object(gathered, wanted, group=env.world_group)   # gathered[q][s]: rows of block s that reader q needs
        lay = schedule.compact_layout(gathered, me, [stages[i].root_in_group for i in kept])
        for q, _ in lay['packs']:                                         # the rows a reader asks for must exist in this rank's block
            ids = gathered[q][me]
            if len(ids) and (int(ids.min()) < 0 or int(ids.max()) >= n):
                raise RuntimeError(f'rank {q} asked rank {me} for rows outside its block of {n} rows')
        packs = [(torch.from_numpy(gathered[q][me]).to(env.device), offset) for q, offset in lay['packs']]
    else:
        stage_rows = [b[3] for b in blocks]
        offsets = [sum(stage_rows[:j]) for j in range(len(stage_rows))]
        lay = dict(stage_rows=stage_rows, area_offsets=offsets, area_rows=sum(stage_rows), stage_offsets=[0] * len(stage_rows),
                   send_rows=n, sizes=None)
        packs = []
    plans, plan_slices, plan_last = [], [], []
    first = 0
    for count in group_sizes(len(kept), env.stage_group):
        row, col, val, rows_total = schedule.join_packed_blocks(blocks, lay['area_offsets'], first, count)
        plans.append(spmm_cpp.SpmmPlan(row.to(torch.int32), col.to(torch.int32).contiguous(), val.contiguous(), n, rows_total).tile())
        plan_slices.append((lay['area_offsets'][first], rows_total))
        plan_last.append(first + count - 1)
        first += count
    ex = dict(own=own, remote=kept, plans=plans, plan_slices=plan_slices, plan_last=plan_last, packs=packs, lists=lists,
              roots=[stages[i].root_in_group for i in own + kept],
              stage_rows=lay['stage_rows'], stage_offsets=lay['stage_offsets'], area_offsets=lay['area_offsets'],
              area_rows=lay['area_rows'], send_rows=lay['send_rows'], sizes=lay['sizes'])
    _compact_cache[key] = (adj_parts, ex)
    return ex


def ordered_products(env, adj_parts, stages, x, rotate=False):
    """Arguments (roots, landing, products) of spmm_cpp.bcast_spmm_ordered / peer_spmm for the stage orders that multiply
    this rank's own block first, straight from x: the remote blocks land side by side in one receive area, in transfer
    order, and are multiplied env.stage_group at a time as they arrive.
    rotate=False: transfers in schedule order, the same on every rank (collective broadcasts need that).
    rotate=True:  each rank lists its own stages first and then the remote ones starting with the rank after itself, so
                  that at any moment every send buffer serves one reader (peer copies need no common order)."""
    me, size = env.col_comm.rank, env.col_comm.size
    n, width = x.shape
    if rotate:
        own, remote = schedule.pull_order(stages, me, size)
    else:
        remote = [i for i, st in enumerate(stages) if st.root_in_group != me]
        own = [i for i, st in enumerate(stages) if st.root_in_group == me]
    area = env.recv_buffers(max(len(remote), 1) * n, width, nbuf=1)[0]
    issue = own + remote if rotate else list(range(len(stages)))        # the order the transfers are listed in
    position = {i: pos for pos, i in enumerate(issue)}
    landing = [None] * len(stages)
    for pos, i in enumerate(remote):
        landing[position[i]] = area[pos * n:(pos + 1) * n]
    products = [(spmm_cpp.plan_for(adj_parts[stages[i].part]), x, -1) for i in own]
    group = max(1, min(env.group_k, len(remote)))
    plans = group_plans(adj_parts, [stages[i].part for i in remote], group) if remote else []
    for g, plan in enumerate(plans):
        members = remote[g * group:(g + 1) * group]
        products.append((plan, area[g * group * n:(g * group + len(members)) * n], max(position[i] for i in members)))
    return [stages[i].root_in_group for i in issue], landing, products


_group_plan_cache = {}


def drop_cached_plans():
    """Forgets the joined plans and exchange tables kept per graph (they hold the graph's blocks alive)."""
    _compact_cache.clear()
    _group_plan_cache.clear()


def group_plans(adj_parts, parts, group):
    """Plans of the stage loop's products.  group = 1: one per column block, as the reference multiplies them.
    group = k: the blocks of k consecutive stages are joined side by side into one n x (k*n) block (entries stay in
    ascending (stage, column) order inside every row, so the sum order of the stage-by-stage loop is kept)."""
    if group == 1:
        return [spmm_cpp.plan_for(adj_parts[p]) for p in parts]
    key = (id(adj_parts), tuple(parts), group)
    hit = _group_plan_cache.get(key)
    if hit is not None and hit[0] is adj_parts:
        return hit[1]
    plans = []
    for g0 in range(0, len(parts), group):
        blocks = [adj_parts[p] for p in parts[g0:g0 + group]]
        n = blocks[0].size(0)
        offsets, total = [], 0
        for b in blocks:
            offsets.append(total)
            total += b.size(1)
        row = torch.cat([b.indices()[0] for b in blocks])
        col = torch.cat([b.indices()[1] + off for b, off in zip(blocks, offsets)])
        val = torch.cat([b.values() for b in blocks])
        order = torch.sort(row * total + col).indices
        plans.append(spmm_cpp.SpmmPlan(row[order].to(torch.int32), col[order].to(torch.int32), val[order].contiguous(), n, total).tile())
    _group_plan_cache[key] = (adj_parts, plans)
    return plans


def _all_reduce(t):
    env = DistEnv.env
    if env.world_size == 1:
        env.timer.empty_region('all_reduce')
        return
    with env.timer.timing_cuda('all_reduce'):
        env.all_reduce_sum(t)


class DistGCNLayer(torch.autograd.Function):
    """forward(features, weight, adj_parts, tag) as in the reference (gcn.py:35-53).  Optional flags let GCN fuse the
    ReLU between two layers into the dense kernels instead of running it (and its backward) as separate passes:

    relu            the layer returns max(out, 0).  Its backward then expects a grad_output that is ALREADY zero where
                    the returned activation is zero - which is what the next layer delivers when it is called with
    input_is_relu   this layer's input is such an activation: the gradient it returns for the input is zeroed where
                    the input is <= 0 (the ReLU's backward, applied in the epilogue of AG * W^T).
    Used as a pair they compute exactly  relu(layer(x))  and its gradient; one without the other does not.

    product         a precomputed  sum_s A[rank, s] X_s  for these very features (GCN's cache of the first layer's
                    product, whose operand never changes): the stage loop of the forward pass is skipped.
    shortcut        only with `product`, and only when the input needs no gradient: the weight gradient is taken as
                    product^T * grad_output instead of X^T * (A * grad_output), which skips the backward stage loop too.
                    Summed over the ranks the two are the same matrix when A is symmetric - the assumption the reference
                    already makes by multiplying with the un-transposed row block in backward (gcn.py:47) - but each
                    rank's term, and the rounding, differ.
    transform_first for a layer without ReLU whose output is narrower than its input (the last one: 256 -> 47), compute
                    A (X W) instead of (A X) W: the stage loop then runs at the output width.  Same result up to rounding,
                    same backward pass.
    constant_input  the features are the network's input, which stays as it is from step to step: where its rows have to be
                    padded, the padded copy is kept until the tensor is modified."""

    @staticmethod
    def forward(ctx, features, weight, adj_parts, tag, relu=False, input_is_relu=False, product=None, shortcut=False,
                transform_first=False, constant_input=False):
        ctx.adj_parts, ctx.tag, ctx.input_is_relu = adj_parts, tag, input_is_relu
        ctx.weight_key = weight                      # the caller's tensor object: key of the split-weight cache
        ctx.shortcut = bool(shortcut and product is not None)
        if transform_first and product is None and not relu and weight.size(1) < features.size(1):
            # A (X W) instead of (A X) W: the same matrix up to rounding, with the distributed SpMM at the narrower output
            # width.  The backward pass below is unchanged: AG = A G, dX = AG W^T and dW = X^T AG are what both orders need.
            ctx.save_for_backward(features, weight)
            with DistEnv.env.timer.timing_cuda('mm'):
                y = dense_mm(features, weight, weight_key=weight)
            return broadcast(adj_parts, y, 'Forward' + tag)
        z_local = product if product is not None else _distributed_spmm(adj_parts, features, constant_input)
        ctx.save_for_backward(z_local if ctx.shortcut else features, weight)
        with DistEnv.env.timer.timing_cuda('mm'):
            z_local = dense_mm(z_local, weight, relu=relu, weight_key=weight)
        return z_local

    @staticmethod
    def backward(ctx, grad_output):
        features, weight = ctx.saved_tensors
        if ctx.shortcut and not ctx.needs_input_grad[0]:
            with DistEnv.env.timer.timing_cuda('mm'):
                grad_weight = dense_mm(features, grad_output, ta=True, constant_a=True)      # `features` holds the saved product here
            _all_reduce(grad_weight)
            return (None, grad_weight) + (None,) * 8
        if ctx.shortcut:
            raise RuntimeError('the gradient shortcut needs an input that requires no gradient')
        ag = broadcast(ctx.adj_parts, grad_output, 'Backward' + ctx.tag)
        with DistEnv.env.timer.timing_cuda('mm'):
            grad_features = None
            if ctx.needs_input_grad[0]:
                grad_features = dense_mm(ag, weight, tb=True, mask=features if ctx.input_is_relu else None, weight_key=ctx.weight_key)
            grad_weight = dense_mm(features, ag, ta=True, constant_a=not ctx.needs_input_grad[0])
        _all_reduce(grad_weight)
        return (grad_features, grad_weight) + (None,) * 8


class GCN(nn.Module):
    """num_layers DistGCNLayers with ReLU between them, no bias (gcn.py:56-72).  Weights are drawn as the reference
    draws them - torch.rand on the host after manual_seed(0), layer by layer - unless `weights` injects them.
    The ReLUs run inside the dense kernels (FUSE_RELU); with DIST_GNN_FUSE_RELU=0 they are F.relu calls as in the
    reference.

    cache_input_product     keep the first layer's  sum_s A[rank, s] X_s  between epochs: its operand is the input
                            features, which never change (gcn.py:69 recomputes it every epoch).  Exact: the losses are
                            bit-identical to the uncached run.  The cache is dropped when a different features tensor
                            is passed in or the tensor is modified in place.
    input_gradient_shortcut with the cache, also take the first layer's weight gradient from the cached product (see
                            DistGCNLayer `shortcut`): no stage loop at all for layer 1.  Equal to the reference's
                            gradient for a symmetric adjacency up to rounding, not bit for bit.
    transform_first         the last layer multiplies by its weight before the stage loop when that is the narrower side
                            (DistGCNLayer `transform_first`): a 47-wide distributed SpMM instead of a 256-wide one.
    All are off by default: the like-for-like epoch computes what the reference computes, in its order."""

    def __init__(self, g, env, hidden_dim=16, num_layers=3, weights=None, cache_input_product=False, input_gradient_shortcut=False,
                 transform_first=False):
        super().__init__()
        self.g, self.env, self.num_layers = g, env, num_layers
        self.cache_input_product = bool(cache_input_product or input_gradient_shortcut)
        self.input_gradient_shortcut = bool(input_gradient_shortcut)
        self.transform_first = bool(transform_first)
        self._product = None        # (features tensor, its version, the cached product)
        in_dim, out_dim = g.features.size(1), g.num_classes
        dims = [in_dim] + [hidden_dim] * (num_layers - 1) + [out_dim]
        torch.manual_seed(0)
        for l in range(num_layers):
            w = torch.rand(dims[l], dims[l + 1]) if weights is None else weights[l].detach().clone().float()
            assert tuple(w.shape) == (dims[l], dims[l + 1])
            setattr(self, f'weight{l + 1}', nn.Parameter(w.to(env.device)))

    def weights(self):
        return [getattr(self, f'weight{l + 1}') for l in range(self.num_layers)]

    def input_product(self, features):
        """The cached first-layer product for `features`, computed on first use (None when caching is off or the features
        take part in autograd)."""
        if not self.cache_input_product or features.requires_grad:
            return None
        hit = self._product
        if hit is None or hit[0] is not features or hit[1] != features._version:
            with torch.no_grad():
                z = broadcast(self.g.adj_parts, features, 'ForwardL1')
                z = z.clone() if z.data_ptr() != z.untyped_storage().data_ptr() or not z.is_contiguous() else z   # own its memory
            self._product = hit = (features, features._version, z)
        return hit[2]

    def _one_rank_plan(self, features, weights):
        """The plan to run all layers on in one call, or None when a layer has to be called by itself: a rank with peers, one of
        the options above, another dense mode, an input that wants a gradient, or operands the kernels do not take."""
        env, parts = DistEnv.env, self.g.adj_parts
        if (env is None or env.world_size != 1 or len(parts) != 1 or not FUSE_RELU or not PAD_ODD_WIDTHS or DENSE_MODE != 'tcgen05'
                or self.cache_input_product or self.transform_first or not features.is_cuda or features.requires_grad
                or features.dtype != torch.float32 or features.dim() != 2 or features.size(0) < 1 or features.size(1) < 1):
            return None
        width = features.size(1)
        for w in weights:
            if (w.device != features.device or w.dtype != torch.float32 or w.dim() != 2 or w.size(0) != width or w.size(1) < 1
                    or not w.is_contiguous()):
                return None
            width = w.size(1)
        plan = spmm_cpp.plan_for(parts[0])
        return plan if plan.m == plan.k == features.size(0) and plan.device == features.device else None

    def _one_rank_forward(self, plan, features, weights):
        """All layers on a rank without peers, forward and backward, from one library call each (dg_gcn_forward,
        dg_gcn_backward behind the binding's autograd node): the products and transforms of the chained DistGCNLayers in the
        same order on the same operands, the same bits, without the host's work between them."""
        env = DistEnv.env
        plan.value_ptr()                                    # values changed in place: their tiles go first
        timer = env.timer
        out = spmm_cpp.binding().gcn(plan.ref, features, _product_operand(env, features, True), weights, timer.ident)
        timer.bound_regions()
        return out

    def forward(self, features):
        h = features
        last = self.num_layers - 1
        weights = self.weights()
        plan = self._one_rank_plan(features, weights)
        if plan is not None:
            return self._one_rank_forward(plan, features, weights)
        for l, w in enumerate(weights):
            product = self.input_product(h) if l == 0 else None
            shortcut = self.input_gradient_shortcut and product is not None
            if FUSE_RELU:
                h = DistGCNLayer.apply(h, w, self.g.adj_parts, f'L{l + 1}', l < last, l > 0, product, shortcut, self.transform_first, l == 0)
            else:
                h = DistGCNLayer.apply(h, w, self.g.adj_parts, f'L{l + 1}', False, False, product, shortcut,
                                       self.transform_first and l == last, l == 0)
                if l < last:
                    h = F.relu(h)
        return h
