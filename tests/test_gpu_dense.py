"""The tcgen05 dense transform (three TF32 passes, fp32 accumulation in tensor memory) against float64.  Needs a GPU."""
import numpy as np
import pytest
import torch

from conftest import assert_close

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize('M,K,N', [(128, 32, 16), (128, 256, 256), (1000, 256, 256), (300, 100, 256), (129, 256, 47),
                                   (5000, 32, 16), (77, 8, 8), (4096, 256, 128), (513, 100, 47), (400000, 256, 256)])
def test_dense_nt_matches_float64(M, K, N):
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    a = torch.randn(M, K, device='cuda', generator=g)
    bt = torch.randn(N, K, device='cuda', generator=g)
    c = spmm_cpp.dense_nt(a, bt)
    assert c is not None and c.shape == (M, N)
    want = a.double() @ bt.double().t()
    assert_close(c.cpu().numpy(), want.cpu().numpy(), TOL, f'{M}x{K}x{N}')
    r = spmm_cpp.dense_nt(a, bt, relu=True)
    assert_close(r.cpu().numpy(), want.clamp(min=0).cpu().numpy(), TOL, f'relu {M}x{K}x{N}')
    assert spmm_cpp.dense_status() == 0


def test_dense_split_is_exact_and_unsupported_shapes_fall_back():
    import spmm_cpp
    w = torch.randn(64, 48, device='cuda')
    head, tail = spmm_cpp.dense_split(w)
    assert torch.equal(head + tail, w)
    assert torch.equal(head.view(torch.int32) & 8191, torch.zeros_like(head, dtype=torch.int32))
    assert spmm_cpp.dense_nt(torch.randn(100, 47, device='cuda'), torch.randn(16, 47, device='cuda')) is None     # 188-byte rows


@pytest.mark.parametrize('M,K,N', [(29121, 602, 256), (1000, 64, 300), (3000, 256, 602), (515, 604, 41)])
def test_dense_nt_on_the_reddit_shaped_widths(M, K, N):
    """Config 1's layer shapes (602 -> 256 -> 41 on 29,121-row blocks): an inner dimension of 602 read from rows padded to
    604 floats, and results wider than one 256-column accumulator computed in panels."""
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    wide = torch.randn(M, K + (-K) % 4, device='cuda', generator=g)
    a = wide[:, :K]                                                # what the stage loop hands over for K = 602
    w = torch.randn(K, N, device='cuda', generator=g)              # layer weight [in x out]
    c = spmm_cpp.dense_nt(a, w, transposed=True, relu=True)
    assert c is not None and c.shape == (M, N)
    want = (a.double() @ w.double()).clamp(min=0)
    assert_close(c.cpu().numpy(), want.cpu().numpy(), TOL, f'{M}x{K}x{N}')
    # the split copy of a weight is kept until the weight changes in place
    p = torch.nn.Parameter(w.clone())
    first = spmm_cpp.dense_nt(a, p, transposed=True, cache_key=p)
    assert torch.equal(first, spmm_cpp.dense_nt(a, p, transposed=True, cache_key=p))
    with torch.no_grad():
        p.mul_(2.0)
    assert_close(spmm_cpp.dense_nt(a, p, transposed=True, cache_key=p).cpu().numpy(), (2 * (a.double() @ w.double())).cpu().numpy(), TOL, 'after an in-place update')
    assert spmm_cpp.dense_status() == 0


@pytest.mark.parametrize('n,Km,Nn', [(29121, 602, 256), (2000, 300, 300), (777, 256, 602), (4100, 604, 44)])
def test_dense_tn_in_panels(n, Km, Nn):
    """Weight gradients wider than two accumulators (config 1: X^T * AG with 602 input features) as 256 x 256 panels."""
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(n + Km + Nn)
    x = torch.randn(n, Km + (-Km) % 4, device='cuda', generator=g)[:, :Km]
    y = torch.randn(n, Nn + (-Nn) % 4, device='cuda', generator=g)[:, :Nn]
    d = spmm_cpp.dense_tn(x, y)
    assert d is not None and d.shape == (Km, Nn)
    assert_close(d.cpu().numpy(), (x.double().t() @ y.double()).cpu().numpy(), TOL, f'{n}x{Km}x{Nn}')
    assert torch.equal(d, spmm_cpp.dense_tn(x, y))
    assert spmm_cpp.dense_status() == 0


def test_dense_mm_pads_odd_row_strides_instead_of_leaving_the_tensor_cores():
    """models.gcn.dense_mm on operands whose rows are not 16-byte multiples (602 input features, 41 classes, contiguous):
    they are copied once into padded rows and still run on the hand-written kernels (the launch counter moves)."""
    import spmm_cpp
    from models.gcn import dense_mm
    g = torch.Generator(device='cuda').manual_seed(602)
    x = torch.randn(5000, 602, device='cuda', generator=g)
    ag = torch.randn(5000, 41, device='cuda', generator=g)
    w = torch.randn(602, 41, device='cuda', generator=g)
    before = spmm_cpp.dense_launches
    dw = dense_mm(x, ag, ta=True, constant_a=True)
    out = dense_mm(x, w)
    dx = dense_mm(ag, w, tb=True)
    assert spmm_cpp.dense_launches > before + 3
    assert_close(dw.cpu().numpy(), (x.double().t() @ ag.double()).cpu().numpy(), TOL, 'dW 602 x 41')
    assert_close(out.cpu().numpy(), (x.double() @ w.double()).cpu().numpy(), TOL, 'X W')
    assert_close(dx.cpu().numpy(), (ag.double() @ w.double().t()).cpu().numpy(), TOL, 'AG W^T, 602 wide')
    assert spmm_cpp.dense_status() == 0


def test_bounded_wait_gives_up_and_leaves_the_context_usable():
    """The dense kernels bound every mbarrier wait.  dg_dense_wait_selftest runs that path on purpose - a wait on a barrier
    nothing arrives at, with a short limit - and must report that the wait ran out, free its tensor memory and return;
    the real kernels then run as before and their status word is untouched."""
    import spmm_cpp
    assert spmm_cpp.dense_wait_selftest() is True
    a = torch.randn(300, 64, device='cuda')
    w = torch.randn(64, 32, device='cuda')
    c = spmm_cpp.dense_nt(a, w, transposed=True)                   # needs the tensor memory the self-test held
    assert_close(c.cpu().numpy(), (a.double() @ w.double()).cpu().numpy(), TOL, 'product after the self-test')
    assert spmm_cpp.dense_status() == 0
    spmm_cpp.check_dense_status()


@pytest.mark.parametrize('n,Km,Nn', [(16, 32, 16), (1000, 256, 256), (5000, 100, 256), (300, 128, 48), (70000, 256, 256),
                                     (33, 8, 8), (4099, 100, 64), (250000, 256, 128)])
def test_dense_tn_matches_float64(n, Km, Nn):
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(n + Km + Nn)
    x = torch.randn(n, Km, device='cuda', generator=g)
    y = torch.randn(n, Nn, device='cuda', generator=g)
    d = spmm_cpp.dense_tn(x, y)
    assert d is not None and d.shape == (Km, Nn)
    want = x.double().t() @ y.double()
    assert_close(d.cpu().numpy(), want.cpu().numpy(), TOL, f'{n}x{Km}x{Nn}')
    assert torch.equal(d, spmm_cpp.dense_tn(x, y))                 # partials are added in a fixed order
    assert spmm_cpp.dense_status() == 0


def test_dense_tn_error_does_not_grow_with_the_row_count():
    """All-positive operands over the full benchmark row count: the worst case for the truncating tensor-core accumulator,
    whose error without the periodic flush is 3e-4 here (and linear in the number of rows)."""
    import spmm_cpp
    n = 2449029
    g = torch.Generator(device='cuda').manual_seed(5)
    x = torch.rand(n, 256, device='cuda', generator=g)
    y = torch.rand(n, 256, device='cuda', generator=g)
    want = torch.zeros(256, 256, device='cuda', dtype=torch.float64)
    for s in range(0, n, 200000):
        want += x[s:s + 200000].double().t() @ y[s:s + 200000].double()
    d = spmm_cpp.dense_tn(x, y)
    assert_close(d.cpu().numpy(), want.cpu().numpy(), TOL, 'full-size weight gradient')
    assert spmm_cpp.dense_status() == 0


@pytest.mark.parametrize('M,N,K', [(1000, 256, 256), (777, 100, 48), (130, 47, 256)])
def test_dense_nt_mask_zeroes_where_the_activation_is_zero(M, N, K):
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(M + N)
    a = torch.randn(M, K, device='cuda', generator=g)
    bt = torch.randn(N, K, device='cuda', generator=g)
    act = torch.relu(torch.randn(M, N, device='cuda', generator=g))       # about half zeros, like a ReLU output
    out = spmm_cpp.dense_nt(a, bt, mask=act)
    plain = spmm_cpp.dense_nt(a, bt)
    assert out is not None and plain is not None
    assert torch.equal(out, plain * (act > 0))
    want = (a.double() @ bt.double().t()) * (act > 0)
    assert_close(out.cpu().numpy(), want.cpu().numpy(), TOL, f'masked {M}x{N}x{K}')
    with pytest.raises(RuntimeError):
        spmm_cpp.dense_nt(a, bt, mask=act[:, :-1])


def test_dense_kernels_take_column_slices_of_padded_buffers():
    """47 columns held in rows of 48 floats (what the stage loop returns for an odd class count): both products read the
    slice in place and ignore the padding column."""
    import spmm_cpp
    n = 20000
    g = torch.Generator(device='cuda').manual_seed(47)
    wide = torch.randn(n, 48, device='cuda', generator=g)
    ag = wide[:, :47]
    w = torch.randn(256, 47, device='cuda', generator=g)          # layer weight [in x out]: dX = AG * W^T
    h = torch.randn(n, 256, device='cuda', generator=g)
    dx = spmm_cpp.dense_nt(ag, w)
    assert dx is not None and dx.shape == (n, 256)
    assert_close(dx.cpu().numpy(), (ag.double() @ w.double().t()).cpu().numpy(), TOL, 'dX from a 47-of-48 slice')
    dw = spmm_cpp.dense_tn(h, ag)
    assert dw is not None and dw.shape == (256, 47)
    assert_close(dw.cpu().numpy(), (h.double().t() @ ag.double()).cpu().numpy(), TOL, 'dW from a 47-of-48 slice')
    with pytest.raises(RuntimeError):
        spmm_cpp.dense_tn(h, wide.t()[:47].t()[:, ::2])           # not row-major
    assert spmm_cpp.dense_status() == 0


def test_dense_tn_unsupported_shapes_fall_back():
    import spmm_cpp
    assert spmm_cpp.dense_tn(torch.randn(100, 47, device='cuda'), torch.randn(100, 16, device='cuda')) is None      # 188-byte rows


@pytest.mark.parametrize('M', [1, 127, 129, 256, 257, 19073])
@pytest.mark.parametrize('N,K', [(65, 4), (96, 16), (97, 20), (255, 36), (256, 100), (130, 8)])
def test_dense_nt_by_cta_pairs(M, N, K):
    """Results wider than 64 columns: tiles of 256 rows with a half that has few rows or none, more tiles than pairs, columns that end inside
    a 32-column piece, rows of C and of the mask that are no 16-byte multiples, depths below and beside a half slab of 16."""
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(M + 1000 * N + K)
    a = torch.randn(M, K, device='cuda', generator=g)
    bt = torch.randn(N, K, device='cuda', generator=g)
    want = a.double() @ bt.double().t()
    plain = spmm_cpp.dense_nt(a, bt)
    assert_close(plain.cpu().numpy(), want.cpu().numpy(), TOL, f'{M}x{N}x{K}')
    assert torch.equal(spmm_cpp.dense_nt(a, bt, relu=True), plain.clamp(min=0))
    act = torch.relu(torch.randn(M, N, device='cuda', generator=g))
    assert torch.equal(spmm_cpp.dense_nt(a, bt, mask=act), plain * (act > 0))
    wide = torch.nn.functional.pad(act, (0, (-N) % 4))[:, :N]
    assert torch.equal(spmm_cpp.dense_nt(a, bt, mask=wide), plain * (act > 0))
    assert spmm_cpp.dense_status() == 0


@pytest.mark.parametrize('K', [16, 64, 100, 192, 196, 256, 604])
@pytest.mark.parametrize('N', [64, 65, 80, 81, 96, 128, 129])
def test_dense_nt_rows_do_not_depend_on_the_kernel(N, K):
    """One tile per CTA or CTA pairs, by rows, columns, depth and mask: on either side of every limit a row is the same bits."""
    import spmm_cpp
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    counts = [128 * sms, 128 * sms + 1, 256 * sms, 256 * sms + 1]
    g = torch.Generator(device='cuda').manual_seed(1000 * N + K)
    a = torch.randn(counts[-1], K, device='cuda', generator=g)
    bt = torch.randn(N, K, device='cuda', generator=g)
    act = torch.randn(counts[-1], N, device='cuda', generator=g)
    plain, masked = spmm_cpp.dense_nt(a, bt), spmm_cpp.dense_nt(a, bt, mask=act)
    assert_close(plain.cpu().numpy(), (a.double() @ bt.double().t()).cpu().numpy(), TOL, f'{N}x{K}')
    assert torch.equal(masked, plain * (act > 0))
    for M in counts[:-1]:
        assert torch.equal(spmm_cpp.dense_nt(a[:M], bt), plain[:M]) and torch.equal(spmm_cpp.dense_nt(a[:M], bt, mask=act[:M]), masked[:M])
    assert spmm_cpp.dense_status() == 0


@pytest.mark.parametrize('n', [1, 15, 17, 257, 4096 + 5, 148 * 256 + 1])
@pytest.mark.parametrize('Km,Nn', [(129, 130), (256, 193), (256, 128), (128, 256), (10, 200), (200, 5), (1, 40), (96, 96)])
@pytest.mark.parametrize('ctas', [1, 5, 148])
def test_dense_tn_roles_and_ranges(n, Km, Nn, ctas):
    """Either operand along the rows of the MMAs, alone or by CTA pairs; ranges without rows, an odd number of them for the last pair, fewer
    rows than a slab, several flushes in a range; the scratch exactly as large as documented, with a guard behind it.  An element's error
    goes with sqrt(n) (1.2e-6 of it; TOL leaves 8 times that), so results are compared over at least 40 elements: one that cancels to a
    fourteenth of sqrt(n) is 1.6e-5 off by itself."""
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(n + 1000 * Km + Nn)
    x = torch.randn(n, Km + (-Km) % 4, device='cuda', generator=g)
    y = torch.randn(n, Nn + (-Nn) % 4, device='cuda', generator=g)
    need = min(ctas, (n + 15) // 16) * (-(-Km // 128) * 128) * (-(-Nn // 16) * 16)
    scratch = torch.full((need + 1024,), 3.5, device='cuda')
    d = torch.full((Km, Nn + 3), -1.0, device='cuda')
    spmm_cpp.check(spmm_cpp.lib().dg_dense_tn(x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), d.data_ptr(), Nn + 3, n, Km, Nn, scratch.data_ptr(), need,
                                              ctas, spmm_cpp._stream()))
    assert_close(d[:, :Nn].cpu().numpy(), (x[:, :Km].double().t() @ y[:, :Nn].double()).cpu().numpy(), TOL, f'{n}x{Km}x{Nn} on {ctas}')
    assert bool((d[:, Nn:] == -1).all()) and bool((scratch[need:] == 3.5).all()) and spmm_cpp.dense_status() == 0


@pytest.mark.parametrize('ctas,floats', [(1, 128 * 256), (3, 2 * 256 * 256), (5, 4 * 256 * 256)])
def test_dense_tn_runs_no_more_ctas_than_it_may(ctas, floats):
    """Operands that CTA pairs would share, with an odd number of CTAs allowed: the partial results of whole pairs (of one CTA's half of X
    at a time) have to do, so that no further CTA can have written any; the same bits as two halves multiplied one by one."""
    import spmm_cpp
    n, Km, Nn = 5000, 256, 256
    g = torch.Generator(device='cuda').manual_seed(ctas)
    x, y = torch.randn(n, Km, device='cuda', generator=g), torch.randn(n, Nn, device='cuda', generator=g)
    scratch = torch.full((floats + 1024,), 3.5, device='cuda')

    def product(a, allowed, room):
        d = torch.empty(a.size(1), Nn, device='cuda')
        spmm_cpp.check(spmm_cpp.lib().dg_dense_tn(a.data_ptr(), a.stride(0), y.data_ptr(), Nn, d.data_ptr(), Nn, n, a.size(1), Nn, scratch.data_ptr(), room, allowed,
                                                  spmm_cpp._stream()))
        return d

    d = product(x, ctas, floats)
    assert_close(d.cpu().numpy(), (x.double().t() @ y.double()).cpu().numpy(), TOL, f'{ctas} CTAs')
    ranges = max(1, ctas & ~1)
    assert torch.equal(d, torch.cat([product(x[:, h:h + 128], ranges, ranges * 128 * 256) for h in (0, 128)]))
    assert bool((scratch[floats:] == 3.5).all()) and spmm_cpp.dense_status() == 0


@pytest.mark.parametrize('n,Km,Nn', [(1500, 256, 256), (2300, 100, 47)])
def test_dense_tn_on_two_streams_at_once(n, Km, Nn):
    """Weight gradients that are under way at the same time on two streams, with SMs left for each other, are what each is alone: their
    partial results share no memory."""
    import spmm_cpp
    g = torch.Generator(device='cuda').manual_seed(n)
    pairs = [(torch.randn(n, Km + (-Km) % 4, device='cuda', generator=g)[:, :Km], torch.randn(n, Nn + (-Nn) % 4, device='cuda', generator=g)[:, :Nn]) for _ in range(2)]
    alone = [spmm_cpp.dense_tn(x, y) for x, y in pairs]
    for (x, y), d in zip(pairs, alone):
        assert_close(d.cpu().numpy(), (x.double().t() @ y.double()).cpu().numpy(), TOL, f'{n}x{Km}x{Nn}')
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], [[], []]
    for _ in range(40):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                got[i].append(spmm_cpp.dense_tn(*pairs[i]))
    torch.cuda.synchronize()
    for d, same in zip(alone, got):
        assert all(torch.equal(d, e) for e in same)
    assert spmm_cpp.dense_status() == 0


def test_copies_that_are_kept_are_ready_on_every_stream():
    """A weight's split copy and an input's padded copy, made on a stream that is held up, and used meanwhile on another one."""
    import spmm_cpp
    from models.gcn import _rows
    g = torch.Generator(device='cuda').manual_seed(3)
    a = torch.randn(500, 100, device='cuda', generator=g)
    weight = torch.nn.Parameter(torch.randn(100, 64, device='cuda', generator=g))
    x = torch.randn(70001, 41, device='cuda', generator=g)
    want = spmm_cpp.dense_nt(a, weight, transposed=True)
    junk = [torch.full((1 << 20,), float('nan'), device='cuda') for _ in range(24)]
    torch.cuda.synchronize()
    del junk                                                      # what an early reader would find
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(20_000_000)                             # some ten milliseconds
        one = spmm_cpp.dense_nt(a, weight, transposed=True, cache_key=weight)
        kept = _rows(x, keep=True)
    with torch.cuda.stream(second):
        two = spmm_cpp.dense_nt(a, weight, transposed=True, cache_key=weight)
        other = _rows(x, keep=True)
        copy = other.clone()
    torch.cuda.synchronize()
    assert torch.equal(one, want) and torch.equal(two, want)
    assert other.data_ptr() == kept.data_ptr() and torch.equal(copy, x)
    with torch.no_grad():
        weight.mul_(2.0)
    assert torch.equal(spmm_cpp.dense_nt(a, weight, transposed=True, cache_key=weight), 2 * want)


@pytest.mark.parametrize('warm', [False, True])
def test_kept_copies_under_capture(warm):
    """A captured product that reads a kept padded copy, made before on another stream or not at all; the copy of a capture is not kept."""
    import spmm_cpp
    from models.gcn import dense_mm
    g = torch.Generator(device='cuda').manual_seed(4)
    x = torch.randn(3001, 41, device='cuda', generator=g)
    y = torch.randn(3001, 64, device='cuda', generator=g)
    if warm:
        dense_mm(x, y, ta=True, constant_a=True)
    else:
        dense_mm(x.clone(), y, ta=True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = dense_mm(x, y, ta=True, constant_a=True)
    eager = dense_mm(x, y, ta=True, constant_a=True)
    graph.replay()
    assert torch.equal(out, eager)
    assert_close(eager.cpu().numpy(), (x.double().t() @ y.double()).cpu().numpy(), TOL, 'captured')
    assert spmm_cpp.dense_status() == 0
