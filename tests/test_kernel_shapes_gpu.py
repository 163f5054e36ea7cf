"""Kernels at the sizes where their splits, tails and vector widths change, against 64-bit or CPU formulas."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from autoparallel_b200.ops import cuda_impl, library

    cuda_impl.ensure_loaded()
    yield library, cuda_impl
    cuda_impl.check_status()


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    assert a.shape == b.shape
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V,D,T,ids", [
    (7, 8, 1, "random"),          # one token, table smaller than a block's rows
    (50, 33, 64, "same"),         # rows that are no whole vectors; exactly one chunk of one row
    (50, 64, 65, "same"),         # one token more: the row is summed from two chunks
    (1000, 256, 5000, "skewed"),  # long and short lists side by side, more tokens than rows
    (300, 4096, 1000, "same"),    # many chunks, rows wider than a block
    (20000, 768, 9000, "random"),  # more tokens than threads of the grouping cluster, mostly empty rows
    (40, 16, 0, "random"),        # no tokens: the gradient is zero
])
def test_embedding_gradient_over_list_lengths(K, dtype, V, D, T, ids):
    lib, _ = K
    g = torch.Generator().manual_seed(V + T)
    if ids == "same":
        idx = torch.full((T,), V - 1)
    elif ids == "skewed":
        idx = (torch.rand(T, generator=g) ** 4 * V).long()
    else:
        idx = torch.randint(0, V, (T,), generator=g)
    dy = torch.randn(T, D, generator=g).to(dtype)
    out = lib.ops.embedding_bwd(dy.cuda(), idx.cuda(), V)
    ref = torch.zeros(V, D, dtype=torch.float64).index_add_(0, idx, dy.double())
    assert out.dtype == dtype and out.shape == (V, D)
    # fp32 sums of at most T terms (each partial sum rounds once: 2^-24 sqrt(T) of the norm, bounded generously), then one rounding
    assert _rel(out, ref) <= (2**-8 if dtype == torch.bfloat16 else 2**-24 * max(T, 1) ** 0.5 * 4)
    assert torch.equal(out.cpu()[torch.bincount(idx, minlength=V) == 0], torch.zeros(int((torch.bincount(idx, minlength=V) == 0).sum()), D, dtype=dtype))


@pytest.mark.parametrize("dtype,V,D,T,ids,sorts", [
    (torch.bfloat16, 40000, 1024, 1, "same", True),      # one token of a long table
    (torch.bfloat16, 40000, 1024, 32, "same", True),     # exactly one chunk, which is no long row
    (torch.bfloat16, 40000, 1024, 33, "same", True),     # the shortest long row
    (torch.bfloat16, 50257, 1000, 9000, "skewed", True),  # long and short lists, a last slice that is not full
    (torch.bfloat16, 20000, 4096, 5000, "same", True),   # many chunks, several slices of the columns
    (torch.bfloat16, 40000, 1025, 300, "random", True),  # rows that are no whole vectors
    (torch.bfloat16, 40000, 1024, 1024, "same", True),   # the longest row of the rows kernel
    (torch.bfloat16, 40000, 1024, 1025, "same", True),   # one chunk more: three groups of blocks
    (torch.bfloat16, 40000, 1025, 1600, "same", True),   # the same in rows that are no whole vectors
    (torch.bfloat16, 100, 1024, 80000, "skewed", True),  # every row long
    (torch.float32, 100, 1024, 80000, "skewed", True),
    (torch.float32, 300, 1000, 60000, "same", True),
    (torch.float32, 5, 1020, 60000, "random", True),
    (torch.float32, 5, 1023, 60000, "random", False),    # fp32 rows that are no whole vectors
    (torch.bfloat16, 1000, 256, 16384, "skewed", False),
    (torch.bfloat16, 100000, 16, 513, "random", False),
    (torch.float32, 50257, 1024, 300, "skewed", False),
])
def test_embedding_gradient_by_both_forms(K, dtype, V, D, T, ids, sorts):
    lib, impl = K
    assert impl.extension().embedding_bwd_sorts(T, V, D, dtype == torch.bfloat16) == sorts
    g = torch.Generator(device="cuda").manual_seed(V + T)
    idx = torch.randint(0, V, (T,), device="cuda", generator=g)
    if ids == "same":
        idx.fill_(V - 1)
    elif ids == "skewed":
        idx = (torch.rand(T, device="cuda", generator=g) ** 4 * V).long()
    dy = torch.randn(T, D, device="cuda", generator=g).to(dtype)
    out = lib.ops.embedding_bwd(dy, idx, V)
    ref = torch.zeros(V, D, device="cuda", dtype=torch.float64).index_add_(0, idx, dy.double())
    assert out.dtype == dtype and out.shape == (V, D)
    err = ((out.double() - ref).norm() / ref.norm()).item()
    # fp32 sums of at most T terms (each partial sum rounds once: 2^-24 sqrt(T) of the norm, bounded generously), then one rounding
    assert err <= (2**-8 if dtype == torch.bfloat16 else 2**-24 * T ** 0.5 * 4)
    assert not out[torch.bincount(idx, minlength=V) == 0].any()


@pytest.mark.parametrize("ids", ["same", "skewed", "random"])
@pytest.mark.parametrize("dtype,V,D,T", [
    (torch.bfloat16, 8003, 2048, 2000),  # the most tokens for which zeros come first, in rows of 4 KB; the last block of zeros is partial
    (torch.bfloat16, 8003, 2048, 2001),
    (torch.bfloat16, 32000, 2056, 3200),  # in longer rows
    (torch.bfloat16, 32000, 2056, 3201),
    (torch.bfloat16, 30000, 1032, 1),
    (torch.float32, 40000, 4096, 4000),
])
def test_embedding_gradient_with_zeros_first(K, dtype, V, D, T, ids):
    """Every row is written, whatever the buffer held; ids outside the table are skipped."""
    _, impl = K
    ext = impl.extension()
    if not ext.embedding_bwd_sorts(T, V, D, dtype == torch.bfloat16):
        pytest.skip("the other form")
    g = torch.Generator(device="cuda").manual_seed(V + T)
    idx = torch.randint(0, V, (T,), device="cuda", generator=g)
    if ids == "same":
        idx.fill_(V - 1)
    elif ids == "skewed":
        idx = (torch.rand(T, device="cuda", generator=g) ** 4 * V).long()
    if T > 1:
        idx[T // 2], idx[T // 3] = V, -1
    dy = torch.randn(T, D, device="cuda", generator=g).to(dtype)
    out = torch.full((V, D), float("nan"), device="cuda", dtype=dtype)
    ext.embedding_bwd(dy, idx, out)
    inside = (idx >= 0) & (idx < V)
    ref = torch.zeros(V, D, device="cuda", dtype=torch.float64).index_add_(0, idx[inside], dy[inside].double())
    err = ((out.double() - ref).norm() / ref.norm()).item()
    assert err <= (2**-8 if dtype == torch.bfloat16 else 2**-24 * T ** 0.5 * 4)  # as above
    assert not out[torch.bincount(idx[inside], minlength=V) == 0].any()


@pytest.mark.parametrize("dtype,V,D,T", [
    (torch.bfloat16, 30000, 1032, 0),
    (torch.bfloat16, 30000, 1032, 1),
    (torch.bfloat16, 8000, 2048, 2001),
    (torch.bfloat16, 100, 64, 0),  # by atomics
    (torch.float32, 40000, 4096, 0),
])
def test_embedding_gradient_counts_what_it_launches(K, dtype, V, D, T):
    _, impl = K
    cudart = pytest.importorskip("cuda.bindings.runtime")
    ext = impl.extension()
    dy, ids = torch.ones(T, D, device="cuda", dtype=dtype), torch.arange(T, device="cuda")
    out = torch.full((V, D), float("nan"), device="cuda", dtype=dtype)
    ext.embedding_bwd(dy, ids, out)
    assert torch.equal(out.sum(1), torch.where(torch.arange(V, device="cuda") < T, float(D), 0.0).to(dtype))
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        said = ext.embedding_bwd(dy, ids, out)
    assert cudart.cudaGraphGetNodes(cudart.cudaGraph_t(graph.raw_cuda_graph()))[-1] == said


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [8, 1024, 1032, 1536, 2048, 3072, 4096, 8192, 8200])
def test_a_row_is_normalised_to_the_same_bits_in_any_call(K, D, dtype):
    lib, _ = K
    g = torch.Generator(device="cuda").manual_seed(D)
    x, w = torch.randn(4100, D, device="cuda", generator=g).to(dtype), torch.randn(D, device="cuda", generator=g).to(dtype)
    y, rstd = lib.ops.rms_norm(x, w, 1e-5)
    for rows in (1, 256, 257, 1023, 1024, 4095, 4096):
        part = x[-rows:].clone()
        got = lib.ops.rms_norm(part, w, 1e-5)
        assert torch.equal(got[0], y[-rows:]) and torch.equal(got[1].view(-1), rstd.view(-1)[-rows:]), rows


def test_embedding_gradient_of_an_unaligned_view(K):
    lib, _ = K
    flat = torch.randn(1 + 12 * 16, device="cuda").to(torch.bfloat16)
    dy, idx = flat[1:].view(12, 16), torch.arange(12, device="cuda") % 5
    ref = torch.zeros(5, 16, dtype=torch.float64).index_add_(0, idx.cpu(), dy.double().cpu())
    assert _rel(lib.ops.embedding_bwd(dy, idx, 5), ref) <= 2**-8


@pytest.mark.parametrize("T,k,E,C,nb,d", [
    (8, 2, 4, 3, 1, 64),        # one chunk of assignments, drops
    (2048, 8, 64, 300, 1, 40),  # 32 chunks of 512; rows of 80 bytes
    (1000, 3, 16, 50, 8, 129),  # odd block sizes, rows that are no whole vectors, nine assignments past a warp
    (512, 9, 500, 16, 1, 2304),  # more choices than one gather step, more experts than threads per group, wide rows
    (70000, 8, 8, 4000, 1, 8),  # more assignments than two rounds of all CTAs
])
@pytest.mark.parametrize("dtype,wdtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16)])
def test_moe_dispatch_over_shapes(K, T, k, E, C, nb, d, dtype, wdtype):
    lib, impl = K
    from autoparallel_b200.ops import moe_ops

    g = torch.Generator().manual_seed(T + k)
    idx = (torch.rand(T, E, generator=g) + torch.linspace(0.3, 0, E)).topk(k).indices
    x, w = torch.randn(T, d, generator=g).to(dtype), torch.rand(T, k, generator=g).to(wdtype)
    before = dict(impl.library_fallbacks)
    slot = lib.ops.moe_slots(idx.cuda(), E, C, nb)
    rslot = moe_ops._moe_slots(idx, E, C, nb)
    assert torch.equal(slot.cpu(), rslot)
    buf = lib.ops.moe_scatter(x.cuda(), slot, w.cuda(), E, C, nb)
    rbuf = moe_ops._moe_scatter(x, rslot, w, E, C, nb)
    assert torch.equal(buf.cpu(), rbuf)  # one product per element, empty rows zero
    flat, ec = moe_ops._buf_rows(rbuf.double())
    picked = flat[moe_ops._rows(rslot, nb, ec)].view(T, k, -1)
    tol = 2**-8 if dtype == torch.bfloat16 else 2**-20
    assert _rel(lib.ops.moe_gather(buf, slot, w.cuda()), (picked * w.to(dtype).double().unsqueeze(2)).sum(1)) <= tol
    assert _rel(lib.ops.moe_gate_grad(buf, slot, x.cuda()), (picked * x.double().unsqueeze(1)).sum(-1)) <= 2**-18
    assert impl.library_fallbacks == before, "the kernels cover these shapes"


@pytest.mark.parametrize("T,k,E,C,nb,d", [
    (96, 40, 64, 50, 1, 264),   # more choices than lanes, a second piece of a row that is not full
    (9600, 2, 8, 2600, 1, 520),  # one warp takes all columns of its token
    (3, 1, 4, 1, 1, 8),         # fewer tokens than warps of a block
])
@pytest.mark.parametrize("dtype,wdtype", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)])
def test_moe_gather_over_warps_and_choices(K, T, k, E, C, nb, d, dtype, wdtype):
    test_moe_dispatch_over_shapes(K, T, k, E, C, nb, d, dtype, wdtype)


@pytest.mark.parametrize("T,k,nb,launches", [(16, 2, 1, 1), (510, 1, 1, 1), (513, 1, 1, 1), (512, 2, 1, 1), (4096, 2, 8, 1), (513, 2, 1, 2), (2050, 2, 2, 2)])
@pytest.mark.parametrize("E", [8, 372, 700])
def test_moe_slots_around_one_and_two_rounds(K, T, k, nb, launches, E):
    """One round, two rounds of one CTA, and the first sizes that are cut into chunks."""
    lib, impl = K
    from autoparallel_b200.ops import moe_ops

    idx = torch.randint(0, E, (T, k), generator=torch.Generator().manual_seed(T))
    idx[0] = idx[-1] = 3  # (one expert past its capacity wherever it is small)
    before, fallbacks = impl.launch_count, dict(impl.library_fallbacks)
    slot = lib.ops.moe_slots(idx.cuda(), E, 5, nb)
    assert torch.equal(slot.cpu(), moe_ops._moe_slots(idx, E, 5, nb))
    assert impl.launch_count - before == launches and impl.library_fallbacks == fallbacks


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_moe_rows_of_a_buffer_of_more_than_half_of_l2(K, dtype):
    """66 and 132 MB: rows that are stored to leave L2 first, and a gather that fills the SMs."""
    lib, _ = K
    T, k, E, C, d = 6001, 4, 32, 1000, 1032
    g = torch.Generator(device="cuda").manual_seed(5)
    idx = torch.rand(T, E, device="cuda", generator=g).topk(k).indices
    w = torch.rand(T, k, device="cuda", generator=g).to(dtype)
    x = torch.randn(T, d, device="cuda", generator=g).to(dtype)
    slot = lib.ops.moe_slots(idx, E, C, 1)
    buf = lib.ops.moe_scatter(x, slot, w, E, C, 1)
    kept = (slot >= 0) & (slot < E * C)
    assert kept.any() and (slot[kept].unique().numel() == int(kept.sum()))
    ref = torch.zeros(E * C, d, device="cuda", dtype=dtype)
    ref[slot[kept]] = (x.float().unsqueeze(1) * w.float().unsqueeze(2)).to(dtype)[kept]
    assert torch.equal(buf.view(E * C, d), ref)
    out = lib.ops.moe_gather(buf, slot, w)
    rows = torch.where(kept.unsqueeze(2), ref[slot.clamp(0, E * C - 1)].double(), 0.0)
    # fp32 sums of four products, one rounding
    assert _rel(out, (rows * w.double().unsqueeze(2)).sum(1)) <= 2**-22 + (2**-8 if dtype == torch.bfloat16 else 0)


@pytest.mark.parametrize("T,k,rows,nb", [(32, 2, 40, 1), (6000, 8, 40, 1), (6000, 8, 40000, 1), (3000, 3, 600, 3)])
def test_moe_scatter_of_repeated_slots(K, T, k, rows, nb):
    """The last choice that names a row has it, as if they were stored in order, whatever the table of rows held before and however
    often it is repeated."""
    lib, _ = K
    E, d = 8, 8
    C = rows // E
    g = torch.Generator(device="cuda").manual_seed(T)
    slot = torch.randint(0, E * C + 1, (T, k), device="cuda", generator=g)
    x = torch.randn(T, d, device="cuda", generator=g)
    w = torch.rand(T, k, device="cuda", generator=g)
    flat = torch.zeros(nb, E * C + 1, d).numpy()
    block = (torch.arange(T) // (T // nb)).unsqueeze(1).expand(T, k)
    rows_of_x = (x.unsqueeze(1) * w.unsqueeze(2)).reshape(T * k, d).cpu().numpy()
    flat[block.reshape(-1).numpy(), slot.reshape(-1).cpu().numpy()] = rows_of_x  # (in order)
    ref = torch.from_numpy(flat)[:, :E * C].view(nb, E, C, d).transpose(0, 1).contiguous()
    for i in range(100):
        junk = torch.full((E * nb * C,), T * k - 1, device="cuda")
        if i % 2:
            junk.random_(-3, T * k + 3, generator=g)
        del junk  # (the table takes its memory)
        assert torch.equal(lib.ops.moe_scatter(x, slot, w, E, C, nb).cpu(), ref)


def test_moe_dispatch_leaves_nothing_of_the_old_buffer(K):
    """Every row of the buffer is written, also those no assignment names, whatever the memory held before."""
    lib, _ = K
    idx = torch.zeros(64, 1, dtype=torch.long, device="cuda")
    slot = lib.ops.moe_slots(idx, 4, 128, 1)
    x = torch.randn(64, 256, device="cuda", dtype=torch.bfloat16)
    for _ in range(3):
        junk = [torch.full((4 * 128 * 256,), float("nan"), device="cuda", dtype=torch.bfloat16),
                torch.arange(4 * 128, device="cuda")]  # what the buffer and the row table may be allocated over
        del junk
        buf = lib.ops.moe_scatter(x, slot, torch.ones(64, 1, device="cuda", dtype=torch.bfloat16), 4, 128, 1)
        assert torch.equal(buf[0, 0, :64], x) and not buf[0, 0, 64:].any() and not buf[1:].any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 3, 149, 5000])
@pytest.mark.parametrize("D", [8, 256, 264, 768, 1032, 2048, 4096, 5120, 8192, 16384])
def test_rms_norm_gradients_over_row_widths(K, dtype, rows, D):
    """One row, fewer rows than SMs, one more, several steps per block; widths on both sides of every block size and, in
    fp32, past what the staged form holds."""
    lib, _ = K
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    x = torch.randn(rows, D, device="cuda", generator=g).to(dtype)
    w = (1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(dtype)
    dy = torch.randn(rows, D, device="cuda", generator=g).to(dtype)
    _, rstd = lib.ops.rms_norm(x, w, 1e-5)
    dx, dw = lib.ops.rms_norm_bwd(dy, x, w, rstd)
    xd, wd, gd, rd = x.double(), w.double(), dy.double(), rstd.double().unsqueeze(-1)
    xh = xd * rd
    gw = gd * wd
    # fp32 sums over a row (dx) and over the rows (dw): 2^-24 times the square root of their length, generously, then one rounding
    tol = 2**-8 if dtype == torch.bfloat16 else 2**-24 * 16 * max(rows, D) ** 0.5
    assert _rel(dx, rd * (gw - xh * (gw * xh).mean(-1, keepdim=True))) <= tol
    assert _rel(dw, (gd * xh).sum(0)) <= tol


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,D", [(5, 8), (20000, 8), (148, 256), (9000, 256), (700, 2048), (5000, 4096), (600, 8192), (300, 10240), (200, 16384)])
def test_allocation_free_rms_norm_gradients_over_shared_rows(K, dtype, rows, D):
    """One partial row, several, the most that fit; each width that changes their number."""
    import ctypes

    from autoparallel_b200.ops import build

    so = ctypes.CDLL(build.so_path())
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, D, device="cuda", generator=g).to(dtype)
    w = (1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(dtype)
    dy = torch.randn(rows, D, device="cuda", generator=g).to(dtype)
    rstd = torch.rsqrt(x.float().pow(2).mean(-1) + 1e-5)
    dx, dw = torch.empty_like(x), torch.empty_like(w)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (dy, x, w, rstd, dx, dw)]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert so.apb_rms_norm_bwd_noalloc(*p, ctypes.c_longlong(rows), D, int(dtype == torch.bfloat16), st) == 0
    xd, wd, gd, rd = x.double(), w.double(), dy.double(), rstd.double().unsqueeze(-1)
    xh, gw = xd * rd, gd * wd
    # as above: fp32 sums over a row (dx) and over the rows (dw), then one rounding
    tol = 2**-8 if dtype == torch.bfloat16 else 2**-24 * 16 * max(rows, D) ** 0.5
    assert _rel(dx, rd * (gw - xh * (gw * xh).mean(-1, keepdim=True))) <= tol
    assert _rel(dw, (gd * xh).sum(0)) <= tol


@pytest.mark.parametrize("M,N,K_", [
    (256, 256, 64),     # one pair tile, one k-block
    (4104, 4104, 64),   # every pair busy, both edges end inside a 32-row / 64-column store
    (5000, 4136, 136),  # a row edge inside a warp's block, K past a k-block
    (20000, 264, 8),    # a column tile of eight columns
])
@pytest.mark.parametrize("ta,tb", [(False, True), (True, False)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("pair", [True, False])
def test_gemm_stores_whole_tiles_and_nothing_else(K, M, N, K_, ta, tb, out_dtype, pair):
    lib, impl = K
    ext = impl.extension()
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn((K_, M) if ta else (M, K_), device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn((N, K_) if tb else (K_, N), device="cuda", generator=g).to(torch.bfloat16)
    back = torch.full((M + 2, N + 64), 7.0, device="cuda", dtype=out_dtype)  # the result is a window of a wider matrix
    c = back[1:M + 1, 32:N + 32]
    prev = ext.gemm_get_pair_mode()
    ext.gemm_set_pair_mode(pair)
    try:
        ext.gemm(a, b, c, ta, not tb, impl.status_buffer(a.device))
        torch.cuda.synchronize()
    finally:
        ext.gemm_set_pair_mode(prev)
    ref = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    # fp32 accumulation of K products (2^-24 sqrt(K), generously), one rounding to bf16
    assert _rel(c, ref) <= (2**-8 if out_dtype == torch.bfloat16 else 2**-24 * 8 * K_ ** 0.5)
    back[1:M + 1, 32:N + 32] = 7.0
    assert bool((back == 7.0).all()), "nothing outside the window is written"


@pytest.mark.parametrize("E,M,N,K_", [(5, 160, 1408, 136), (3, 320, 72, 64), (4, 1000, 264, 72)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_grouped_gemm_keeps_group_edges(K, E, M, N, K_, out_dtype):
    """M and N end inside a store block: the next group's first rows must not be overwritten."""
    lib, _ = K
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(E, M, K_, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(E, K_, N, device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randn(E, M, N, device="cuda", generator=g).to(torch.bfloat16)
    bf16 = out_dtype == torch.bfloat16
    assert _rel(lib.ops.grouped_mm(a, w, False, out_dtype), a.double() @ w.double()) <= (2**-8 if bf16 else 2**-24 * 8 * K_ ** 0.5)
    assert _rel(lib.ops.grouped_mm_wgrad(a, dy, out_dtype), a.double().transpose(1, 2) @ dy.double()) <= (2**-8 if bf16 else 2**-24 * 8 * M ** 0.5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [8, 1024, 4096 + 8, 8192, 16384 - 8, 16384, 16384 + 4096 + 8, 128256])
def test_cross_entropy_over_row_widths(K, dtype, V):
    """Rows below, at and past a full unrolled step of every block size; rows with masked (-inf and lowest) entries."""
    lib, _ = K
    g = torch.Generator(device="cuda").manual_seed(V)
    rows = 5
    logits = (3 * torch.randn(rows, V, device="cuda", generator=g)).to(dtype)
    labels = torch.randint(0, V, (rows,), device="cuda", generator=g)
    logits[1, : V // 2] = float("-inf")
    logits[2, V // 2:] = torch.finfo(dtype).min
    labels[1], labels[2] = V - 1, 0
    loss, lse = lib.ops.cross_entropy(logits, labels)
    ld = logits.double()
    ref = torch.logsumexp(ld, -1)
    picked = ld.gather(-1, labels.unsqueeze(-1)).squeeze(-1)
    # the exponentials are the hardware's (2^-21 relative each); their sum is fp32, the values are of order 10
    assert _rel(lse, ref) <= 2**-19 and (loss.double() - (ref - picked)).abs().max().item() <= 2**-19 * 16
    dl = torch.randn(rows, device="cuda", generator=g)
    d = lib.ops.cross_entropy_bwd(dl, logits, labels, lse)
    p = torch.softmax(ld, -1)
    p[torch.arange(rows), labels] -= 1
    assert _rel(d, p * dl.double().unsqueeze(-1)) <= (2**-8 if dtype == torch.bfloat16 else 2**-18)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [8, 2048, 4096 + 8, 8192 + 8, 24000, 36000, 60008, 140008])
def test_cross_entropy_with_more_rows_than_two_per_sm(K, dtype, V):
    """The block sizes of long batches; a last vector that only some threads have."""
    lib, _ = K
    g = torch.Generator(device="cuda").manual_seed(V)
    rows = 300
    logits = (3 * torch.randn(rows, V, device="cuda", generator=g)).to(dtype)
    labels = torch.randint(0, V, (rows,), device="cuda", generator=g)
    logits[1, : V // 2] = float("-inf")
    labels[1] = V - 1
    loss, lse = lib.ops.cross_entropy(logits, labels)
    dl = torch.randn(rows, device="cuda", generator=g)
    d = lib.ops.cross_entropy_bwd(dl, logits, labels, lse)
    ld = logits.double()
    ref = torch.logsumexp(ld, -1)
    # bounds as above
    assert _rel(lse, ref) <= 2**-19 and (loss.double() - (ref - ld.gather(-1, labels.unsqueeze(-1)).squeeze(-1))).abs().max().item() <= 2**-19 * 16
    p = torch.softmax(ld, -1)
    p[torch.arange(rows), labels] -= 1
    assert _rel(d, p * dl.double().unsqueeze(-1)) <= (2**-8 if dtype == torch.bfloat16 else 2**-18)


@pytest.mark.parametrize("M,N,K_", [(1, 8, 8), (16, 4096, 4096), (64, 2048, 8192), (129, 264, 520), (1000, 1408, 2048), (300, 72, 1096)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("bn,slices", [(0, 0), (64, 8), (64, 1), (128, 3), (256, 5), (256, 2)])
def test_gemm_split_over_tiles_and_slices(K, M, N, K_, ta, tb, bn, slices):
    """Tile widths and slice counts, ragged in every dimension, inside a wider matrix; (0, 0) = what the rule picks."""
    lib, impl = K
    ext = impl.extension()
    if (ta and M % 8) or slices > (K_ + 63) // 64:
        pytest.skip("not a form of this kernel")
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn((K_, M) if ta else (M, K_), device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn((N, K_) if tb else (K_, N), device="cuda", generator=g).to(torch.bfloat16)
    ref = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    for dtype in (torch.float32, torch.bfloat16):
        back = torch.full((M + 2, N + 64), 7.0, device="cuda", dtype=dtype)
        c = back[1:M + 1, 32:N + 32]
        if bn:
            ext.gemm_split(a, b, c, ta, not tb, bn, slices, impl.status_buffer(a.device))
        else:
            ext.gemm(a, b, c, ta, not tb, impl.status_buffer(a.device))
        # fp32 accumulation of K products (2^-24 sqrt(K), generously), one rounding to bf16
        assert _rel(c, ref) <= (2**-8 if dtype == torch.bfloat16 else 2**-24 * 8 * max(K_, 64) ** 0.5)
        back[1:M + 1, 32:N + 32] = 7.0
        assert bool((back == 7.0).all()), "nothing outside the window is written"


@pytest.mark.parametrize("groups,M,N,K_,split", [
    (0, 16, 4096, 4096, True),       # few rows
    (0, 64, 2048, 8192, True),       # a router's weight gradient
    (0, 512, 256, 256, True),        # four pair tiles
    (16, 64, 704, 1024, True),       # a stack of small products
    (0, 8192, 4096, 4096, False),    # more tiles than SMs
    (64, 160, 1408, 2048, False),
    (0, 300, 64, 64, False),         # one k-block, no more CTAs to be had than the persistent kernel uses
    (0, 4858, 16, 80, False),
])
def test_which_products_are_split(K, groups, M, N, K_, split):
    _, impl = K
    ext = impl.extension()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    bn, s = ext.gemm_split_choice(groups, M, N, K_)
    assert (bn != 0) == split
    prev = ext.gemm_get_reserved_sms()
    try:
        for reserved in (0, 40, sms):
            ext.gemm_set_reserved_sms(reserved)
            bn, s = ext.gemm_split_choice(groups, M, N, K_)
            if bn:
                ctas = max(groups, 1) * -(-M // 128) * -(-N // bn) * s
                assert ctas <= sms - reserved and (s == 1 or 2 * s <= -(-K_ // 64)) and (bn, s) != (256, 1)
    finally:
        ext.gemm_set_reserved_sms(prev)


@pytest.mark.parametrize("M,N,K_", [(512, 512, 2048), (300, 264, 520), (2000, 1544, 136)])
@pytest.mark.parametrize("stages,dynamic", [(4, False), (5, False), (6, True)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_pairs_that_make_room_for_communication(K, M, N, K_, stages, dynamic, out_dtype):
    """Fewer stages, and dynamic tiles that answer a request for SM pairs: also in products with few tiles, which would be split."""
    lib, impl = K
    ext = impl.extension()
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K_, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(N, K_, device="cuda", generator=g).to(torch.bfloat16)
    prev = ext.gemm_get_pair_stages(), ext.gemm_get_dynamic_tiles()
    ext.gemm_set_pair_stages(stages)
    ext.gemm_set_dynamic_tiles(dynamic)
    try:
        if dynamic:
            ext.gemm_yield_request(1)
            assert ext.gemm_yield_outstanding() == 1
        c = lib.ops.gemm(a, b, False, True, out_dtype)
        assert ext.gemm_yield_outstanding() == 0  # (half of a launch of two pairs or more may go)
    finally:
        ext.gemm_set_pair_stages(prev[0])
        ext.gemm_set_dynamic_tiles(prev[1])
    # fp32 accumulation of K products (2^-24 sqrt(K), generously), one rounding to bf16
    assert _rel(c, a.double() @ b.double().t()) <= (2**-8 if out_dtype == torch.bfloat16 else 2**-24 * 8 * K_ ** 0.5)


@pytest.mark.parametrize("bn,slices", [(64, 2), (128, 1), (256, 3)])
def test_grouped_gemm_split(K, bn, slices):
    lib, impl = K
    E, M, N, K_ = 3, 200, 328, 264
    g = torch.Generator(device="cuda").manual_seed(bn)
    a = torch.randn(E, M, K_, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(E, K_, N, device="cuda", generator=g).to(torch.bfloat16)
    c = torch.empty(E, M, N, device="cuda", dtype=torch.float32)
    impl.extension().gemm_split(a, w, c, False, True, bn, slices, impl.status_buffer(a.device))
    assert _rel(c, a.double() @ w.double()) <= 2**-24 * 8 * K_ ** 0.5


@pytest.mark.parametrize("M", [129, 136, 160, 248])
@pytest.mark.parametrize("ta", [False, True])
def test_pairs_with_less_than_two_full_row_tiles(K, M, ta):
    """The odd CTA of a pair holds 1 to 120 rows; enough columns and groups that the persistent pair kernels run."""
    lib, impl = K
    if ta and M % 8:
        pytest.skip("rows of 16 bytes")
    E, N, K_ = 24, 1408, 1288  # (a contraction long enough for pairs)
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(*((E, K_, M) if ta else (E, M, K_)), device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(E, K_, N, device="cuda", generator=g).to(torch.bfloat16)
    if ta:
        got, ref = lib.ops.grouped_mm_wgrad(a, w, torch.float32), a.double().transpose(1, 2) @ w.double()
    else:
        got, ref = lib.ops.grouped_mm(a, w, False, torch.float32), a.double() @ w.double()
    assert _rel(got, ref) <= 2**-24 * 8 * K_ ** 0.5  # fp32 accumulation of K products
    x, y = a[0], torch.randn(K_, 20480, device="cuda", generator=g).to(torch.bfloat16)
    out = lib.ops.gemm(x, y, ta, False, torch.float32)
    assert _rel(out, (x.double().t() if ta else x.double()) @ y.double()) <= 2**-24 * 8 * K_ ** 0.5


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("G,M,N,Kd", [
    (0, 4361, 1800, 72),   # pairs: groups of 16 tile rows and one of 2, a last tile row of 9 rows, a last column tile of 8 columns
    (0, 100, 40000, 72),   # one CTA per tile, more tiles than SMs
    (3, 2600, 1032, 40),   # grouped: several groups per CTA pair, one k-block that is not full
    (0, 5000, 5128, 6552),  # a long contraction, rounds of tiles that read 70 MB, a last k-block that is not full
    (0, 128, 39000, 26000),  # the same with one CTA per tile
    (70, 160, 520, 1288),  # grouped, an odd CTA with 32 rows
])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True)])
def test_gemm_tiles_land_where_they_belong(K, G, M, N, Kd, a_mn, b_mn, out):
    """Whole numbers: every sum is exact.  The plain product writes into the middle of a wider matrix, whose margins stay."""
    _, impl = K
    ext = impl.extension()
    if a_mn and M % 8:
        M += 8 - M % 8  # (rows of 16 bytes)
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    lead = (G,) if G else ()
    a = torch.randint(-1, 2, (*lead, M, Kd), device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randint(-1, 2, (*lead, N, Kd), device="cuda", generator=gen).to(torch.bfloat16)
    ref = (a.float() @ b.float().transpose(-1, -2)).to(out)
    a = a.transpose(-1, -2).contiguous() if a_mn else a
    b = b.transpose(-1, -2).contiguous() if b_mn else b
    if G:
        c = torch.full((G, M, N), 99.0, device="cuda", dtype=out)
        ext.gemm_grouped(a, b, c, a_mn, b_mn, impl.status_buffer(c.device))
        assert torch.equal(c, ref)
        return
    for pad in (8, 1):  # rows of whole 16-byte vectors, and rows that are not
        wide = torch.full((M + 2, N + 8 + pad), 99.0, device="cuda", dtype=out)
        flat = wide.view(-1)
        c = flat[8:8 + (M - 1) * wide.shape[1] + N].as_strided((M, N), (wide.shape[1], 1))  # (starts on a 16-byte boundary)
        ext.gemm(a, b, c, a_mn, b_mn, impl.status_buffer(c.device))
        assert torch.equal(c, ref)
        c.fill_(99.0)
        assert bool((wide == 99.0).all())


@pytest.mark.parametrize("G,M,N,Kd", [
    (0, 1504, 4104, 72),    # 102 pair tiles: a wave of whole ones, the others in halves, a last column tile of 8 columns
    (0, 1500, 4232, 72),    # a last column tile of 136 columns
    (0, 4360, 4872, 6552),  # wide tiles, a last column tile of 8 columns, the rest of the waves column tile by column tile
    (0, 5896, 4104, 6552),  # wide tiles, an odd number of column tiles: the last wide one has 8 columns
    (0, 4100, 1032, 72),    # whole tiles only, 8 columns in the last column tile
    (64, 160, 1416, 136),   # grouped
    (20, 2304, 2184, 8200),  # grouped, a long contraction in column tiles of their own
    (10, 2304, 4104, 8200),  # grouped, wide
])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("dynamic", [False, True])
def test_whole_and_half_and_wide_tiles(K, G, M, N, Kd, a_mn, b_mn, dynamic):
    """Whole numbers first: every sum is exact, and nothing is written past the result.  Then columns that repeat every 128 and rows that
    repeat every 4: their results are the same bits in whatever kind of tile they lie."""
    _, impl = K
    ext = impl.extension()
    if (a_mn and M % 8) or (dynamic and G):
        pytest.skip("rows of 16 bytes; grouped products have no dynamic tiles")
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    lead = (G,) if G else ()
    prev = ext.gemm_get_dynamic_tiles()
    ext.gemm_set_dynamic_tiles(dynamic)
    try:
        for random in (False, True):
            if random:
                a = torch.randn(*lead, 4, Kd, device="cuda", generator=gen).to(torch.bfloat16).repeat(*([1] * len(lead)), M // 4, 1)
                b = torch.randn(*lead, 128, Kd, device="cuda", generator=gen).to(torch.bfloat16).repeat(*([1] * len(lead)), N // 128 + 1, 1)
                b = b[..., :N, :].contiguous()
            else:
                a = torch.randint(-1, 2, (*lead, M, Kd), device="cuda", generator=gen).to(torch.bfloat16)
                b = torch.randint(-1, 2, (*lead, N, Kd), device="cuda", generator=gen).to(torch.bfloat16)
            x = a.transpose(-1, -2).contiguous() if a_mn else a
            y = b.transpose(-1, -2).contiguous() if b_mn else b
            flat = torch.full(((G or 1) * M * N + 4096,), 99.0, device="cuda")
            c = flat[:-4096].view(*lead, M, N)
            if G:
                ext.gemm_grouped(x, y, c, a_mn, b_mn, impl.status_buffer(c.device))
            else:
                ext.gemm(x, y, c, a_mn, b_mn, impl.status_buffer(c.device))
            assert bool((flat[-4096:] == 99.0).all())
            if random:
                first = c[..., :4, :128].repeat(*([1] * len(lead)), M // 4, N // 128 + 1)[..., :N]
                assert torch.equal(c, first)
            else:
                assert torch.equal(c, a.float() @ b.float().transpose(-1, -2))
    finally:
        ext.gemm_set_dynamic_tiles(prev)


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("N,Kd", [
    (16, 8),       # one block, one warp with work, a step that is not full
    (24, 40),      # a block with 8 of its 16 columns
    (1000, 520),   # warps with one step and with two
    (2376, 1024),  # more blocks than SMs
    (1024, 2048),  # fewer, and a long contraction
    (4096, 4096),
    (520, 8192),   # the longest contraction with up to 8 rows
    (9480, 304),   # three rounds of blocks
    (56, 14344),   # the split kernel's
])
def test_gemm_of_a_few_rows(K, M, N, Kd, out):
    """Around the blocks of 8 rows and of 16 columns; rows of the operands and of the result that lie further apart than they are long."""
    _, impl = K
    ext = impl.extension()
    gen = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    a = torch.randn(M + 1, Kd + 8, device="cuda", generator=gen).to(torch.bfloat16)[:M, :Kd]
    w = torch.randn(N, Kd + 16, device="cuda", generator=gen).to(torch.bfloat16)[:, :Kd]
    whole = torch.full((M + 1, N + 8), 99.0, device="cuda", dtype=out)
    c = whole[:M, :N]
    ext.gemm(a, w, c, False, False, impl.status_buffer(c.device))
    ref = a.double() @ w.double().t()
    # fp32 accumulation of K products, then one rounding
    assert _rel(c, ref) <= 2**-24 * 8 * Kd ** 0.5 + (2**-8 if out == torch.bfloat16 else 0)
    c.fill_(99.0)
    assert bool((whole == 99.0).all())


@pytest.mark.parametrize("pair", [True, False])
def test_gemm_bits_do_not_depend_on_the_launch(K, pair):
    """Products whose rounds of tiles read more than L2 holds: equal rows and columns of the operands give equal results wherever they lie,
    and reserved SMs or tiles handed out at run time change no bit."""
    _, impl = K
    ext = impl.extension()
    M, N, K_, rows, cols = 5120, 5120, 8192, 512, 512
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(rows, K_, device="cuda", generator=g).to(torch.bfloat16).repeat(M // rows, 1)
    b = torch.randn(cols, K_, device="cuda", generator=g).to(torch.bfloat16).repeat(N // cols, 1)
    prev = ext.gemm_get_pair_mode(), ext.gemm_get_reserved_sms(), ext.gemm_get_dynamic_tiles()
    ext.gemm_set_pair_mode(pair)
    try:
        first = None
        for reserved, dynamic in ((0, False), (16, False), (50, False), (0, True), (16, True)):
            ext.gemm_set_reserved_sms(reserved)
            ext.gemm_set_dynamic_tiles(dynamic)
            c = torch.empty(M, N, device="cuda")
            ext.gemm(a, b, c, False, False, impl.status_buffer(c.device))
            blocks = c.view(M // rows, rows, N // cols, cols)
            assert torch.equal(blocks, blocks[:1, :, :1].expand_as(blocks)), (reserved, dynamic)
            first = c if first is None else first
            assert torch.equal(c, first), (reserved, dynamic)
    finally:
        ext.gemm_set_pair_mode(prev[0])
        ext.gemm_set_reserved_sms(prev[1])
        ext.gemm_set_dynamic_tiles(prev[2])


def test_communication_kernels_fit_beside_a_gemm_cta(K):
    """Threads, registers (in units of 256 per warp) and shared memory (1 KB more per CTA than it asks for) of an SM."""
    kinds = K[1].extension().kernel_footprints()
    sm = torch.cuda.get_device_properties(0)
    registers = lambda threads, per_thread: threads // 32 * (-(-32 * per_thread // 256) * 256)
    for kind in ("gemm", "split"):
        for gemm in kinds[kind]:
            for other in kinds["beside"]:
                assert gemm[0] + other[0] <= sm.max_threads_per_multi_processor
                assert registers(*gemm[:2]) + registers(*other[:2]) <= sm.regs_per_multiprocessor, (kind, gemm, other)
                assert gemm[2] + other[2] + 2 * 1024 <= sm.shared_memory_per_multiprocessor, (kind, gemm, other)


@pytest.mark.parametrize("groups,M,N,K_,bn,slices", [
    (0, 2514, 256, 1096, 128, 2), (0, 2615, 176, 3416, 256, 4), (4, 1470, 200, 2024, 256, 2), (0, 155, 472, 7304, 128, 8), (0, 121, 10624, 2360, 256, 2)])
def test_a_faster_form_has_no_longer_chains(K, groups, M, N, K_, bn, slices):
    """The error of an fp32 result grows with the blocks that one chain of sums runs through; the form that the rule picks is as exact as
    the one given, which it took before the kernels got faster (a tenth for the order of the sums)."""
    _, impl = K
    ext = impl.extension()
    g = torch.Generator(device="cuda").manual_seed(M)
    lead = (groups,) if groups else ()
    a = torch.randn(*lead, M, K_, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(*lead, N, K_, device="cuda", generator=g).to(torch.bfloat16)
    ref = a.double() @ b.double().transpose(-1, -2)
    c, given = torch.empty(*lead, M, N, device="cuda"), torch.empty(*lead, M, N, device="cuda")
    (ext.gemm_grouped if groups else ext.gemm)(a, b, c, False, False, impl.status_buffer(a.device))
    ext.gemm_split(a, b, given, False, False, bn, slices, impl.status_buffer(a.device))
    assert _rel(c, ref) <= 1.1 * _rel(given, ref)


@pytest.mark.parametrize("M,N,K_", [(129, 265, 520), (1, 7, 1024), (260, 130, 72)])
@pytest.mark.parametrize("bn,slices", [(64, 1), (64, 2), (128, 1), (128, 7), (256, 1), (256, 4)])
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
def test_gemm_split_rows_that_are_no_whole_vectors(K, M, N, K_, bn, slices, out):
    """Leading dimensions that are multiples of four, of two and odd, columns past the last whole vector: element by element, for one slice
    as for more.  Whole numbers: every sum is exact."""
    _, impl = K
    ext = impl.extension()
    if slices > (K_ + 63) // 64:
        pytest.skip("not a form of this kernel")
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randint(-1, 2, (M, K_), device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randint(-1, 2, (N, K_), device="cuda", generator=gen).to(torch.bfloat16)
    ref = (a.float() @ b.float().t()).to(out)
    for ld in (-(-N // 8) * 8 + 4, -(-N // 8) * 8 + 2, -(-N // 8) * 8 + 1):
        flat = torch.full((8 + M * ld + 8,), 99.0, device="cuda", dtype=out)
        c = flat[8:].as_strided((M, N), (ld, 1))  # (starts on a 16-byte boundary)
        ext.gemm_split(a, b, c, False, False, bn, slices, impl.status_buffer(c.device))
        assert torch.equal(c, ref), ld
        c.fill_(99.0)
        assert bool((flat == 99.0).all()), ld


@pytest.mark.parametrize("sizes", [[1], [0, 5, 0], [2047, 2048, 2049, 8], [16] * 48, [24] * 49 + [1 << 20, 3]])
def test_cast_many(K, sizes):
    """Blocks that are not full, empty tensors, as many tensors as one launch takes and more; tensors that go one by one."""
    lib, impl = K
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    xs = [torch.randn(n, device="cuda", generator=g) for n in sizes]
    before = impl.launch_count
    out = lib.ops.cast_many(xs, torch.bfloat16)
    assert impl.launch_count - before == -(-sum(n > 0 for n in sizes) // 48)
    assert all(o.dtype == torch.bfloat16 and torch.equal(o, x.to(torch.bfloat16)) for o, x in zip(out, xs))
    odd = [torch.randn(9, device="cuda")[1:], torch.randn(4, 6, device="cuda").t(), torch.randn(8, device="cuda").bfloat16(), *xs[:1]]
    got = lib.ops.cast_many(odd, torch.bfloat16)
    assert all(o.dtype == torch.bfloat16 and torch.equal(o, x.to(torch.bfloat16)) for o, x in zip(got, odd))
    assert all(torch.equal(o, x.float()) for o, x in zip(lib.ops.cast_many(out, torch.float32), out))
