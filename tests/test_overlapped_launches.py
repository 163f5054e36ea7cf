"""Kernels that are launched to overlap with the end of the one before them (ops/csrc/launch.cuh)."""
import glob
import os
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autoparallel_b200", "ops", "csrc")


def _kernels(text):
    """(name, head, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\(", text):
        i = text.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), text[m.start():i], text[i:j]


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", f.read())


def test_what_an_overlapped_kernel_reads_is_not_declared_constant():
    """Its inputs may be written while it is resident: a load that promises read-only data may be moved above the wait."""
    seen = 0
    for name, text in _sources():
        waits = [k for k in _kernels(text) if re.search(r"\b(after_previous|wait_previous|gemm_cta)\b", k[2])]
        seen += len(waits)
        for kernel, head, _ in waits:
            assert "__restrict__" not in head, (name, kernel)
        if waits:
            assert "__ldg(" not in text and "ld.global.nc" not in text, name
    assert seen > 25


def _chain(ops, state, sync):
    """Short launches that each read what the one before them wrote, in memory that the allocator hands out again and again."""
    x, w1, w2, norm, cos, sin, ids, slots, gates = state
    out = []

    def do(fn, *args):
        r = fn(*args)
        sync()
        return r

    for _ in range(3):
        h = do(ops.dtype_cast, x, torch.bfloat16)
        a = do(ops.mm_nd, h, w1, True, torch.bfloat16)
        y, rstd = do(ops.rms_norm, a, norm, 1e-5)
        s = do(ops.swiglu, y, a)
        r = do(ops.rope, s.view(1, s.shape[0], 4, -1), cos, sin, False).view_as(s)
        buf = do(ops.moe_scatter, r, slots, gates, 4, 8, 1)
        g = do(ops.moe_gather, buf, slots, gates)
        loss, lse = do(ops.cross_entropy, g, ids)
        dg = do(ops.cross_entropy_bwd, loss, g, ids, lse)
        dx, dw = do(ops.rms_norm_bwd, dg, a, norm, rstd)
        e = do(ops.embedding_bwd, dx, ids, 300)
        t = do(ops.embedding, e, ids)
        x = do(ops.dtype_cast, do(ops.mm_nd, t, w2, True, torch.bfloat16), torch.float32)
        out += [a, y, r, g, loss, dg, dx, dw, e, x]
    return out


def _state(seed, rows=8, d=512):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    bf = torch.bfloat16
    ids = torch.randperm(300, device="cuda", generator=g)[:rows]  # (one token a row: sums in one order)
    slots = torch.randperm(32, device="cuda", generator=g)[:2 * rows].view(rows, 2)
    w1, w2 = ((r(d, d) / d**0.5).to(bf) for _ in range(2))
    return (r(rows, d), w1, w2, (1 + 0.1 * r(d)).to(bf), r(rows, d // 8), r(rows, d // 8), ids, slots,
            torch.rand(rows, 2, device="cuda", generator=g).to(bf))


@pytest.fixture(scope="module")
def ops():
    from autoparallel_b200.ops import cuda_impl, library

    cuda_impl.ensure_loaded()
    yield library.ops
    cuda_impl.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 8, 13])
def test_chains_of_short_launches_give_the_bits_of_separate_ones(ops, rows):
    for seed in range(20):
        state = _state(seed, rows)
        ref = _chain(ops, state, torch.cuda.synchronize)
        torch.cuda.synchronize()
        for _ in range(5):
            got = _chain(ops, state, lambda: None)
            assert all(torch.equal(a, b) for a, b in zip(got, ref))
        assert all(torch.isfinite(t).all() for t in ref)


@pytest.mark.gpu
def test_chains_across_two_streams(ops):
    """Every launch goes to the other stream than the one before it, behind an event."""
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for seed in range(10):
        state = _state(seed)
        ref = _chain(ops, state, torch.cuda.synchronize)
        torch.cuda.synchronize()
        turn, keep = [0], []

        def hop():
            e = torch.cuda.Event()
            e.record(streams[turn[0]])
            turn[0] ^= 1
            streams[turn[0]].wait_event(e)
            torch.cuda.set_stream(streams[turn[0]])

        before = torch.cuda.current_stream()
        try:
            torch.cuda.set_stream(streams[0])

            def kept(fn):  # (no memory is handed out again while the other stream may read it)
                def run(*args):
                    r = fn(*args)
                    keep.append((args, r))
                    return r
                return run

            class Kept:
                def __getattr__(self, name):
                    return kept(getattr(ops, name))

            got = _chain(Kept(), state, hop)
        finally:
            torch.cuda.set_stream(before)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, ref))


@pytest.mark.gpu
def test_captured_chains(ops):
    state = _state(0)
    ref = _chain(ops, state, torch.cuda.synchronize)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _chain(ops, state, lambda: None)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _chain(ops, state, lambda: None)
    for seed in range(5):
        for a, b in zip(state, _state(seed)):
            a.copy_(b)
        ref = [t.clone() for t in _chain(ops, state, torch.cuda.synchronize)]
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, ref))


def _edges(fn):
    """Edges between the launches of a captured graph: (overlapping, all)."""
    cudart = pytest.importorskip("cuda.bindings.runtime")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    raw = cudart.cudaGraph_t(graph.raw_cuda_graph())
    get = getattr(cudart, "cudaGraphGetEdges_v2", cudart.cudaGraphGetEdges)
    n = get(raw)[-1]
    err, _, _, data, _ = get(raw, n)
    assert err == cudart.cudaError_t.cudaSuccess
    kind = cudart.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic
    return sum(int(d.type) == int(kind) for d in data[:n]), n


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["dynamic", "stages", "reserved"])
def test_no_launch_overlaps_where_room_is_made(ops, mode):
    """Neither the products, nor those of a few rows, nor anything between them."""
    from autoparallel_b200.ops import cuda_impl

    ext = cuda_impl.extension()
    get, put, value = {"dynamic": (ext.gemm_get_dynamic_tiles, ext.gemm_set_dynamic_tiles, True),
                       "stages": (ext.gemm_get_pair_stages, ext.gemm_set_pair_stages, 5),
                       "reserved": (ext.gemm_get_reserved_sms, ext.gemm_set_reserved_sms, 8)}[mode]
    state, large = _state(0), torch.randn(2048, 512, device="cuda").to(torch.bfloat16)

    def work():
        _chain(ops, state, lambda: None)
        ops.swiglu(ops.mm_nd(large, state[1], True, torch.bfloat16), large)

    work()
    before = get()
    overlapping, n = _edges(work)
    assert overlapping > n // 2
    put(value)
    try:
        work()
        assert _edges(work)[0] == 0
    finally:
        put(before)
