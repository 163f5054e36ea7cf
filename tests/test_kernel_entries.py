"""The extension's C entries on arguments that they answer without a GPU."""
import ctypes
import os
import subprocess
import sys
import threading
import time
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from autoparallel_b200.ops import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
needs_ext = pytest.mark.skipif(not os.path.exists(build.so_path()), reason="the extension is not built")


def _run(code):
    """In a process of its own: a fault in an entry ends the process."""
    head = "import ctypes, torch\nfrom autoparallel_b200.ops import build\nso = ctypes.CDLL(build.so_path())\n"
    r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    return r.stdout.split()


@needs_ext
def test_slot_workspace_of_an_empty_dispatch():
    """No choices, no tokens, no experts: no workspace, and no division by the empty size."""
    out = _run(
        "f = so.apb_moe_slots_workspace\nf.restype = ctypes.c_longlong\n"
        "print(f(1, 0, 8, 148), f(0, 16, 8, 148), f(1, 16, 0, 148), f(2, 1024, 8, 148) > 0)"
    )
    assert out == ["0", "0", "0", "True"]


@needs_ext
def test_wide_tiles_take_hardly_more_waves():
    """A product goes to tiles of two column tiles only where a pair's share of them is at most a seventh larger, with an odd number
    of column tiles a twentieth (74 pairs)."""
    import random

    def halves(tiles, columns, units):  # of column tiles that a pair goes through; a last wave that fits runs in halves
        whole, rest = divmod(tiles, units)
        return 2 * columns * whole + (0 if rest == 0 else columns if 2 * rest <= units else 2 * columns)

    rng = random.Random(7)
    wide = [(0, 8192, 4096, 8192), (0, 8192, 4096, 128256), (0, 128256, 4096, 8192), (0, 8192, 10240, 8192), (0, 5896, 4104, 6552),
            (10, 2304, 4104, 8200), (0, 4096, 4096, 8192), (0, 16384, 1024, 6144)]
    narrow = [(0, 32768, 256, 8192), (0, 16384, 768, 8192), (0, 8192, 1280, 8192), (0, 4096, 2304, 5120), (0, 4096, 3328, 8192),
              (0, 8192, 4096, 4096), (0, 4096, 2560, 8192), (0, 8192, 1792, 8192), (0, 2048, 5120, 11008)]
    drawn = [(rng.choice((0, 0, 4, 16)), rng.randrange(256, 40000), rng.randrange(64, 20000), rng.randrange(4096, 20000))
             for _ in range(400)]
    shapes = wide + narrow + drawn
    code = "i3 = (ctypes.c_int * 3)()\n" + f"for s in {shapes!r}:\n    so.apb_gemm_pair_tiles(*s, 74, i3)\n    print(*i3)\n"
    out = [int(x) for x in _run(code)]
    taken = 0
    for i, (G, M, N, K) in enumerate(shapes):
        is_wide, tiles, whole = out[3 * i:3 * i + 3]
        m, n = -(-M // 256) * max(G, 1), -(-N // 256)
        assert tiles == m * (-(-n // 2) if is_wide else n) and 0 <= whole <= tiles and 2 * tiles - whole >= tiles
        assert whole == tiles or (whole % 74 == 0 and 2 * (tiles - whole) <= 74)
        taken += is_wide
        if is_wide:
            more, of = (21, 20) if n % 2 else (8, 7)
            assert n > 1 and of * halves(tiles, 2, 74) <= more * halves(m * n, 1, 74), (G, M, N, K)
    assert out[:3 * len(wide):3] == [1] * len(wide) and not any(out[3 * len(wide):3 * len(wide + narrow):3])
    assert 20 < taken < 380


@needs_ext
def test_products_of_a_few_rows_go_to_the_faster_kernel():
    """Sizes on both sides of the line, each timed with both kernels (148 SMs); what the few-row kernel cannot take stays out."""
    rows = [(8, 256, 256), (8, 4096, 4096), (8, 32064, 4096), (8, 14336, 1024), (1, 512, 8192), (8, 1024, 8192), (16, 256, 2048),
            (16, 2048, 2048), (16, 4096, 4096), (16, 6144, 512), (16, 14336, 1024), (32, 1024, 1024), (24, 2048, 2048),
            (32, 4096, 1024), (17, 64, 64)]
    split = [(8, 14336, 256), (8, 32064, 512), (8, 256, 8192), (8, 6144, 8192), (1, 256, 14336), (16, 512, 4096), (16, 14336, 512),
             (16, 4096, 8192), (32, 1024, 2048), (32, 6144, 256), (32, 14336, 256), (32, 2048, 4096), (17, 1024, 64)]
    never = [(33, 1024, 1024), (8, 256, 252), (0, 256, 256), (8, 0, 256), (8, 256, 0), (8, 256, -8)]
    out = _run(f"for s in {rows + split + never!r}:\n    print(so.apb_gemm_rows_takes(*s, 148))\n")
    assert out == ["1"] * len(rows) + ["0"] * len(split + never)


@needs_ext
def test_the_extension_brings_no_cxx_library_of_its_own():
    """With a static copy inside, an error with a number in its message ends the process (see ops/build.py)."""
    with open(build.so_path(), "rb") as f:
        assert b"\0libstdc++.so.6\0" in f.read()


@needs_ext
def test_entries_refuse_bases_off_a_16_byte_boundary():
    """The kernels move 16 bytes at a time; nothing is launched (there is no GPU here to launch on: that would be code 4)."""
    out = _run("""
V, LL, F, N = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_float, None
A = 1 << 20  # never read
def entry(name, args, pointers):
    f = getattr(so, name)
    if not torch.cuda.is_available():
        assert f(*args) == 4, (name, "an aligned call gets as far as the launch", f(*args))
    for i in pointers:
        bad = list(args)
        bad[i] = V(A + 8)
        print(f(*bad))
p = V(A)
entry("apb_rms_norm_fwd", [p, p, p, p, LL(4), 64, F(1e-5), 1, N], [0, 1, 2])
entry("apb_rms_norm_bwd", [p, p, p, p, p, p, p, LL(4), 64, 1, 148, N], [0, 1, 2, 4])
entry("apb_cast", [p, p, LL(64), 0, 1, 148, N], [0, 1])
entry("apb_rope", [p, p, p, p, LL(1), 4, 2, 64, 0, 1, 148, N], [0, 1, 2, 3])
entry("apb_swiglu_fwd", [p, p, p, LL(64), 1, 148, N], [0, 1, 2])
entry("apb_swiglu_bwd", [p, p, p, p, p, LL(64), 1, 148, N], [0, 1, 2, 3, 4])
entry("apb_xent_fwd", [p, p, p, p, LL(4), 64, 1, N], [0])
entry("apb_xent_bwd", [p, p, p, p, p, LL(4), 64, 1, N], [1, 4])
entry("apb_embedding_fwd", [p, p, p, LL(4), 64, LL(8), 1, N], [0, 2])
""")
    assert out == ["3"] * 26
    out = _run("""
V, LL = ctypes.c_void_p, ctypes.c_longlong
p, bad = V(1 << 20), V((1 << 20) + 8)
for i in (0, 1, 2, 4, 5):
    a = [p] * 6
    a[i] = bad
    print(so.apb_rms_norm_bwd_noalloc(*a, LL(4), 64, 1, None))
""")
    assert out == ["9"] * 5


@needs_ext
def test_pair_gemm_with_fewer_stages_leaves_their_shared_memory():
    """What the switch is for: room for a communication kernel's CTA beside a GEMM CTA (32 KB a stage, nothing else in their place)."""
    out = _run("print(*[so.apb_gemm_pair_smem_bytes(s) for s in (4, 5, 6)])")
    four, five, six = map(int, out)
    assert (four, five) == (4 * 32768 + 1280, 5 * 32768 + 1280) and six <= 227 * 1024


def test_one_status_word_per_device_whichever_thread_is_first(monkeypatch):
    """Both sides of the binding keep the word they got first: two threads at the first use of a device must get the same one."""
    from autoparallel_b200.ops import cuda_impl

    together = threading.Barrier(2)

    def zeros(*shape, **kw):  # (stands in for the device; slow enough for the other thread to come past the look-up)
        time.sleep(0.3)
        return torch.empty(*shape, dtype=kw["dtype"])

    def first_use(_):
        together.wait(timeout=10)
        return cuda_impl.status_buffer(torch.device("cuda", 0))

    monkeypatch.setattr(cuda_impl, "_status", {})
    monkeypatch.setattr(cuda_impl.torch, "zeros", zeros)
    with ThreadPoolExecutor(2) as pool:
        first, second = pool.map(first_use, range(2))
    assert first is second is cuda_impl.status_buffer(torch.device("cuda", 0))
