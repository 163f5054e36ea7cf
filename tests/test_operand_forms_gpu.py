"""Operand forms at the edge of what the kernels read - one row, views, empty sizes - against the CPU formulas."""
import copy

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


BF16_TOL = 2**-8  # fp32 sums of a few hundred products, one rounding to bf16


@pytest.mark.parametrize("row", [
    lambda g: torch.randn(3, 67, generator=g)[0:1, :64],   # odd leading stride
    lambda g: torch.randn(64, 1, generator=g).t(),         # strides (1, 1)
    lambda g: torch.randn(1, 130, generator=g)[:, ::2][:, :64],  # every other element
])
def test_products_with_a_single_row_of_any_stride(K, row):
    """``contiguous()`` ignores the stride of a dimension of size one; a tensor map does not."""
    lib, impl = K
    g = torch.Generator().manual_seed(0)
    a, w, dy = row(g).bfloat16(), torch.randn(96, 64, generator=g).bfloat16(), torch.randn(1, 96, generator=g).bfloat16()
    assert a.shape == (1, 64)
    ad = torch.empty_strided(a.size(), a.stride(), dtype=a.dtype, device="cuda").copy_(a)
    before = dict(impl.library_fallbacks)
    assert _rel(lib.ops.mm_nd(ad, w.cuda(), True, torch.bfloat16), a.double() @ w.double().t()) <= BF16_TOL
    assert _rel(lib.ops.mm_nd(dy.cuda(), w.cuda(), False, torch.bfloat16), dy.double() @ w.double()) <= BF16_TOL
    assert _rel(lib.ops.mm_wgrad(dy.cuda(), ad, torch.float32), dy.double().t() @ a.double()) <= 2**-22  # one product per element
    assert _rel(lib.ops.mm_wgrad(ad, dy.cuda(), torch.float32), a.double().t() @ dy.double()) <= 2**-22
    assert impl.library_fallbacks == before


def test_matrices_without_columns_stay_refused(K):
    lib, _ = K
    with pytest.raises(RuntimeError, match="cannot reshape tensor of 0 elements"):
        lib.ops.mm_nd(torch.empty(4, 0, device="cuda", dtype=torch.bfloat16), torch.empty(8, 0, device="cuda", dtype=torch.bfloat16), True,
                      torch.bfloat16)


def test_slots_without_choices_stay_refused(K):
    lib, _ = K
    with pytest.raises(RuntimeError, match="apb_moe_slots"):
        lib.ops.moe_slots(torch.empty(16, 0, device="cuda", dtype=torch.long), 4, 8, 1)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_contractions_over_no_tokens_are_zero(K, out_dtype):
    """A weight gradient when no token arrived (an expert's or a rank's share of a batch), over memory that held something else."""
    lib, _ = K
    a, b = torch.empty(0, 64, device="cuda", dtype=torch.bfloat16), torch.empty(0, 96, device="cuda", dtype=torch.bfloat16)
    ga, gb = torch.empty(3, 0, 64, device="cuda", dtype=torch.bfloat16), torch.empty(3, 0, 96, device="cuda", dtype=torch.bfloat16)
    for shape, f in [
        ((64, 96), lambda: lib.ops.mm_wgrad(a, b, out_dtype)),
        ((64, 96), lambda: lib.ops.mm_wgrad(a.view(2, 0, 64), b.view(2, 0, 96), out_dtype)),
        ((64, 96), lambda: lib.ops.gemm(a, b, True, False, out_dtype)),
        ((3, 64, 96), lambda: lib.ops.grouped_mm_wgrad(ga, gb, out_dtype)),
        ((3, 8, 96), lambda: lib.ops.grouped_mm(ga.view(3, 64, 0)[:, :8], gb, False, out_dtype)),
    ]:
        for _ in range(2):
            junk = torch.full(shape, float("nan"), device="cuda", dtype=out_dtype)
            del junk  # (what the result is allocated over)
            out = f()
            assert out.shape == shape and out.dtype == out_dtype and not out.any()
    assert lib.ops.mm_nd(a, torch.ones(96, 64, device="cuda", dtype=torch.bfloat16), True, out_dtype).shape == (0, 96)
    # a window of a wider matrix: nothing beside it is touched
    from autoparallel_b200.ops import cuda_impl

    back = torch.full((6, 32), 7.0, device="cuda", dtype=out_dtype)
    cuda_impl.extension().gemm(torch.empty(0, 4, device="cuda", dtype=torch.bfloat16), b[:, :16], back[1:5, 8:24], True, True, cuda_impl.status_buffer(back.device))
    assert not back[1:5, 8:24].any()
    back[1:5, 8:24] = 7.0
    assert bool((back == 7.0).all())


def _off(t, elements=1):
    """``t`` as a dense view that starts ``elements`` past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
    v = flat[elements:elements + t.numel()].view(t.shape)
    assert v.is_contiguous() and v.data_ptr() % 16 != 0
    return v.copy_(t)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_dense_views_off_a_16_byte_boundary(K, dtype):
    """``contiguous()`` returns such a view as it is; the kernels' accesses are 16 bytes wide."""
    lib, _ = K
    from autoparallel_b200.ops import library

    g = torch.Generator().manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype)  # noqa: E731
    tol = BF16_TOL if dtype == torch.bfloat16 else 2**-16  # (fp32: the hardware exponential and reciprocal square root)
    ref = library.reference_impls
    x, w, dy = r(9, 64), r(64), r(9, 64)
    cases = [
        ("rms_norm", (x, w), (1e-5,)),
        ("rms_norm_bwd", (dy, x, w), (torch.rand(9, generator=g) + 0.5,)),
        ("rope", (r(2, 8, 4, 16), torch.randn(8, 8, generator=g), torch.randn(8, 8, generator=g)), (False,)),
        ("swiglu", (x, dy), ()),
        ("swiglu_bwd", (dy, x, r(9, 64)), ()),
        ("cross_entropy", (x,), (torch.arange(9),)),
        ("cross_entropy_bwd", (torch.rand(9, generator=g), x), (torch.arange(9), torch.logsumexp(x.float(), -1))),
        ("embedding", (r(20, 64),), (torch.arange(9) % 5,)),
        ("embedding_bwd", (dy,), (torch.arange(9) % 5, 20)),
        ("dtype_cast", (x,), (torch.float32 if dtype == torch.bfloat16 else torch.bfloat16,)),
    ]
    if dtype == torch.bfloat16:
        cases += [
            ("mm_nd", (r(2, 9, 64), r(32, 64)), (True, dtype)),
            ("mm_wgrad", (r(9, 64), r(9, 32)), (dtype,)),
            ("gemm", (r(64, 24), r(32, 64)), (True, True, dtype)),
            ("grouped_mm", (r(3, 9, 64), r(3, 64, 32)), (False, dtype)),
            ("grouped_mm_wgrad", (r(3, 9, 64), r(3, 9, 32)), (dtype,)),
        ]
    for name, tensors, rest in cases:
        want = ref[name](*tensors, *rest)
        rest = [t.cuda() if isinstance(t, torch.Tensor) else t for t in rest]
        for i in range(len(tensors)):  # each operand in turn, and a clean run beside it
            args = [_off(t) if j == i else t.cuda() for j, t in enumerate(tensors)]
            got = getattr(lib.ops, name)(*args, *rest)
            for a, b in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
                assert _rel(a, b) <= tol, (name, i)


def test_adamw_steps_on_the_loaded_state(K):
    """Parameters and gradients keep their addresses when a state is loaded; the moments are other tensors."""
    from autoparallel_b200.optim import AdamW

    g = torch.Generator().manual_seed(3)
    p0, g0 = torch.randn(1000, generator=g), torch.randn(1000, generator=g)

    def make(first):
        p = torch.nn.Parameter(p0.cuda())
        opt = AdamW([p], lr=1e-2)
        p.grad = (first * g0).cuda()
        opt.step()
        with torch.no_grad():
            p.copy_(p0)
            p.grad.copy_(g0)
        return p, opt

    p, opt = make(1.0)
    q, other = make(-3.0)
    opt.load_state_dict(copy.deepcopy(other.state_dict()))
    opt.step(), other.step()
    assert torch.equal(p, q)
    for k in ("exp_avg", "exp_avg_sq"):
        assert torch.equal(opt.state[p][k], other.state[q][k])


def test_adamw_where_other_parameters_have_gradients_each_step(K):
    """One at a time, large after small and small after large."""
    from autoparallel_b200.optim import AdamW

    g = torch.Generator().manual_seed(4)
    sizes = [5, 200000, 1024, 70001]
    own = [torch.nn.Parameter(torch.randn(n, generator=g).cuda()) for n in sizes]
    ref = [torch.nn.Parameter(p.detach().cpu().double()) for p in own]
    opt, std = (cls(ps, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1) for cls, ps in ((AdamW, own), (torch.optim.AdamW, ref)))
    for i in (0, 1, 0, 2, 3, 2, 1):
        grad = torch.randn(sizes[i], generator=g)
        for j, (p, q) in enumerate(zip(own, ref)):
            p.grad, q.grad = (grad.cuda(), grad.double()) if j == i else (None, None)
        opt.step(), std.step()
    for p, q in zip(own, ref):
        assert _rel(p.detach(), q.detach()) <= 2**-20  # fp32 steps of the size of lr


@pytest.mark.parametrize("odd", ["param", "grad", "exp_avg", "exp_avg_sq"])
def test_adamw_takes_views_off_a_16_byte_boundary(K, odd):
    """A parameter, gradient or state out of a flat buffer: the same step as on tensors of their own."""
    from autoparallel_b200.optim import AdamW

    g = torch.Generator().manual_seed(2)
    n = 70001  # two chunks of the kernel, and a tail
    t = {k: torch.randn(n, generator=g) for k in ("param", "grad", "exp_avg")}
    t["exp_avg_sq"] = torch.rand(n, generator=g)

    def step(view):
        v = {k: (_off(x) if view and k == odd else x.cuda()) for k, x in t.items()}
        p = torch.nn.Parameter(v["param"])
        opt = AdamW([p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
        p.grad = v["grad"]
        opt._init_state(p)
        opt.state[p]["exp_avg"], opt.state[p]["exp_avg_sq"] = v["exp_avg"], v["exp_avg_sq"]
        opt.step()
        return p.detach(), opt.state[p]["exp_avg"], opt.state[p]["exp_avg_sq"]

    for a, b in zip(step(True), step(False)):
        assert _rel(a, b) <= 2**-21  # (the vector and the scalar path round a product and sum differently, a few ulp)
