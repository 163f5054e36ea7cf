"""The C++ gradient formulas of CUDA calls against the Python ones that every other device uses, and what must stay refused."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from autoparallel_b200.ops import cuda_impl, library

    cuda_impl.ensure_loaded()
    return library.ops


def _case(name):
    g = torch.Generator().manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    bf = torch.bfloat16
    idx = torch.rand(32, 8, generator=g).topk(2).indices
    slot = (torch.arange(64) % 40).reshape(32, 2)
    return {
        "dtype_cast": ((r(8, 16),), (bf,)),
        "mm_nd": ((r(2, 24, 64).to(bf), r(32, 64).to(bf)), (True, bf)),
        "mm_nd_kn": ((r(2, 24, 64).to(bf), r(64, 32).to(bf)), (False, bf)),
        "gemm": ((r(64, 24).to(bf), r(32, 64).to(bf)), (True, True, bf)),
        "grouped_mm": ((r(4, 24, 64).to(bf), r(4, 64, 32).to(bf)), (False, bf)),
        "rms_norm": ((r(9, 64).to(bf), r(64).to(bf)), (1e-5,)),
        "rope": ((r(2, 8, 4, 16).to(bf), r(8, 8), r(8, 8)), (False,)),
        "swiglu": ((r(9, 64).to(bf), r(9, 64).to(bf)), ()),
        "attention": ((r(1, 128, 4, 64).to(bf), r(1, 128, 2, 64).to(bf), r(1, 128, 2, 64).to(bf)), (True, 0.125)),
        "cross_entropy": ((r(9, 64).to(bf), torch.arange(9)), ()),
        "embedding": ((r(20, 64).to(bf), torch.arange(9) % 5), ()),
        "moe_scatter": ((r(32, 64).to(bf), torch.arange(64).reshape(32, 2), r(32, 2).to(bf)), (8, 8, 1)),
        "moe_gather": ((r(8, 1, 5, 64).to(bf), slot, r(32, 2).to(bf)), ()),
    }[name], idx


NAMES = ["dtype_cast", "mm_nd", "mm_nd_kn", "gemm", "grouped_mm", "rms_norm", "rope", "swiglu", "attention", "cross_entropy", "embedding",
         "moe_scatter", "moe_gather"]


def _op(ops, name):
    return getattr(ops, "mm_nd" if name == "mm_nd_kn" else name)


def _first(o):
    return o[0] if isinstance(o, tuple) else o


def _grads(ops, name, device):
    (tensors, rest), _ = _case(name)
    ins = [t.to(device) for t in tensors]
    diff = [t.requires_grad_() for t in ins if t.is_floating_point()]
    if name == "rope":
        diff = diff[:1]
        ins[1].requires_grad_(False), ins[2].requires_grad_(False)
    out = _first(_op(ops, name)(*ins, *rest))
    dy = torch.linspace(-1, 1, out.numel()).reshape(out.shape).to(out.dtype).to(device)
    return out, torch.autograd.grad(out, diff, dy), ins, rest


@pytest.mark.parametrize("name", NAMES)
def test_gradients_match_the_portable_formulas(ops, name):
    out, got, ins, _ = _grads(ops, name, "cuda")
    assert "CppNode" in type(out.grad_fn).__name__ or "torch::autograd" in out.grad_fn.name(), out.grad_fn.name()
    _, ref, _, _ = _grads(ops, name, "cpu")
    for a, b in zip(got, ref):
        assert a.dtype == b.dtype and a.shape == b.shape
        # bf16 operands and results, sums of at most 64 terms: a few roundings of 2^-9 relative to the norm
        assert ((a.cpu().double() - b.double()).norm() / b.double().norm()).item() <= 2**-6


@pytest.mark.parametrize("name", ["rms_norm", "attention", "cross_entropy"])
def test_the_second_output_has_no_gradient_of_its_own(ops, name):
    """Used alone it gives zeros, as the zeros that stood for the first one's gradient did; used beside the first it adds nothing."""
    (tensors, rest), _ = _case(name)
    ins = [t.cuda() for t in tensors]
    diff = [t.requires_grad_() for t in ins if t.is_floating_point()]
    for x in torch.autograd.grad(_op(ops, name)(*ins, *rest)[1].sum(), diff):
        assert x.abs().max().item() == 0
    first, second = _op(ops, name)(*ins, *rest)
    both = torch.autograd.grad(first.float().sum() + second.sum(), diff)
    alone = torch.autograd.grad(_op(ops, name)(*ins, *rest)[0].float().sum(), diff)
    # (one rounding apart at most: the library's attention backward may add up in another order)
    assert all((a - b).float().norm() <= 2**-8 * b.float().norm() for a, b in zip(both, alone))


@pytest.mark.parametrize("name", NAMES)
def test_no_gradient_is_recorded_when_none_is_asked_for(ops, name):
    (tensors, rest), _ = _case(name)
    ins = [t.cuda() for t in tensors]
    assert not _first(_op(ops, name)(*ins, *rest)).requires_grad
    with torch.no_grad():
        assert not _first(_op(ops, name)(*[t.requires_grad_() if t.is_floating_point() else t for t in ins], *rest)).requires_grad


def test_hooks_checkpointing_partial_and_second_gradients(ops):
    a = torch.randn(16, 64, device="cuda").bfloat16().requires_grad_()
    w = torch.randn(32, 64, device="cuda").bfloat16().requires_grad_()
    f = lambda a, w: ops.mm_nd(a, w, True, torch.bfloat16)  # noqa: E731
    dy = torch.randn(16, 32, device="cuda").bfloat16()
    ref = torch.autograd.grad(f(a, w), [a, w], dy)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        out = f(a, w)
    assert len(packed) == 2
    assert all(torch.equal(x, y) for x, y in zip(torch.autograd.grad(out, [a, w], dy), ref))
    out = torch.utils.checkpoint.checkpoint(f, a, w, use_reentrant=False)
    assert all(torch.equal(x, y) for x, y in zip(torch.autograd.grad(out, [a, w], dy), ref))
    assert torch.equal(torch.autograd.grad(f(a.detach(), w), [w], dy)[0], ref[1])
    (da,) = torch.autograd.grad(f(a, w), [a], dy, create_graph=True)
    (dw2,) = torch.autograd.grad(da, [w], torch.ones_like(da))  # d/dw of sum(dy w)
    assert ((dw2.float() - dy.float().sum(0).unsqueeze(1).expand(32, 64)).norm() / dw2.float().norm()).item() < 2**-6
    out = f(a, w)
    with torch.no_grad():
        w.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, [a], dy)


def test_transforms_stay_refused(ops):
    a = torch.randn(16, 64, device="cuda").bfloat16()
    w = torch.randn(32, 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: ops.mm_nd(t, w, True, torch.bfloat16).sum())(a)
    import torch.autograd.forward_ad as fwd

    with pytest.raises((RuntimeError, NotImplementedError)), fwd.dual_level():
        ops.mm_nd(fwd.make_dual(a.requires_grad_(), torch.ones_like(a)), w, True, torch.bfloat16)


@pytest.mark.parametrize("name", NAMES)
def test_every_recorded_call_refuses_transforms_and_forward_mode(ops, name):
    """As the Python registration does.  (A dual tensor in a call that records nothing loses its tangent, on every device: what is
    refused is the recorded form.)"""
    import torch.autograd.forward_ad as fwd

    (tensors, rest), _ = _case(name)
    first, *others = [t.cuda() for t in tensors]
    with pytest.raises(RuntimeError, match="functorch transforms"):
        torch.func.grad(lambda t: _first(_op(ops, name)(t, *others, *rest)).float().sum())(first)
    with pytest.raises((RuntimeError, NotImplementedError), match="jvp"), fwd.dual_level():
        _op(ops, name)(fwd.make_dual(first.requires_grad_(), torch.ones_like(first)), *others, *rest)


@pytest.mark.parametrize("shape", [(16, 64), (2, 8, 64)])
def test_a_projection_changed_in_place_keeps_its_gradient_or_refuses(ops, shape):
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(*shape, device="cuda", generator=g).bfloat16()
    w = torch.randn(32, 64, device="cuda", generator=g).bfloat16()
    want = 2 * w.double().sum(0).expand(shape)
    a.requires_grad_()
    y = ops.mm_nd(a, w, True, torch.bfloat16)
    try:
        y.mul_(2)
    except RuntimeError as e:
        assert "view" in str(e)
        return
    (da,) = torch.autograd.grad(y.float().sum(), a)
    assert ((da.double() - want).norm() / want.norm()).item() <= 2**-7


def test_modes_below_autograd_still_see_the_operators(ops):
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Log(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    x = torch.randn(9, 64, device="cuda").bfloat16().requires_grad_()
    w = torch.ones(64, device="cuda").bfloat16().requires_grad_()
    with Log():
        y = ops.rms_norm(x, w, 1e-5)[0]
        y.backward(torch.ones_like(y))
    assert "apb200.rms_norm.default" in seen and "apb200.rms_norm_bwd.default" in seen


def _entry_cases():
    r = lambda *s, dt=torch.bfloat16: torch.randn(*s, device="cuda").to(dt)
    f32, bf, f16 = torch.float32, torch.bfloat16, torch.float16
    idx = torch.randint(0, 6, (24, 2), device="cuda")
    slot = torch.randperm(48, device="cuda").clamp_(max=6 * 5).view(24, 2)  # every row once, the other assignments dropped
    return [
        ("mm_nd", (r(2, 5, 64), r(48, 64), True, bf)),
        ("mm_nd", (r(2, 5, 64)[:, ::2], r(64, 48), False, f32)),
        ("mm_nd", (r(4, 64), r(48, 64), True, f16)),             # a result type of the library's
        ("mm_nd", (r(4, 60, dt=f32), r(7, 60, dt=f32), True, f32)),  # operands of the library's
        ("mm_nd", (r(4, 64), r(50, 64), True, bf)),              # a width that is no whole vector
        ("mm_wgrad", (r(3, 8, 64), r(3, 8, 40), f32)),
        ("mm_wgrad", (r(24, 62), r(24, 40), bf)),
        ("grouped_mm", (r(3, 9, 64), r(3, 64, 40), False, bf)),
        ("grouped_mm", (r(3, 9, 64), r(3, 42, 64), True, bf)),
        ("grouped_mm_wgrad", (r(3, 9, 64), r(3, 9, 40).transpose(1, 2).contiguous().transpose(1, 2), f32)),
        ("grouped_mm_wgrad", (r(3, 9, 63), r(3, 9, 40), f32)),
        ("dtype_cast", (r(7, 16, dt=f32), bf)),
        ("dtype_cast", (r(7, 16, dt=f32)[:, 1:], bf)),
        ("dtype_cast", (r(7, 16), f32)),
        ("dtype_cast", (r(7, 16), f16)),
        ("dtype_cast", (torch.arange(9, device="cuda"), f32)),
        ("rms_norm", (r(2, 3, 64)[:, :2], r(64, dt=f32), 1e-5)),
        ("rms_norm_bwd", (r(6, 64), r(6, 64), r(64, dt=f32), r(6, dt=f32).abs())),
        ("rope", (r(2, 6, 4, 32), r(6, 16), r(6, 16), True)),
        ("swiglu", (r(6, 64).t().contiguous().t(), r(6, 64))),
        ("swiglu_bwd", (r(6, 64), r(6, 64).t().contiguous().t(), r(6, 64))),
        ("cross_entropy", (r(2, 5, 64)[:, 1:], torch.randint(0, 64, (2, 4), device="cuda"))),
        ("cross_entropy_bwd", (r(2, 4), r(2, 4, 64), torch.randint(0, 64, (2, 4), device="cuda"), r(2, 4, dt=f32))),
        ("embedding", (r(9, 64), torch.randint(0, 9, (2, 4), device="cuda"))),
        ("embedding", (r(9, 63), torch.randint(0, 9, (2, 4), device="cuda"))),
        ("embedding_bwd", (r(2, 4, 64, dt=f32), torch.randint(0, 9, (2, 4), device="cuda"), 9)),
        ("moe_slots", (idx, 6, 5, 2)),
        ("moe_slots", (idx, 9000, 5, 2)),                        # more experts than the kernel counts
        ("moe_scatter", (r(24, 16), slot, r(24, 2, dt=f32), 6, 5, 1)),
        ("moe_scatter", (r(24, 16, dt=f16), slot, r(24, 2, dt=f16), 6, 5, 1)),
        ("moe_gather", (r(6, 1, 5, 16), slot, r(24, 2, dt=f16))),
        ("moe_gather", (r(6, 1, 5, 16, dt=f16), slot, r(24, 2, dt=f16))),
        ("moe_gate_grad", (r(6, 1, 5, 16), slot, r(24, 16))),
        ("moe_gate_grad", (r(6, 1, 5, 16), slot, r(24, 16, dt=f32))),
    ]


def test_native_entries_answer_as_the_python_ones():
    """Every form: the same values, launches and library calls as the function of ops/cuda_impl.py that the entry stands for."""
    from autoparallel_b200.ops import cuda_impl, library, moe_ops  # noqa: F401

    cuda_impl.ensure_loaded()
    torch.manual_seed(0)
    for name, args in _entry_cases():
        results = []
        for fn in (getattr(library.ops, name), library._cuda_table[name]):
            launches, calls = cuda_impl.launch_count, dict(cuda_impl.library_fallbacks)
            out = fn(*args)
            out = out if isinstance(out, tuple) else (out,)
            library_calls = {k: v - calls.get(k, 0) for k, v in cuda_impl.library_fallbacks.items() if v != calls.get(k, 0)}
            results.append((out, cuda_impl.launch_count - launches, library_calls))
        (a, la, fa), (b, lb, fb) = results
        assert la == lb and fa == fb, name
        for x, y in zip(a, b, strict=True):
            assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride(), name
            if name == "embedding_bwd":  # (atomics in this form)
                assert torch.allclose(x, y, atol=1e-5), name
            else:
                assert torch.equal(x, y), name


def test_native_cast_hands_out_the_optimizers_copy():
    from autoparallel_b200.ops import library, shadow

    p, copy = torch.randn(8, 16, device="cuda"), torch.zeros(8, 16, device="cuda", dtype=torch.bfloat16)
    shadow.clear()
    assert torch.equal(library.ops.dtype_cast(p, torch.bfloat16), p.bfloat16())
    shadow.publish(p, copy)
    try:
        assert library.ops.dtype_cast(p, torch.bfloat16).data_ptr() == copy.data_ptr()
        p.mul_(2)  # no longer what was copied
        assert torch.equal(library.ops.dtype_cast(p, torch.bfloat16), p.bfloat16())
    finally:
        shadow.clear()
    assert torch.equal(library.ops.dtype_cast(p, torch.bfloat16), p.bfloat16())


@pytest.mark.parametrize("name", [
    "mm_nd", "mm_wgrad", "grouped_mm", "grouped_mm_wgrad", "dtype_cast", "rms_norm", "rms_norm_bwd", "rope", "swiglu", "swiglu_bwd", "cross_entropy",
    "cross_entropy_bwd", "embedding", "embedding_bwd", "moe_slots", "moe_scatter", "moe_gather", "moe_gate_grad"])
def test_an_installed_wrapper_is_what_the_next_call_runs(name):
    """register_cuda_impl after the extension is loaded: the operator runs the function, and the kernel again once its own is back."""
    from autoparallel_b200.ops import cuda_impl, library, register_cuda_impl

    cuda_impl.ensure_loaded()
    torch.manual_seed(0)
    own = library._cuda_table[name]
    args = next(a for n, a in _entry_cases() if n == name)
    want = getattr(library.ops, name)(*args)
    calls = []

    def mine(*a):
        calls.append(len(a))
        return own(*a)

    def equal(x, y):
        x, y = (x, y) if isinstance(x, tuple) else ((x,), (y,))
        same = (lambda p, q: torch.allclose(p, q, atol=1e-5)) if name == "embedding_bwd" else torch.equal  # (atomics)
        return all(map(same, x, y))

    register_cuda_impl(name, mine)
    try:
        assert equal(getattr(library.ops, name)(*args), want) and calls == [len(args)]
    finally:
        register_cuda_impl(name, own)
    assert equal(getattr(library.ops, name)(*args), want) and calls == [len(args)]
