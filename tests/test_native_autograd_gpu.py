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
