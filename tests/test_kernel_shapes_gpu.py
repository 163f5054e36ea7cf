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


def test_embedding_gradient_of_an_unaligned_view(K):
    lib, _ = K
    flat = torch.randn(1 + 12 * 16, device="cuda").to(torch.bfloat16)
    dy, idx = flat[1:].view(12, 16), torch.arange(12, device="cuda") % 5
    ref = torch.zeros(5, 16, dtype=torch.float64).index_add_(0, idx.cpu(), dy.double().cpu())
    assert _rel(lib.ops.embedding_bwd(dy, idx, 5), ref) <= 2**-8
