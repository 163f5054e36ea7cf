"""init_weights interception (both modes), tied parameters, buffer re-assignment and parameter shard layout."""
import pytest
import torch
import torch.nn as nn
from torch.distributed.tensor import DTensor
from torch.distributed.tensor.placement_types import Shard

from autoparallel_b200 import AutoParallel
from autoparallel_b200.parallel.lower.init_weights import wrap_init_weights


class Net(nn.Module):
    def __init__(self, v=64, d=32):
        super().__init__()
        self.emb = nn.Embedding(v, d)
        self.mid = nn.Linear(d, d)
        self.out = nn.Linear(d, v, bias=False)
        self.out.weight = self.emb.weight  # tied
        self.register_buffer("table", torch.zeros(v))

    def forward(self, t):
        return self.out(torch.relu(self.mid(self.emb(t)))) + self.table

    def init_weights(self, value=0.5):
        with torch.no_grad():
            nn.init.constant_(self.mid.weight, value)          # in-place initialiser
            self.mid.bias.copy_(torch.arange(32.0))            # copy_ from a plain tensor
            self.emb.weight = nn.Parameter(torch.arange(64.0 * 32).view(64, 32))   # slot re-assignment (tied slot)
            self.table = torch.arange(64.0)                    # buffer re-assignment
        return "done"


def _build(mesh):
    with torch.device("meta"):
        m = Net()
    with AutoParallel(m, lambda: torch.randint(0, 64, (16, 8)), mesh) as ap:
        ap.add_parameter_memory_constraint()
        ap.add_input_constraints([(Shard(0),)])
        ap.optimize_placement()
        pm = ap.apply_placement()
    pm.to_empty(device="cpu")
    return pm


@pytest.mark.parametrize("mode", ["materialize", "intercept"])
def test_init_weights_modes_give_the_same_sharded_values(mesh_1d, mode):
    pm = _build(mesh_1d)
    del pm.__dict__["init_weights"]
    wrap_init_weights(pm, mode=mode)
    assert pm.init_weights(value=0.25) == "done"  # arguments and the return value pass through
    assert isinstance(pm.mid.weight, DTensor) and isinstance(pm.table, DTensor)  # slots still hold the sharded tensors
    assert pm.out.weight is pm.emb.weight  # tie survives the re-assignment
    # fake ranks do not exchange data: check what rank 0 holds, the first shard of each global value
    def first_shard(dt, full):
        for i, pl in enumerate(dt.placements):
            if isinstance(pl, Shard):
                full = full.chunk(mesh_1d.shape[i], pl.dim)[0]
        return full

    assert torch.all(pm.mid.weight._local_tensor == 0.25)
    assert torch.equal(pm.mid.bias._local_tensor, first_shard(pm.mid.bias, torch.arange(32.0)))
    assert torch.equal(pm.emb.weight._local_tensor, first_shard(pm.emb.weight, torch.arange(64.0 * 32).view(64, 32)))
    assert torch.equal(pm.table._local_tensor, first_shard(pm.table, torch.arange(64.0)))
    assert pm.emb.weight.requires_grad
    assert any(isinstance(pl, Shard) for pl in pm.emb.weight.placements)  # the memory constraint shards it


def test_init_weights_shape_change_is_refused(mesh_1d):
    pm = _build(mesh_1d)

    def bad_init():
        pm.mid.weight = nn.Parameter(torch.zeros(3, 3))

    pm.__dict__["init_weights"] = None
    pm.init_weights = bad_init
    wrap_init_weights(pm, mode="materialize")
    with pytest.raises(RuntimeError, match="changed the shape"):
        pm.init_weights()


def test_gradients_of_all_shards_come_from_one_node(mesh_1d):
    """What one ``to_local`` per parameter gave: placements, partial and frozen gradients, hooks, no recording without gradients."""
    from autoparallel_b200.api import _as_shard, _local_params

    pm = _build(mesh_1d)
    names = [n for n, _ in pm.named_parameters()]
    params = [p for _, p in pm.named_parameters()]
    with torch.no_grad():
        for p in params:
            p.to_local().copy_(torch.arange(p.to_local().numel()).view_as(p.to_local()))
        assert all(t is p._local_tensor for t, p in zip(_local_params(params), params))  # nothing is recorded
    pm.mid.bias.requires_grad_(False)
    seen = []
    pm.mid.weight.register_hook(lambda g: seen.append(type(g)))
    shards = _local_params(params)
    assert len({id(s.grad_fn) for s in shards if s.requires_grad}) == 1
    for s, p in zip(shards, params):
        assert torch.equal(s, p.to_local()) and s.data_ptr() == p.to_local().data_ptr()
    sum((i + 2) * s.sum() for i, s in enumerate(shards)).backward(retain_graph=True)
    for i, (n, p) in enumerate(zip(names, params)):
        if n == "mid.bias":
            assert p.grad is None
            continue
        assert isinstance(p.grad, DTensor) and p.grad.placements == p.placements
        assert p.grad.shape == p.shape and p.grad.stride() == p.stride()
        assert torch.all(p.grad.to_local() == i + 2)
    assert seen == [DTensor]
    w = names.index("mid.weight")
    (g,) = torch.autograd.grad(shards[w].square().sum(), [params[w]])
    assert torch.equal(g.to_local(), 2 * params[w].to_local())
    with torch.no_grad():
        shards = _local_params(params)
    assert not any(s.requires_grad for s in shards)
    y = _local_params(params)[w].square().sum()
    with torch.no_grad():
        params[w].to_local().add_(1)  # a change between forward and backward is noticed
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()
    local = params[w].to_local()
    turned = _as_shard(torch.ones(local.shape[::-1]).t(), params[w]._spec, local.stride())  # a gradient laid out otherwise
    assert turned.to_local().is_contiguous() and turned.shape == params[w].shape and turned.stride() == params[w].stride()

