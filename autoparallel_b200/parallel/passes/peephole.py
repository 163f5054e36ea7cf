"""Local rewrites on the lowered graph that remove memory round trips.

* ``dtype_cast(gemm_like(a, b, .., bf16), fp32)`` with a single consumer becomes the GEMM with an
  fp32 epilogue: the weight-gradient GEMM writes the fp32 gradient the reduce-scatter wants
  directly (one full read+write of every gradient less, and no bf16 rounding before the
  reduction).
* small parameters' ``dtype_cast``s to bf16 become one ``cast_many`` at the head of a graph without collectives: a launch
  and 7 us of host time for each of them otherwise, twice a step.
"""
from __future__ import annotations

import operator

import torch
import torch.fx as fx

apb = torch.ops.apb200

_GEMM_OUT_DTYPE_POS = {apb.mm_wgrad.default: 2, apb.mm_nd.default: 3, apb.gemm.default: 4}


def fuse_cast_into_gemm(gm: fx.GraphModule) -> int:
    n_fused = 0
    for n in list(gm.graph.nodes):
        if n.op != "call_function" or n.target is not apb.dtype_cast.default:
            continue
        src = n.args[0]
        if not (isinstance(src, fx.Node) and src.op == "call_function" and src.target in _GEMM_OUT_DTYPE_POS):
            continue
        if len(src.users) != 1 or n.args[1] not in (torch.float32, torch.bfloat16):
            continue
        pos = _GEMM_OUT_DTYPE_POS[src.target]
        args = list(src.args)
        args[pos] = n.args[1]
        src.args = tuple(args)
        src.meta["val"] = n.meta["val"]
        n.replace_all_uses_with(src)
        gm.graph.erase_node(n)
        n_fused += 1
    if n_fused:
        gm.graph.lint()
        gm.recompile()
    return n_fused


# Largest tensor (elements) that is cast with others - its own launch is worth as much as its bytes then, 1.7 us - and the elements that one
# graph casts at its head: their copies live from there to their last use.
CAST_TOGETHER, CAST_AT_HEAD = 1 << 20, 1 << 24


def merge_parameter_casts(gm: fx.GraphModule) -> int:
    """Returns the number of casts that became one.  Graphs with collectives are left alone: there a cast feeds the gather that the
    overlap scheduler places."""
    from ...runtime import comm_ops

    nodes = list(gm.graph.nodes)
    if any(n.op == "call_function" and n.target in comm_ops.COLLECTIVE_OPS for n in nodes):
        return 0
    casts, elements = [], 0
    for n in nodes:
        if n.op != "call_function" or n.target is not apb.dtype_cast.default:
            continue
        if n.args[1] is not torch.bfloat16 or n.args[0].op != "placeholder":
            continue
        val = n.args[0].meta.get("val")
        if not isinstance(val, torch.Tensor) or val.dtype is not torch.float32 or not all(isinstance(d, int) for d in val.shape):
            continue
        if val.numel() > CAST_TOGETHER or elements + val.numel() > CAST_AT_HEAD:
            continue
        casts.append(n)
        elements += val.numel()
    if len(casts) < 2:
        return 0
    last = [n for n in nodes if n.op == "placeholder"][-1]
    with gm.graph.inserting_after(last):
        many = gm.graph.call_function(apb.cast_many.default, ([n.args[0] for n in casts], torch.bfloat16))
    many.meta["val"] = [n.meta.get("val") for n in casts]
    after = many
    for i, n in enumerate(casts):
        with gm.graph.inserting_after(after):
            item = gm.graph.call_function(operator.getitem, (many, i))
        item.meta.update(n.meta)
        n.replace_all_uses_with(item)
        gm.graph.erase_node(n)
        after = item
    gm.graph.lint()
    gm.recompile()
    return len(casts)
