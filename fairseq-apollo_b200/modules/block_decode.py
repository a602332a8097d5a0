"""Single-token decoding of the causal Mega block in one library call (mega_block_step): the L == 1 case of
MovingAverageGatedAttention.forward with an incremental state
(fairseq/modules/moving_average_gated_attention.py:282-414).

The keys and values of a chunk live in buffers with room for more than there are; the state's ``prev_key`` /
``prev_value`` are views of their first rows, so a step appends a row instead of copying the cache.  Rows that a
view covers are never written again: a step appends only behind the views that the step before handed out, and
any other state (a new generation, reordered beams, a copied state) gets buffers of its own.  They go with the state.
"""
from typing import Optional

import torch
from torch import Tensor
from torch.nn.modules.module import _has_any_global_hook

from .. import _lib, ops
from ..block_function import _own, projections_plain
from ..ops import _raw_stream
from .fused import _ema_params, _param_names, _seed_decode_state

_POLES = {False: (4, 8, 16, 32), True: (2, 4, 8, 16, 32)}


# submodules that a step stands for (from the third on it stands for calling them, so they have to be without hooks and
# forwards of their own, at every step), and the parameters it takes: (owner, 0 the block itself, then in this order; name)
_SUBMODULES = ("norm", "move", "v_proj", "mx_proj", "h_proj", "efficient_attn", "rel_pos_bias")


def _names(blk):
    n = _param_names(blk.move)
    return [(1, n[0]), (1, n[1]), (2, n[2]), (2, n[3]), (2, n[4]), (2, n[5]), (2, n[6]), (3, 'weight'), (3, 'bias'),
            (4, 'weight'), (4, 'bias'), (5, 'weight'), (0, 'gamma'), (0, 'beta')]


def applicable(blk, x) -> bool:
    """Whether the block and x (B, 1, D) are in the step's envelope (checked once per plan)."""
    norm, move = blk.norm, blk.move
    weights = (blk.v_proj.weight, blk.v_proj.bias, blk.mx_proj.weight, blk.mx_proj.bias, blk.h_proj.weight)
    chunk = blk.chunk_size
    return (blk.efficient_attn is not None and _own(blk.efficient_attn, "EfficientAttention") and projections_plain(blk)
            and isinstance(blk.move_act, torch.nn.SiLU) and _own(blk.rel_pos_bias, "RotaryEmbedding") and not move.bidirectional
            and norm.num_groups in (None, norm.num_features) and move.ndim in _POLES[move.complex]
            and (chunk < 0 or chunk > 1) and x.dtype in (torch.bfloat16, torch.float16)
            and all(w is not None and w.dtype == x.dtype and w.is_cuda and w.is_contiguous() and w.data_ptr() % 16 == 0
                    for w in weights)
            and blk.gamma.dtype == blk.beta.dtype and blk.gamma.dtype in (torch.float32, x.dtype)
            and blk.gamma.is_contiguous() and blk.beta.is_contiguous()
            and x.size(0) <= 64 and blk.zdim in (64, 128, 256) and blk.embed_dim % 32 == 0 and blk.hdim % 32 == 0
            and x.size(0) * (max(blk.embed_dim, blk.hdim) * 2 + 64) <= 200 * 1024)


def step(blk, x: Tensor, incremental_state) -> Optional[Tensor]:
    """One token through the block, or None when the call is not the library's (the caller then runs the
    block's own sequence of operations).  Called with gradients disabled, x (B, 1, D) contiguous, no masks."""
    if _has_any_global_hook() or torch.is_autocast_enabled():
        return None
    if x.data_ptr() % 16:   # (a slice of a larger tensor: the step reads whole 16-byte pieces)
        x = x.clone()
    out = _lib.host().block_step(blk, x, incremental_state)
    if out is None and _build(blk, x, _raw_stream(x.device.index), incremental_state):
        out = _lib.host().block_step(blk, x, incremental_state)
        if out is None:
            raise RuntimeError("single-token step: a freshly built plan does not match its own inputs")
    return out


def _build(blk, x, stream, incremental_state):
    if not applicable(blk, x):
        return False
    norm, move = blk.norm, blk.move
    bsz, _, dim = x.shape
    dev = x.device
    akey = blk._get_full_incremental_state_key("attn_state")
    astate = incremental_state.get(akey) or {}
    k, v = astate.get("prev_key"), astate.get("prev_value")
    if astate.get("prev_key_padding_mask") is not None or astate.get("prev_padding_mask") is not None:
        return False
    n = 0 if k is None else k.size(1)
    chunk = blk.chunk_size
    if (k is None) != (v is None) or (chunk > 0 and n >= chunk):
        return False
    if n and (k.dtype != x.dtype or v.dtype != x.dtype or k.size(0) != bsz or k.stride(-1) != 1 or v.stride(-1) != 1):
        return False
    # running statistics and pole states, as the norm -> EMA step keeps them
    nkey = norm._get_full_incremental_state_key("norm_state")
    ekey = move._get_full_incremental_state_key("ema_state")
    nstate, estate = incremental_state.get(nkey), incremental_state.get(ekey)
    if nstate is None or estate is None or 'prev_mean' not in nstate or estate.get('prev_state') is None:
        nstate, estate = _seed_decode_state(norm, move, bsz, dim, dev, incremental_state)
    sdtype = torch.complex64 if move.complex else torch.float32
    for d, key, dt in ((nstate, 'prev_mean', torch.float32), (nstate, 'prev_var', torch.float32),
                       (nstate, 'prev_count', torch.int64), (estate, 'prev_state', sdtype)):
        if d[key].dtype != dt or not d[key].is_contiguous():
            d[key] = d[key].to(dt).contiguous()
    mean, var, count, h = nstate['prev_mean'], nstate['prev_var'], nstate['prev_count'], estate['prev_state']
    count_next = torch.empty_like(count)
    if chunk > 49152:
        return False
    cap = max(256, 2 * n)   # (a chunk is not laid out in full for its first tokens; the next plan has room for twice as many)
    cap = min(cap, chunk) if chunk > 0 else cap
    if cap > 49152:
        return False
    keys = torch.empty(bsz, cap, blk.zdim, dtype=x.dtype, device=dev)
    keys_rot = torch.empty_like(keys)
    values = torch.empty(bsz, cap, blk.hdim, dtype=x.dtype, device=dev)
    rot = torch.view_as_real(blk.rel_pos_bias._angles(0, max(cap, 1)))
    lib = _lib.lib()
    dt = ops._dt(x)
    with torch.cuda.device(dev):
        if n:
            _lib.check(lib.mega_block_cache_fill(
                k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0), v.stride(1), rot.data_ptr(), rot.size(0),
                dt, bsz, n, blk.zdim, blk.hdim, keys.data_ptr(), keys_rot.data_ptr(), values.data_ptr(), cap,
                stream), "block_cache_fill")
        work = torch.empty(lib.mega_block_step_work(dt, bsz, dim, blk.zdim, blk.hdim, cap), dtype=torch.uint8, device=dev)
    gamma_eff, beta = ops.norm_prepare(norm.weight, norm.bias)
    p, q, g, omega = _ema_params(move)
    args = _lib.BlockStepArgs(
        dtype=dt, batch=bsz, embed=dim, zdim=blk.zdim, hdim=blk.hdim, ndim=move.ndim, complex_poles=int(move.complex),
        positions=rot.size(0), norm_gamma=gamma_eff.data_ptr(), norm_beta=beta.data_ptr(),
        p=p.data_ptr(), q=q.data_ptr(), gamma_hat=g.data_ptr(), omega=omega.data_ptr(),
        v_weight=blk.v_proj.weight.data_ptr(), v_bias=blk.v_proj.bias.data_ptr(),
        mx_weight=blk.mx_proj.weight.data_ptr(), mx_bias=blk.mx_proj.bias.data_ptr(),
        h_weight=blk.h_proj.weight.data_ptr(), qk_gamma=blk.gamma.data_ptr(), qk_beta=blk.beta.data_ptr(),
        rot=rot.data_ptr(), keys=keys.data_ptr(), keys_rot=keys_rot.data_ptr(), values=values.data_ptr(),
        work=work.data_ptr(), norm_eps=norm.eps, qk_eps=1e-5, cap=cap, pos=n,
        qk_dtype=ops._dt(blk.gamma))
    names = _names(blk)
    owners = [blk] + [blk._modules[m] for m in _SUBMODULES]
    plans = blk.__dict__.get("_block_plan")   # (None in a copy of a block)
    if plans is None:
        plans = blk._block_plan = _lib.host().BlockPlans()
    plans.add(_lib.host().BlockPlan(
        bytes(args), owners, list(_SUBMODULES), names, [owners[i]._parameters[name] for i, name in names], [nkey, ekey, akey],
        [count, count_next, mean, var, h, k, v], keys, values, [keys_rot, work, rot, gamma_eff, beta, p, q, g, omega],
        chunk, x, stream))
    return True
