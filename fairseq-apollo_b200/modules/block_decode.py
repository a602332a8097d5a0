"""Single-token decoding of the causal Mega block in one library call (mega_block_step): the L == 1 case of
MovingAverageGatedAttention.forward with an incremental state
(fairseq/modules/moving_average_gated_attention.py:282-414).

The keys and values of a chunk live in buffers with room for the whole chunk; the state's ``prev_key`` /
``prev_value`` are views of their first rows, so a step appends a row instead of copying the cache.  Rows that a
view covers are never written again: a step appends only behind the views that the step before handed out, and
any other state (a new generation, reordered beams, a copied state) gets buffers of its own.
"""
import ctypes
from typing import Optional

import torch
from torch import Tensor

from .. import _lib, ops
from ..ops import _current_device, _raw_stream
from .fused import _fp32_params, _param_tensors, _seed_decode_state

_POLES = {False: (4, 8, 16, 32), True: (2, 4, 8, 16, 32)}


class _BlockPlan:
    """What a step passes to the library, converted once, with everything it keeps alive.  Valid for the same
    parameters (identity and version counters), state tensors, batch, dtype, device and stream."""

    def __deepcopy__(self, memo):   # (a copied or pickled block builds its own)
        return None

    def __reduce__(self):
        return (type(None), ())

    __slots__ = ("args", "addr", "fn", "key", "dev", "params", "versions", "nkey", "ekey", "akey", "mean", "var", "h",
                 "count", "count_next", "last_key", "last_value", "keys", "values", "pos", "cap", "chunk", "keep")


def _tensors(blk):
    p, v, m, h = blk._parameters, blk._modules['v_proj']._parameters, blk._modules['mx_proj']._parameters, \
        blk._modules['h_proj']._parameters
    return _param_tensors(blk._modules['norm'], blk._modules['move']) + (
        v['weight'], v['bias'], m['weight'], m['bias'], h['weight'], p['gamma'], p['beta'])


def applicable(blk, x) -> bool:
    """Whether the block and x (B, 1, D) are in the step's envelope (checked once per plan)."""
    norm, move = blk.norm, blk.move
    weights = (blk.v_proj.weight, blk.v_proj.bias, blk.mx_proj.weight, blk.mx_proj.bias, blk.h_proj.weight)
    chunk = blk.chunk_size
    return (blk.efficient_attn is not None and isinstance(blk.move_act, torch.nn.SiLU)
            and type(blk.rel_pos_bias).__name__ == "RotaryEmbedding" and not move.bidirectional
            and norm.num_groups in (None, norm.num_features) and move.ndim in _POLES[move.complex]
            and (chunk < 0 or chunk > 1) and x.dtype in (torch.bfloat16, torch.float16)
            and all(w is not None and w.dtype == x.dtype and w.is_cuda and w.is_contiguous() and w.data_ptr() % 16 == 0
                    for w in weights)
            and x.size(0) <= 64 and blk.zdim in (64, 128, 256) and blk.embed_dim % 32 == 0 and blk.hdim % 32 == 0
            and x.size(0) * (max(blk.embed_dim, blk.hdim) * 2 + 64) <= 200 * 1024)


def step(blk, x: Tensor, incremental_state) -> Optional[Tensor]:
    """One token through the block, or None when the call is not the library's (the caller then runs the
    block's own sequence of operations).  Called with gradients disabled, x (B, 1, D) contiguous, no masks."""
    plan = blk.__dict__.get("_block_plan")
    stream = _raw_stream(x.device.index)
    if plan is None or not _matches(plan, blk, x, stream, incremental_state):
        plan = _build(blk, x, stream, incremental_state)
        if plan is None:
            return None
    a = plan.args
    out = torch.empty_like(x)
    a.x = x.data_ptr()
    a.out = out.data_ptr()
    pos = plan.pos
    a.pos = pos
    if _current_device() == plan.dev:
        rc = plan.fn(plan.addr, stream)
    else:
        with torch.cuda.device(plan.dev):
            rc = plan.fn(plan.addr, stream)
    if rc != 0:
        _lib.check(rc, "block_step")
    # the counts alternate between two arrays, the step wrote the second one
    nstate = incremental_state[plan.nkey]
    nstate['prev_count'] = plan.count_next
    plan.count, plan.count_next = plan.count_next, plan.count
    a.count, a.count_next = a.count_next, a.count
    state = incremental_state.get(plan.akey)
    if state is None:
        state = incremental_state[plan.akey] = {}
    pos += 1
    plan.pos = pos
    if plan.chunk < 0 or pos % plan.chunk != 0:
        state["prev_key"] = plan.last_key = plan.keys.narrow(1, 0, pos)
        state["prev_value"] = plan.last_value = plan.values.narrow(1, 0, pos)
        state["prev_key_padding_mask"] = None
    else:   # the chunk is complete: the next token starts another one, in other buffers
        for key in ("prev_key", "prev_value", "prev_key_padding_mask"):
            state.pop(key, None)
        blk._block_plan = None
    return out


def _matches(plan, blk, x, stream, incremental_state):
    nstate, estate = incremental_state.get(plan.nkey), incremental_state.get(plan.ekey)
    if nstate is None or estate is None or plan.pos >= plan.cap:
        return False
    astate = incremental_state.get(plan.akey) or {}
    ps = _tensors(blk)
    return (nstate.get('prev_mean') is plan.mean and nstate.get('prev_var') is plan.var
            and nstate.get('prev_count') is plan.count and estate.get('prev_state') is plan.h
            and astate.get('prev_key') is plan.last_key and astate.get('prev_value') is plan.last_value
            and astate.get('prev_key_padding_mask') is None
            and plan.key == (x.shape[0], x.dtype, x.device.index, stream)
            and all(map(_same, ps, plan.params)) and [p._version for p in ps] == plan.versions)


def _same(a, b):
    return a is b


def _build(blk, x, stream, incremental_state):
    if not applicable(blk, x):
        return None
    norm, move = blk.norm, blk.move
    bsz, _, dim = x.shape
    dev = x.device
    plan = _BlockPlan()
    plan.akey = blk._get_full_incremental_state_key("attn_state")
    astate = incremental_state.get(plan.akey) or {}
    k, v = astate.get("prev_key"), astate.get("prev_value")
    if astate.get("prev_key_padding_mask") is not None or astate.get("prev_padding_mask") is not None:
        return None
    n = 0 if k is None else k.size(1)
    plan.chunk = blk.chunk_size
    if (k is None) != (v is None) or (plan.chunk > 0 and n >= plan.chunk):
        return None
    if n and (k.dtype != x.dtype or v.dtype != x.dtype or k.size(0) != bsz or k.stride(-1) != 1 or v.stride(-1) != 1):
        return None
    # running statistics and pole states, as the norm -> EMA step keeps them
    plan.nkey = norm._get_full_incremental_state_key("norm_state")
    plan.ekey = move._get_full_incremental_state_key("ema_state")
    nstate, estate = incremental_state.get(plan.nkey), incremental_state.get(plan.ekey)
    if nstate is None or estate is None or 'prev_mean' not in nstate or estate.get('prev_state') is None:
        nstate, estate = _seed_decode_state(norm, move, bsz, dim, dev, incremental_state)
    sdtype = torch.complex64 if move.complex else torch.float32
    for d, key, dt in ((nstate, 'prev_mean', torch.float32), (nstate, 'prev_var', torch.float32),
                       (nstate, 'prev_count', torch.int64), (estate, 'prev_state', sdtype)):
        if d[key].dtype != dt or not d[key].is_contiguous():
            d[key] = d[key].to(dt).contiguous()
    plan.mean, plan.var, plan.count, plan.h = nstate['prev_mean'], nstate['prev_var'], nstate['prev_count'], estate['prev_state']
    plan.count_next = torch.empty_like(plan.count)
    cap = plan.chunk if plan.chunk > 0 else max(256, 2 * n)
    if cap > 49152:
        return None
    plan.cap, plan.pos = cap, n
    plan.keys = torch.empty(bsz, cap, blk.zdim, dtype=x.dtype, device=dev)
    keys_rot = torch.empty_like(plan.keys)
    plan.values = torch.empty(bsz, cap, blk.hdim, dtype=x.dtype, device=dev)
    rot = torch.view_as_real(blk.rel_pos_bias._angles(0, max(cap, 1)))
    lib = _lib.lib()
    dt = ops._dt(x)
    with torch.cuda.device(dev):
        if n:
            _lib.check(lib.mega_block_cache_fill(
                k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0), v.stride(1), rot.data_ptr(), rot.size(0),
                dt, bsz, n, blk.zdim, blk.hdim, plan.keys.data_ptr(), keys_rot.data_ptr(), plan.values.data_ptr(), cap,
                stream), "block_cache_fill")
        work = torch.empty(lib.mega_block_step_work(dt, bsz, dim, blk.zdim, blk.hdim, cap), dtype=torch.uint8, device=dev)
    plan.last_key, plan.last_value = k, v
    cache = blk.__dict__.get("_qk_fp32")
    gver = (blk.gamma._version, blk.beta._version)
    if cache is None or cache[0] is not blk.gamma or cache[1] is not blk.beta or cache[2] != gver:
        cache = blk._qk_fp32 = (blk.gamma, blk.beta, gver, blk.gamma.detach().float().contiguous(),
                                blk.beta.detach().float().contiguous())
    gamma_eff, beta, p, q, g, omega = _fp32_params(norm, move)
    plan.params = _tensors(blk)
    plan.versions = [t._version for t in plan.params]
    plan.key = (bsz, x.dtype, dev.index, stream)
    plan.dev = dev.index
    a = plan.args = _lib.BlockStepArgs(
        dtype=dt, batch=bsz, embed=dim, zdim=blk.zdim, hdim=blk.hdim, ndim=move.ndim, complex_poles=int(move.complex),
        positions=rot.size(0), count=plan.count.data_ptr(), count_next=plan.count_next.data_ptr(),
        mean=plan.mean.data_ptr(), var=plan.var.data_ptr(), h=plan.h.data_ptr(), norm_gamma=gamma_eff.data_ptr(),
        norm_beta=beta.data_ptr(), p=p.data_ptr(), q=q.data_ptr(), gamma_hat=g.data_ptr(), omega=omega.data_ptr(),
        v_weight=blk.v_proj.weight.data_ptr(), v_bias=blk.v_proj.bias.data_ptr(),
        mx_weight=blk.mx_proj.weight.data_ptr(), mx_bias=blk.mx_proj.bias.data_ptr(),
        h_weight=blk.h_proj.weight.data_ptr(), qk_gamma=cache[3].data_ptr(), qk_beta=cache[4].data_ptr(),
        rot=rot.data_ptr(), keys=plan.keys.data_ptr(), keys_rot=keys_rot.data_ptr(), values=plan.values.data_ptr(),
        work=work.data_ptr(), norm_eps=norm.eps, qk_eps=1e-5, cap=cap, pos=n)
    plan.addr = ctypes.addressof(a)
    plan.fn = lib.mega_block_step
    plan.keep = (keys_rot, work, rot, cache, gamma_eff, beta, p, q, g, omega)
    blk._block_plan = plan
    return plan
