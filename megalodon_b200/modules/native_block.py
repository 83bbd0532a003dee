"""A MEGA block as one native call each way (csrc/mega_block.h).

A launch through the modules costs the host 20 to 27 us, which bounds everything but the largest models; the native
block launches the same kernels at some 9 us each.  It stands for the calls of the block's own modules, so it is taken
only where those are what the model was built with, without hooks, and where every operator would run on the kernels,
which is asked anew at every call.
"""
from __future__ import annotations

from typing import Optional

import torch
from torch import Tensor

from ..ops import cuda_ops, native_for
from ..ops._ext import require
from ..parallel.initialize import get_chunk_parallel_world_size, get_model_parallel_world_size
from ..parallel.model_parallel import ColumnParallelLinear, RowParallelLinear
from ..utils import is_plain
from .complex_exponential_moving_average import MultiHeadComplexEMA
from .layer_norm import FusedLayerNorm, FusedRMSNorm
from .moving_average_gated_attention import CAUSAL, MovingAverageGatedAttention, _InnerAttention
from .normalized_feedforward_network import NormalizedFeedForwardNetwork
from .timestep_norm import TimestepNorm

# Sub-modules that the block stands for; fc3 only with SwiGLU.
_MEGA = {"timenorm": TimestepNorm, "cema": MultiHeadComplexEMA, "rmsnorm": FusedRMSNorm, "znorm": FusedRMSNorm,
         "wv": ColumnParallelLinear, "wz": ColumnParallelLinear, "wr": ColumnParallelLinear, "wh1": ColumnParallelLinear,
         "wh2": RowParallelLinear, "inner_attention": _InnerAttention}
_NFFN = {"norm": FusedLayerNorm, "fc1": ColumnParallelLinear, "fc2": RowParallelLinear, "fc3": ColumnParallelLinear}


# Places among `_params` of the weights whose gradient is a product, which may land in the flat gradient of a unit (the
# views of other matrices carry a sink too, but their gradients go through autograd).
_PRODUCTS = frozenset((4, 6, 8, 10, 14, 17, 18, 19))


def _params(a, f, am, fm):
    """Parameters in the order of `BlockParam`.  (`am`, `fm`: the sub-modules by name; as attributes of a module they
    cost ten times the look-up.)"""
    t, wv, wz, wr, wh1, norm, fc3 = am["timenorm"], am["wv"], am["wz"], am["wr"], am["wh1"], fm["norm"], fm.get("fc3")
    return [t.weight, t.bias, am["cema"].omega, am["rmsnorm"].weight, wv.weight, wv.bias, wz.weight, wz.bias, wr.weight,
            wr.bias, wh1.weight, wh1.bias, a.gamma, a.beta, am["wh2"].weight, norm.weight, norm.bias, fm["fc1"].weight,
            None if fc3 is None else fc3.weight, fm["fc2"].weight]


def _as_built(a, f, am, fm) -> bool:
    fc3 = fm.get("fc3")
    if not (is_plain(a, MovingAverageGatedAttention) and is_plain(f, NormalizedFeedForwardNetwork)
            and all(is_plain(am.get(n), cls) for n, cls in _MEGA.items())
            and all(is_plain(fm.get(n), cls) for n, cls in _NFFN.items() if n != "fc3" or fc3 is not None)):
        return False
    acts = [am[n].activation for n in ("wv", "wr", "wz", "wh1")] + [fm["fc1"].activation]
    return (am["znorm"].weight is None and acts == ["silu", "silu", None, None, None if f.swiglu else "silu"]
            and (fc3 is not None) == bool(f.swiglu) and (fc3 is None or fc3.activation is None)
            and all(m is None or m.bias is None for m in (am["wh2"], fm["fc1"], fm["fc2"], fc3)) and f.alpha is None
            and a.head_split == 1 and a.local_heads == a.num_heads
            and "forward_channels_last" not in am["cema"].__dict__)


def _takes(a, f, inner, x: Tensor, mask, cache) -> bool:
    """Whether sizes, types and options are the native block's."""
    if (type(x) is not Tensor or not x.is_cuda or x.dim() != 3 or x.numel() == 0
            or x.dtype not in (torch.bfloat16, torch.float16) or not native_for(x)
            or cuda_ops.gemm_backend() != "tcgen05" or cuda_ops._transformed()
            or not cuda_ops._FUSED_SOFTMAX[0] or cuda_ops._RECOMPUTE_SCORES[0]
            or get_model_parallel_world_size() != 1 or get_chunk_parallel_world_size() != 1):
        return False
    if mask is not None and mask is not CAUSAL or mask is None and not a.efficient_attn:
        return False
    if (a.training or inner.training or f.training) and max(a.dropout, a.hidden_dropout,
                                                                        inner.dropout, f.dropout,
                                                                        f.hidden_dropout) > 0.0:
        return False
    L, c = x.shape[1], a.chunk_size
    # one token, or a chunk that begins with cached keys, are the modules'
    if x.shape[0] * L < 2 or L < 2 or (L > c and L % c != 0) or inner.chunk_size != c:
        return False
    if cache is not None:
        kv = cache[0]
        if (torch.is_grad_enabled() or kv is None or isinstance(kv[2], Tensor) or kv[2] != 0
                or (kv[0] is not None and kv[0].size(1) != 0)):
            return False
    D, S, V, F = a.mdim, a.num_heads * a.z_head_dim, a.num_heads * a.v_head_dim, f.hidden_dim
    if (x.shape[2] != D or max(D, S) > 8192 or any(n % 8 for n in (D, a.z_head_dim, a.v_head_dim, F))
            or a.ndim not in (1, 2, 4, 8, 16, 32)
            or not cuda_ops.attention_shapes_ok(x.dtype, a.z_head_dim, a.v_head_dim, min(L, c))):
        return False
    return x.requires_grad or not torch.is_grad_enabled()


def _params_taken(params, x: Tensor) -> bool:
    grad = torch.is_grad_enabled()
    for p in params:
        if p is None:
            continue
        if (p.dtype != x.dtype or p.device != x.device or not p.is_contiguous() or p.data_ptr() & 15
                or (grad and not p.requires_grad)):
            return False
        spec = getattr(p, "_gather_spec", None)
        if spec is not None and spec.pending:
            return False
    return True


class _MegaBlock(torch.autograd.Function):
    """Inputs after `meta`: x, count, mean, var, hx, p, q, gamma, then the parameters."""

    @staticmethod
    def forward(ctx, meta, x, count, mean, var, hx, p, q, gamma, *params):
        dims, eps, freqs, want_last, keep, prior = meta
        D = x.shape[-1]
        p2, q2, g2 = p.reshape(D, -1).float().contiguous(), cuda_ops._c2r(q.reshape(D, -1)), cuda_ops._c2r(gamma.reshape(D, -1))
        h2 = None if hx is None else cuda_ops._c2r(hx)
        outs, saved, launches = require().mega_block_fwd(x, count, mean, var, h2, p2, q2, g2, freqs, list(params), dims, eps,
                                                         want_last, keep, prior, cuda_ops._err_flag(x.device))
        cuda_ops._bump(launches)
        out, count, mean_out, var_out, k, v = outs[:6]
        h = torch.view_as_complex(outs[6]) if want_last else None
        if not keep:
            return out, count, mean_out, var_out, h, k, v
        ctx.some = [t is not None for t in (*saved, h2, *params)]
        ctx.save_for_backward(*[t for t in (*saved, h2, *params) if t is not None], p2, q2, g2, freqs)
        ctx.sinks = [getattr(t, "_wgrad_sink", None) if i in _PRODUCTS else None for i, t in enumerate(params)]
        ctx.meta = dims, eps, mean.dtype, var.dtype, p.shape, p.dtype, q.shape, gamma.shape
        ctx.mark_non_differentiable(count)
        ctx.set_materialize_grads(False)
        return out, count, mean_out, var_out, h

    @staticmethod
    def backward(ctx, dout, _dcount, dmean, dvar, dh):
        dims, eps, mean_type, var_type, p_shape, p_type, q_shape, g_shape = ctx.meta
        *rest, p2, q2, g2, freqs = ctx.saved_tensors
        rest = iter(rest)
        every = [next(rest) if some else None for some in ctx.some]
        n = len(ctx.sinks)
        saved, h2, params = every[:-n - 1], every[-n - 1], every[-n:]
        if dout is None:                    # only the running state was used
            dout = torch.zeros_like(saved[0])
        places = [(None, False) if sink is None else sink() for sink in ctx.sinks]
        grads, launches = require().mega_block_bwd(
            dout, dmean, dvar, None if dh is None else cuda_ops._c2r(dh), saved, h2, p2, q2, g2, freqs, params,
            [t for t, _ in places], [add for _, add in places], dims, eps, cuda_ops._err_flag(dout.device))
        cuda_ops._bump(launches)
        dx, dm, dv, dhx, dp, dq, dg, *dparams = grads
        return (None, dx, None, dm.to(mean_type), dv.to(var_type), None if h2 is None else torch.view_as_complex(dhx),
                dp.view(p_shape).to(p_type), torch.view_as_complex(dq).view(q_shape), torch.view_as_complex(dg).view(g_shape),
                *dparams)


def forward(block, x: Tensor, freqs_cis: Tensor, mask=None, cache=None, carry=None, piece=None):
    """`block.forward` as one call, or None where the modules have to be called."""
    a, f = block.mega, block.nffn
    if not x.is_cuda or type(a) is not MovingAverageGatedAttention or type(f) is not NormalizedFeedForwardNetwork:
        return None
    am, fm = a._modules, f._modules
    if not _as_built(a, f, am, fm) or not _takes(a, f, am["inner_attention"], x, mask, cache):
        return None
    params = _params(a, f, am, fm)
    if not _params_taken(params, x):
        return None
    bsz, L, _ = x.shape
    norm = am["timenorm"]
    streaming = piece is not None
    last_piece = not streaming or piece[0] == piece[1] - 1
    emit = streaming and len(piece) > 3 and bool(piece[3])
    count = mean = var = hx = None
    if cache is not None:
        _, (count, mean, var), hx = cache
    elif carry is not None:
        count, mean, var, hx = carry
    grad = torch.is_grad_enabled()
    # without gradients the kernel spreads the prior over the batch itself
    prior = (not grad and count is None and mean is None and var is None and "initial_stats" not in norm.__dict__
             and norm.prior_mean.dtype == norm.prior_logv.dtype == x.dtype)
    if prior:
        count, mean, var = norm.prior_count, norm.prior_mean, norm.prior_logv
    elif count is None or mean is None or var is None:
        c0, m0, v0 = norm.initial_stats(bsz, x.dtype)
        count, mean, var = (c0 if count is None else count, m0 if mean is None else mean, v0 if var is None else var)
    want_last = cache is not None or (streaming and not last_piece) or emit
    freqs = torch.view_as_real(freqs_cis.to(torch.complex64).contiguous())
    meta = ([norm.groups_per_partition, a.num_heads, a.z_head_dim, a.v_head_dim, a.chunk_size],
            [norm.eps, am["rmsnorm"].eps, am["znorm"].eps, fm["norm"].eps], freqs, want_last, grad, prior)
    args = (meta, x, count, mean, var, hx, *am["cema"].coeffs(), *params)
    if grad:
        out, count, mean, var, h = _MegaBlock.apply(*args)
    else:
        out, count, mean, var, h, k, v = _MegaBlock.forward(None, *args)
    if cache is not None:
        tail = L % a.chunk_size
        keys = tuple(t.view(bsz, L, a.num_heads, -1)[:, L - tail:] for t in (k, v))
        return out, ((*keys, tail), (count, mean, var), h)
    if streaming and not last_piece:
        return out, (count, mean, var, h)
    if emit:
        return out, (count.detach(), mean.detach(), var.detach(), h.detach())
    return out, None
