"""Token-by-token decoding against a fixed-shape state, replayed from a CUDA graph.

The regular cache path (`Mega.forward(tokens, cache)`, reference:
megalodon/model/mega.py:190-233 and generation.py:105-125) grows the key/value
tail by concatenation and tracks lengths in Python, so every token costs a few
hundred eager kernel launches: the 7B model spends about 40 ms of host time per
token.  A `DecodeSession` keeps the whole recurrent state in buffers whose
shapes never change -

    per layer   k, v [B, H, chunk, d]   chunk-local keys / values (entries past `pos` are masked)
                count [B], mean, var [B, G]   TimestepNorm running statistics
                hx [B, D, N] complex          CEMA state
    output norm count, mean, var
    pos [1]     position of the next token inside its chunk (device tensor)

- runs one step through the model's own layers, and after two eager steps
captures the step in a CUDA graph; from then on a token is one graph launch.
On CPU, with tensor-parallel ranks, or with `use_graph=False` the same code
runs eagerly, which is what the tests compare against the regular cache path.

On one GPU with 16-bit weights the step is a chain of native launches
(`_native_step`): per layer four products and four kernels for everything
between them, each a link of a programmatic dependent launch chain, instead of
some thirty-five launches through the modules.
"""
from __future__ import annotations

from typing import List, Optional, Tuple

import torch
from torch import Tensor

from .utils import is_plain


def _unwrap(model):
    while hasattr(model, "_wrapped"):
        model = model._wrapped
    return model


class DecodeSession:
    def __init__(self, model, batch_size: int, dtype: torch.dtype = torch.bfloat16, use_graph: Optional[bool] = None):
        self.model = model
        self.mega = _unwrap(model)
        m = self.mega
        if hasattr(model, "materialize_views"):
            model.materialize_views()         # the step calls sub-modules directly, not the FSDP wrapper
        self.B = batch_size
        self.dtype = dtype
        self.device = next(model.parameters()).device
        # Graph capture is the default on a GPU.  With tensor-parallel ranks the collectives of the step
        # (all-reduce after the row-parallel projections, gathers of feature-sharded activations and of
        # the logits) go through `SmallCollective`: one peer-memory kernel each, whose epoch lives in
        # device memory, so the captured step replays correctly (NCCL inside the capture did not complete).
        self._small = None
        from .parallel.initialize import (get_model_parallel_group, get_model_parallel_world_size,
                                          model_parallel_is_initialized)
        mp = get_model_parallel_world_size() if model_parallel_is_initialized() else 1
        if mp > 1 and self.device.type == "cuda" and use_graph is not False:
            from .parallel.model_parallel import mappings
            from .parallel.symm import SmallCollective
            self._small = SmallCollective(get_model_parallel_group(), self.device, max_bytes=2 << 20)
            mappings.use_small_collective(self._small)
        self.use_graph = (self.device.type == "cuda") if use_graph is None else use_graph
        c = m.chunk_size
        first = _unwrap(m.layers[0]).mega
        H, dk, dv = first.local_heads, first.z_head_dim, first.local_v_head_dim
        G = first.timenorm.groups_per_partition
        D, N = first.local_mdim, first.cema.ndim
        dev = self.device
        self._native = self._native_ok()
        # the native step keeps the running statistics in fp32, the modules hand them on in the compute dtype
        stat_dtype = torch.float32 if self._native else dtype

        def norm_state(groups):
            return [torch.zeros(batch_size, dtype=torch.int64, device=dev),
                    torch.zeros(batch_size, groups, dtype=stat_dtype, device=dev),
                    torch.ones(batch_size, groups, dtype=stat_dtype, device=dev)]

        self.layers: List[dict] = []
        for _ in range(m.num_layers):
            self.layers.append({
                "k": torch.zeros(batch_size, H, c, dk, dtype=dtype, device=dev),
                "v": torch.zeros(batch_size, H, c, dv, dtype=dtype, device=dev),
                "norm": norm_state(G),
                "hx": torch.zeros(batch_size, D, N, dtype=torch.complex64, device=dev),
            })
        self.out_norm = norm_state(m.output.final_norm.groups_per_partition)
        self.pos = torch.zeros(1, dtype=torch.int64, device=dev)
        self.tok = torch.zeros(batch_size, 1, dtype=torch.int64, device=dev)
        self.logits: Optional[Tensor] = None
        self._graph = None
        self._eager_steps = 0
        self._fresh = True           # no statistics yet: the norms start from their priors
        if self._native:
            self._native_buffers()

    # ------------------------------------------------------------------ state import
    @torch.no_grad()
    def load_cache(self, cache) -> None:
        """Take over the state of a regular cache (e.g. after prefilling the prompt)."""
        layers, out_norm = cache
        n = 0
        dsts, srcs = list(self.out_norm), list(out_norm)
        for st, (kv, norm, hx) in zip(self.layers, layers):
            if not self._native:     # (the native step reads no slot past `pos`)
                st["k"].zero_()
                st["v"].zero_()
            n = 0
            if kv is not None and kv[0] is not None:
                n = int(kv[2])
                if n > 0:
                    st["k"][:, :, :n].copy_(kv[0][:, -n:].transpose(1, 2))
                    st["v"][:, :, :n].copy_(kv[1][:, -n:].transpose(1, 2))
            dsts += [*st["norm"], torch.view_as_real(st["hx"])]
            srcs += [*norm, torch.view_as_real(hx)]
        torch._foreach_copy_(dsts, srcs)
        self.pos.fill_(n)
        self._fresh = False

    # ------------------------------------------------------------------ one token, native chain
    def _native_ok(self) -> bool:
        """Whether every layer is inside what the native step covers: one GPU's worth of 16-bit parameters
        in the session's dtype, plain MEGA blocks, sizes the kernels take."""
        from .ops import native_for
        from .ops._ext import require
        m = self.mega
        if self.device.type != "cuda" or self.dtype not in (torch.bfloat16, torch.float16) or self._small is not None:
            return False
        w = m.embed.weight
        if w is None or w.dtype != self.dtype or not native_for(w) or self.B > 64:
            return False
        from .ops import cuda_ops
        if cuda_ops.gemm_backend() != "tcgen05" or m.embed.weight.shape[1] != m.model_dim:
            return False
        # a sharded unit gives its gathered weights back after every call of its own
        if any(u.reshard_after_forward and not u._is_root for u in self._units()) or not self._weights_current():
            return False
        if not self._as_built():
            return False
        C = require()
        for layer in m.layers:
            block = _unwrap(layer)
            a = block.mega
            dims = (a.mdim, a.z_head_dim, a.local_v_head_dim, block.nffn.hidden_dim)
            if (block.nffn.alpha is not None or a.head_split != 1 or a.local_heads != a.num_heads
                    or a.local_mdim != a.mdim or a.mdim > 16384 or any(d % 8 for d in dims) or m.chunk_size > 51200
                    or not C.decode_norm_ema_ok(a.mdim, a.timenorm.groups_per_partition, a.cema.ndim)):
                return False
            if not self._params_ok(self._layer_params(block)):
                return False
        fn, out = m.output.final_norm, m.output.output
        return (C.decode_norm_ema_ok(m.model_dim, fn.groups_per_partition, 2) and out.weight.shape[1] == m.model_dim
                and self._params_ok([fn.weight, fn.bias, out.weight]))

    def _units(self):
        return [u for u in self.model.modules() if hasattr(u, "_full_is_valid")]

    def _weights_current(self) -> bool:
        """Whether the gathered weights are what the units' own calls would use, after bringing them up to date where
        the session's model can (it may have been given the model inside its root unit)."""
        if all(u._full_is_valid() for u in self._units()):
            return True
        if not hasattr(self.model, "materialize_views"):
            return False
        self.model.materialize_views()
        return True

    def _params_ok(self, params) -> bool:
        return all(p.dtype == self.dtype and p.is_contiguous() and p.data_ptr() % 16 == 0 for p in params)

    def _as_built(self) -> bool:
        """Whether every module whose call the native step stands for is the one that the model was built with,
        without hooks, so that taking its parameters comes to the same thing."""
        from .models.mega import MegaBlock, MegaOutputLayer
        from .modules import MovingAverageGatedAttention, NormalizedFeedForwardNetwork, TimestepNorm
        from .modules.complex_exponential_moving_average import MultiHeadComplexEMA
        from .modules.layer_norm import FusedLayerNorm, FusedRMSNorm
        from .modules.moving_average_gated_attention import _InnerAttention
        from .parallel.model_parallel import ColumnParallelLinear, ParallelEmbedding, RowParallelLinear
        m = self.mega
        mods = [(m.embed, ParallelEmbedding), (m.output, MegaOutputLayer), (m.output.final_norm, TimestepNorm),
                (m.output.output, RowParallelLinear)]
        for layer in m.layers:
            while hasattr(layer, "_wrapped"):
                mods.append((layer, type(layer)))
                layer = layer._wrapped
            if type(layer) is not MegaBlock:
                return False
            a, f = layer.mega, layer.nffn
            mods += [(layer, MegaBlock), (a, MovingAverageGatedAttention), (f, NormalizedFeedForwardNetwork),
                     (a.timenorm, TimestepNorm), (a.cema, MultiHeadComplexEMA), (a.rmsnorm, FusedRMSNorm),
                     (a.znorm, FusedRMSNorm), (a.wv, ColumnParallelLinear), (a.wz, ColumnParallelLinear),
                     (a.wr, ColumnParallelLinear), (a.wh1, ColumnParallelLinear), (a.wh2, RowParallelLinear),
                     (a.inner_attention, _InnerAttention), (f.norm, FusedLayerNorm), (f.fc1, ColumnParallelLinear),
                     (f.fc2, RowParallelLinear)]
            if f.fc3 is not None:
                mods.append((f.fc3, ColumnParallelLinear))
        if not all(is_plain(mod, cls) for mod, cls in mods) or m.embed.max_norm is not None:
            return False
        for layer in m.layers:
            a, f = _unwrap(layer).mega, _unwrap(layer).nffn
            acts = [a.wv.activation, a.wr.activation, a.wz.activation, a.wh1.activation, f.fc1.activation]
            if (a.znorm.weight is not None or acts != ["silu", "silu", None, None, None if f.swiglu else "silu"]
                    or (f.fc3 is not None) != bool(f.swiglu) or (f.swiglu and f.fc3.activation is not None)
                    or any(p is not None and p.bias is not None for p in (a.wh2, f.fc1, f.fc2, f.fc3))):
                return False
        return m.output.output.bias is None

    @staticmethod
    def _layer_params(block):
        a, f = block.mega, block.nffn
        ps = [a.gamma, a.beta, a.timenorm.weight, a.timenorm.bias, a.rmsnorm.weight, a.cema.omega, a.wv.weight, a.wv.bias,
              a.wz.weight, a.wz.bias, a.wr.weight, a.wr.bias, a.wh1.weight, a.wh1.bias, a.wh2.weight,
              f.norm.weight, f.norm.bias, f.fc1.weight, f.fc2.weight]
        if f.fc3 is not None:
            ps.append(f.fc3.weight)
        return [p for p in ps if p is not None]

    def _native_buffers(self) -> None:
        """Activations of a step.  They are shared by all layers: a link writes only after its predecessor is
        complete, and by then everything that read the buffer is."""
        m, B, dev = self.mega, self.B, self.device
        a = _unwrap(m.layers[0]).mega
        D, S, V, F = m.model_dim, a.num_heads * a.z_head_dim, a.num_heads * a.local_v_head_dim, \
            _unwrap(m.layers[0]).nffn.hidden_dim
        from .ops._ext import require
        splits = require().decode_attend_splits(B * a.num_heads, m.chunk_size)
        self._buf = {n: torch.empty(B, k, dtype=self.dtype, device=dev) for n, k in
                     dict(t=D, mx=D, z=S, r=V, v=V, h=D, attn=V, y=D, f=D, u=F, x0=D, x1=D).items()}
        # bf16: the EMA output leaves the norm + EMA link before its RMSNorm's factor, which the products apply.  In fp16 it
        # may be an infinity or lose bits below 6e-5 without the factor, so there the link applies it.
        self._buf["sq"] = (torch.empty(B, a.timenorm.groups_per_partition, dtype=torch.float32, device=dev)
                           if self.dtype == torch.bfloat16 else None)
        self._buf["logits"] = torch.empty(B, m.output_size, dtype=torch.float32, device=dev)
        self._buf["part"] = torch.empty(B * a.num_heads * splits * (a.local_v_head_dim + 2), device=dev)

    def _start_stats(self) -> None:
        """A sequence without a past starts from the priors of its norms."""
        for layer, st in zip(self.mega.layers, self.layers):
            for dst, src in zip(st["norm"], _unwrap(layer).mega.timenorm.initial_stats(self.B, torch.float32)):
                dst.copy_(src)
        for dst, src in zip(self.out_norm, self.mega.output.final_norm.initial_stats(self.B, torch.float32)):
            dst.copy_(src)

    @staticmethod
    def _coefficients(a):
        """p, q, gamma, omega of the layer's EMA as the kernels take them."""
        p, q, gamma = a.cema.coeffs()
        return [p.reshape(a.mdim, -1).float().contiguous(), torch.view_as_real(q.reshape(a.mdim, -1).contiguous()),
                torch.view_as_real(gamma.reshape(a.mdim, -1).contiguous()), a.cema.omega.view(a.mdim)]

    def _native_step(self) -> Tensor:
        from .ops import cuda_ops
        from .ops._ext import require
        C, m, b = require(), self.mega, self._buf
        err = cuda_ops._err_flag(self.device)
        if self._fresh:
            self._start_stats()
        table = torch.view_as_real(m.rope.get_freqs_cis(0, m.chunk_size))
        # The links of the chain read these ahead of their wait, so whatever computes them (a model just put in eval
        # mode has none yet) is launched before the first link, which waits for all of it.
        coeffs = [self._coefficients(_unwrap(layer).mega) for layer in m.layers]
        self._keep = [table, coeffs]     # what a captured graph reads besides the session's buffers and the weights

        def products(xs, ws, biases, addends, acts, outs, w2=None, row_sqs=(), row_eps=0.0):
            rc = C.skinny_gemm(xs, ws, [w2] if w2 is not None else [None] * len(xs), biases, addends, acts, outs, True,
                               err, list(row_sqs), row_eps)
            if rc != 0:
                raise RuntimeError(f"decode products: launch failed with code {rc}")

        x = torch.nn.functional.embedding(self.tok[:, 0], m.embed.weight)
        if m.emb_scale is not None:
            x = x * m.emb_scale
        n = 0
        for layer, st in zip(m.layers, self.layers):
            block = _unwrap(layer)
            a, f = block.mega, block.nffn
            count, mean, var = st["norm"]
            C.decode_norm_ema(x, a.timenorm.weight, a.timenorm.bias, count, mean, var, b["t"], *coeffs[n],
                              torch.view_as_real(st["hx"]), a.rmsnorm.weight, b["mx"], None, 0, a.timenorm.eps,
                              a.rmsnorm.eps, b["sq"], n > 0)
            products([b["mx"], b["mx"], b["t"], b["mx"]], [a.wh1.weight, a.wr.weight, a.wv.weight, a.wz.weight],
                     [a.wh1.bias, a.wr.bias, a.wv.bias, a.wz.bias], [x, None, None, None], [0, 1, 1, 0],
                     [b["h"], b["r"], b["v"], b["z"]], None, [b["sq"], b["sq"], None, b["sq"]], a.rmsnorm.eps)
            C.decode_attend(b["z"], a.gamma, a.beta, table, b["v"], st["k"], st["v"], self.pos, b["r"], b["attn"],
                            b["part"], a.znorm.eps, True)
            products([b["attn"]], [a.wh2.weight], [None], [b["h"]], [0], [b["y"]])
            C.decode_layer_norm(b["y"], f.norm.weight, f.norm.bias, b["f"], f.norm.eps, True)
            products([b["f"]], [f.fc1.weight], [None], [None], [2 if f.swiglu else 1], [b["u"]],
                     f.fc3.weight if f.swiglu else None)
            nxt = b["x0"] if n % 2 == 0 else b["x1"]
            products([b["u"]], [f.fc2.weight], [None], [x], [0], [nxt])
            x = nxt
            n += 1
        norm, (count, mean, var) = m.output.final_norm, self.out_norm
        C.decode_norm_ema(x, norm.weight, norm.bias, count, mean, var, b["t"], None, None, None, None, None, None, None,
                          self.pos, m.chunk_size, norm.eps, 0.0, True)
        products([b["t"]], [m.output.output.weight], [None], [None], [0], [b["logits"]])
        cuda_ops._bump(8 * n + 2)        # (attention as two launches, its most; the EMA coefficients count themselves)
        return b["logits"]

    # ------------------------------------------------------------------ one token
    def _step_body(self) -> Tensor:
        # (a hook or an adapter may have come since, an optimiser step or a load)
        if self._native and self._as_built() and self._weights_current():
            return self._native_step()
        m = self.mega
        x = m.embed(self.tok)
        if m.emb_scale is not None:
            x = x * m.emb_scale
        freqs = m.rope.get_freqs_cis(0, m.chunk_size).index_select(0, self.pos)
        for layer, st in zip(m.layers, self.layers):
            norm = self._stats(st["norm"]) if not self._fresh else (None, None, None)
            hx = st["hx"] if not self._fresh else None
            x, (_, new_norm, new_hx) = layer(x, freqs, None, ((st["k"], st["v"], self.pos), norm, hx))
            for dst, src in zip(st["norm"], new_norm):
                dst.copy_(src)
            st["hx"].copy_(new_hx)
        out_norm = self._stats(self.out_norm) if not self._fresh else (None, None, None)
        logits, new_out = m.output(x, out_norm)
        for dst, src in zip(self.out_norm, new_out):
            dst.copy_(src)
        self.pos.add_(1).remainder_(m.chunk_size)
        return logits[:, -1].float()

    def _eager_step(self) -> Tensor:
        logits = self._step_body()
        # (the chain's logits buffer belongs to the next step)
        return logits.clone() if self._native else logits

    def _stats(self, norm):
        """Running statistics as the modules take them."""
        count, mean, var = norm
        return count, mean.to(self.dtype), var.to(self.dtype)

    @torch.no_grad()
    def step(self, tokens: Tensor) -> Tensor:
        """tokens [B] or [B, 1] -> logits [B, V] (fp32) of the next position."""
        self.tok.copy_(tokens.reshape(self.B, 1))
        if self._graph is not None:
            self._graph.replay()
            return self.logits
        was_training = self.model.training
        if was_training:            # eval() drops the cached CEMA coefficients, so only when needed
            self.model.eval()
        try:
            if self._fresh or not self.use_graph or self._eager_steps < 2:
                self.logits = self._eager_step()
                self._fresh = False
                self._eager_steps += 1
                return self.logits
            # capture: the step reads and writes only the session's buffers
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            # with a process group alive its watchdog thread makes CUDA calls of its own; in the default
            # (global) capture mode those would invalidate the capture, so other threads are exempted
            dist_on = torch.distributed.is_available() and torch.distributed.is_initialized()
            mode = {"capture_error_mode": "thread_local"} if dist_on else {}
            try:
                if self._small is not None:
                    from .parallel.model_parallel import mappings
                    mappings.small_collective_strict(True)
                try:
                    with torch.cuda.graph(graph, **mode):
                        captured = self._step_body()
                finally:
                    if self._small is not None:
                        mappings.small_collective_strict(False)
            except Exception as e:  # noqa: BLE001 - an op that cannot be captured: stay on the eager step
                import logging
                logging.getLogger().warning(f"decode step could not be captured in a CUDA graph ({e}); "
                                            "continuing with eager fixed-shape steps")
                torch.cuda.synchronize()
                self.use_graph = False
                self.logits = self._eager_step()
                return self.logits
            self.logits = captured
            self._graph = graph
            # capturing does not execute: run this token now (the state was not advanced yet)
            graph.replay()
            return self.logits
        finally:
            if was_training:
                self.model.train()

    @torch.no_grad()
    def greedy(self, first_token: Tensor, n_tokens: int) -> Tensor:
        """Generate `n_tokens` greedily starting from `first_token` [B]; returns [B, n_tokens]."""
        out = []
        tok = first_token.reshape(self.B)
        for _ in range(n_tokens):
            tok = self.step(tok).argmax(-1)
            out.append(tok.clone())
        return torch.stack(out, dim=1)
