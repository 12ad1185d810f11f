"""Llama-architecture decoder that keeps its KV cache compressed.

Counterpart of the reference's ``ResKVForCausalLM`` (reskv/models/llama.py:25-170):
prefill attends to dense K/V (SDPA) and then compresses them, decode steps call
the fused compressed attention with the dense recent window.  The reference
subclasses the Hugging Face model; this one is a self-contained module over
plain weight tensors so that it does not depend on a transformers version, can
run with random weights of any Llama shape (the benchmarks need no checkpoint)
and can be tensor-parallel: query/KV heads and the FFN are split over the ranks
(every rank keeps the caches of its own KV heads, so compression and attention
stay local) and the only collectives are the sum all-reduces after ``o_proj``
and ``down_proj``.

``cache="dense"`` keeps an ordinary FP16 KV cache instead (SDPA decode): the
baseline the compressed path is measured against.

Dense matrix products use torch (cuBLAS); everything that touches the
compressed cache goes through ``reskv_b200.compress`` / ``attention``.
"""

from __future__ import annotations

import contextlib
import ctypes
import gc
import os
import threading
from dataclasses import dataclass

import torch
import torch.nn.functional as F

from .._attention import attention
from ..cache import ResKVLayerCache
from ..config import ResKVKernelConfig

try:  # dense baseline only: library flash-decoding kernel, if the image has it
    from flash_attn import flash_attn_with_kvcache as _flash_kvcache
except Exception:  # pragma: no cover
    _flash_kvcache = None


@dataclass(frozen=True)
class LlamaShape:
    """Architecture sizes; defaults are Llama-3.1-8B."""

    hidden: int = 4096
    layers: int = 32
    heads: int = 32
    kv_heads: int = 8
    head_dim: int = 128
    ffn: int = 14336
    vocab: int = 128256
    rope_theta: float = 500000.0
    rms_eps: float = 1e-5


def _rms_norm(x, weight, eps):
    v = x.float()
    v = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps)
    return (v * weight.float()).to(x.dtype)


def _rope(x, cos, sin):
    """Half-split RoPE; x [B, H, T, 128], cos/sin [T, 64] (FP32)."""
    a, b = x.float()[..., :64], x.float()[..., 64:]
    return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1).to(x.dtype)


def _dense_half(tensor, shape, device) -> bool:
    """Whether a kernel may read ``tensor`` by its address alone: FP16 of this shape on ``device``, row-major without gaps, on
    a 16-byte boundary.  Everything else that a caller may assign to the model (transposed views, slices of a fused matrix,
    expanded or misaligned tensors, other types, subclasses with a product of their own) is left to tensor operations."""
    return (type(tensor) in (torch.Tensor, torch.nn.Parameter) and tensor.layout == torch.strided
            and tensor.dtype == torch.float16 and tensor.device == device and tensor.shape == shape
            and tensor.is_contiguous() and not tensor.is_neg() and tensor.data_ptr() % 16 == 0)


class _CollectorHold:
    """Keeps Python's cyclic collector from running while any thread is inside: a finaliser that it ran in a stream capture
    (of another graph, an event, a device buffer) could call CUDA there and spoil the capture.  A collection before the
    capture would not rule that out and takes longer than the capture."""

    def __init__(self):
        self._lock, self._inside, self._was_on = threading.Lock(), 0, False

    @contextlib.contextmanager
    def __call__(self):
        with self._lock:
            if self._inside == 0:
                self._was_on = gc.isenabled()
                gc.disable()
            self._inside += 1
        try:
            yield
        finally:
            with self._lock:
                self._inside -= 1
                if self._inside == 0 and self._was_on:
                    gc.enable()


_collector_held = _CollectorHold()
_streams = threading.local()


def _capture_stream(device) -> torch.cuda.Stream:
    """The calling thread's stream for captures on ``device``: one for all models, so that a new model finds the
    library workspaces and cached blocks of that stream instead of allocating them again."""
    by_device = _streams.__dict__.setdefault("by_device", {})
    index = torch.device(device).index
    index = torch.cuda.current_device() if index is None else index
    if index not in by_device:
        by_device[index] = torch.cuda.Stream(device=index)
    return by_device[index]


class _DenseLayerCache:
    """Plain FP16 KV cache of one layer (rotated keys), preallocated."""

    def __init__(self, batch, kv_heads, capacity, device):
        self.k = torch.empty((batch, kv_heads, capacity, 128), dtype=torch.float16, device=device)
        self.v = torch.empty_like(self.k)
        self.length = 0

    def append(self, k_rot, v):
        n = k_rot.shape[2]
        self.k[:, :, self.length:self.length + n].copy_(k_rot)
        self.v[:, :, self.length:self.length + n].copy_(v)
        self.length += n
        return self.k[:, :, :self.length], self.v[:, :, :self.length]


class ResKVLlama:
    """Random-weight or loaded Llama decoder with a compressed (or dense) KV cache.

    ``generate(ids, new_tokens)`` = prefill + greedy decode.  With a process
    group the model is tensor-parallel over ``group`` (heads and FFN columns are
    sharded; ``shape.kv_heads`` must be divisible by the group size).
    """

    def __init__(self, shape: LlamaShape = LlamaShape(), kernel_config: ResKVKernelConfig | None = None, *,
                 cache: str = "reskv", device="cuda", seed: int = 0, group=None, prefill_chunk: int = 65536,
                 sink_tokens: int = 0):
        if cache not in ("reskv", "dense"):
            raise ValueError("cache must be 'reskv' or 'dense'")
        self.shape, self.cache_kind, self.device = shape, cache, torch.device(device)
        self.kernel_config = kernel_config or ResKVKernelConfig()
        if not isinstance(self.kernel_config, ResKVKernelConfig):
            raise TypeError(f"expected ResKVKernelConfig, got {type(self.kernel_config).__name__}")
        self.sink_tokens = int(sink_tokens)  # leading tokens kept dense (attention sinks); compression starts behind them
        self.group = group
        self.tp = 1 if group is None else torch.distributed.get_world_size(group)
        if shape.kv_heads % self.tp or shape.heads % self.tp or shape.ffn % self.tp:
            raise ValueError("heads, kv_heads and ffn must be divisible by the tensor-parallel size")
        self.h_q, self.h_kv, self.ffn = shape.heads // self.tp, shape.kv_heads // self.tp, shape.ffn // self.tp
        self.prefill_chunk = prefill_chunk
        rank = 0 if group is None else torch.distributed.get_rank(group)
        g = torch.Generator(device=self.device).manual_seed(seed)

        def w(rows, cols, std):
            # every rank draws the full matrix from the same seed and keeps its shard, so the
            # model is the same function for every tensor-parallel size
            return (torch.randn(rows, cols, generator=g, device=self.device, dtype=torch.float32) * std).half()

        def rows_of(full, per_rank):
            return full[rank * per_rank:(rank + 1) * per_rank].contiguous()

        d, hd = shape.hidden, shape.head_dim
        self.embed = w(shape.vocab, d, 1.0)
        self.lm_head = w(shape.vocab, d, d**-0.5)
        self.final_norm = torch.ones(d, dtype=torch.float16, device=self.device)
        self.layers = []
        for _ in range(shape.layers):
            wq, wk, wv = w(shape.heads * hd, d, d**-0.5), w(shape.kv_heads * hd, d, d**-0.5), w(shape.kv_heads * hd, d, d**-0.5)
            wo = w(d, shape.heads * hd, (shape.heads * hd) ** -0.5)
            wg, wu = w(shape.ffn, d, d**-0.5), w(shape.ffn, d, d**-0.5)
            wd = w(d, shape.ffn, shape.ffn**-0.5)
            self.layers.append({
                "norm1": torch.ones(d, dtype=torch.float16, device=self.device),
                "norm2": torch.ones(d, dtype=torch.float16, device=self.device),
                # [q | k | v] rows of this rank's heads ([out, in] for F.linear)
                "wqkv": torch.cat((rows_of(wq, self.h_q * hd), rows_of(wk, self.h_kv * hd), rows_of(wv, self.h_kv * hd))),
                "wo": wo[:, rank * self.h_q * hd:(rank + 1) * self.h_q * hd].contiguous(),
                "w_gate_up": torch.cat((rows_of(wg, self.ffn), rows_of(wu, self.ffn))),
                "w_down": wd[:, rank * self.ffn:(rank + 1) * self.ffn].contiguous(),
            })
            del wq, wk, wv, wo, wg, wu, wd
        self.inv_freq = (shape.rope_theta ** (-torch.arange(64, device=self.device).float() / 64)).contiguous()
        self.scaling = hd**-0.5
        self.caches = None
        self.length = 0
        self._lib = None
        # graph decode: the last captured graph (owner of the captures' memory pool), batch sizes whose step has run once
        self._last_graph = None
        self._warm = set()

    # -- helpers -----------------------------------------------------------------------------
    def _all_reduce(self, x):
        if self.tp > 1:
            torch.distributed.all_reduce(x, group=self.group)
        return x

    def _trig(self, start, n):
        ang = torch.arange(start, start + n, device=self.device).float()[:, None] * self.inv_freq[None, :]
        return ang.cos(), ang.sin()

    def _native(self):
        """The library with the model's device current, or ``None`` for a model on the CPU (dense cache only)."""
        from .._extension import bound_library

        if self._lib is None and self.device.type == "cuda":
            self._lib = bound_library(self.device)
        return self._lib

    def _norm(self, x, weight):
        # tensor operations, not the decode step's kernel: what is kept of a prompt's keys hangs on their last bit, and
        # the order of this sum decides it
        return _rms_norm(x, weight, self.shape.rms_eps)

    def _add_projection(self, x, inp, weight):
        """``x += inp @ weight^T`` in place (residual branch), summed over the tensor-parallel group."""
        x += self._all_reduce(F.linear(inp, weight))

    def _add_mlp(self, layer, x):
        """``x += MLP(norm(x))`` in place, at most ``prefill_chunk`` tokens at a time."""
        lib, flat = self._native(), x.view(-1, x.shape[-1])
        for i in range(0, flat.shape[0], self.prefill_chunk):
            part = flat[i:i + self.prefill_chunk]
            gu = F.linear(self._norm(part, layer["norm2"]), layer["w_gate_up"])
            if lib is None or self.ffn % 2:
                act = F.silu(gu[:, :self.ffn])
                act.mul_(gu[:, self.ffn:])
            else:
                from .._extension import _stream, check

                act = torch.empty((gu.shape[0], self.ffn), dtype=gu.dtype, device=gu.device)
                check(lib.reskv_silu_mul(gu.data_ptr(), act.data_ptr(), gu.shape[0], self.ffn, _stream(self.device)))
            del gu
            self._add_projection(part, act, layer["w_down"])

    def _qkv(self, layer, x, trig, k_raw, k_rot, v_all):
        """Projections of ``x [B,T,hidden]``: raw keys, rotated keys and values into the given ``[B,Hkv,T,128]``
        tensors; returns raw and rotated queries ``[B,Hq,T,128]``."""
        b, t, _ = x.shape
        cos, sin = trig
        qkv = F.linear(self._norm(x, layer["norm1"]), layer["wqkv"])
        lib = self._native()
        if lib is not None:
            from .._extension import _stream, check

            q_rot = torch.empty((b, self.h_q, t, 128), dtype=torch.float16, device=self.device)
            check(lib.reskv_rope_prompt(qkv.data_ptr(), b, t, self.h_q, self.h_kv, cos.data_ptr(), sin.data_ptr(),
                                        q_rot.data_ptr(), k_raw.data_ptr(), k_rot.data_ptr(), v_all.data_ptr(),
                                        _stream(self.device)))
            return qkv[..., :self.h_q * 128].unflatten(-1, (self.h_q, 128)).transpose(1, 2), q_rot
        q, k, v = (part.reshape(b, t, -1, 128).transpose(1, 2) for part in
                   qkv.split((self.h_q * 128, self.h_kv * 128, self.h_kv * 128), dim=-1))
        k_raw.copy_(k), v_all.copy_(v), k_rot.copy_(_rope(k, cos, sin))
        return q, _rope(q, cos, sin)

    # -- prefill / decode ----------------------------------------------------------------------
    @torch.no_grad()
    def prefill(self, ids: torch.Tensor, reserve: int = 0) -> torch.Tensor:
        """Run the prompt ``ids [B, T]``; builds the caches; returns last-token logits.

        Norms, projections, RoPE and the dense causal attention run over slices of the batch (at most
        ``prefill_chunk`` tokens at a time) so that their FP32 temporaries stay small at long contexts;
        the cache of a layer receives the whole batch at once."""
        b, t = ids.shape
        trig = self._trig(0, t)
        x = self.embed[ids]
        self.caches = []
        rows = max(1, self.prefill_chunk // t)  # sequences per slice
        half = dict(dtype=torch.float16, device=self.device)
        for layer in self.layers:
            k_raw = torch.empty((b, self.h_kv, t, 128), **half)
            k_rot, v_all = torch.empty_like(k_raw), torch.empty_like(k_raw)
            for i in range(0, b, rows):
                part = slice(i, i + rows)
                _, qr = self._qkv(layer, x[part], trig, k_raw[part], k_rot[part], v_all[part])
                att = F.scaled_dot_product_attention(qr, k_rot[part], v_all[part], is_causal=t > 1, enable_gqa=True,
                                                     scale=self.scaling)
                self._add_projection(x[part], att.transpose(1, 2).reshape(-1, t, self.h_q * 128), layer["wo"])
                del qr, att
            if self.cache_kind == "reskv":
                cache = ResKVLayerCache(self.kernel_config, self.sink_tokens)
                cache.update(k_rot, v_all, {"raw_keys": k_raw})
                if reserve and cache.compressed is not None:
                    cache.compressed = cache.compressed.reserve(cache.compressed.seq_len + reserve)
            else:
                cache = _DenseLayerCache(b, self.h_kv, t + reserve, self.device)
                cache.append(k_rot, v_all)
            self.caches.append(cache)
            del k_raw, k_rot, v_all
            self._add_mlp(layer, x)
        self.length = t
        return self._logits(x[:, -1:])

    def _logits(self, x):
        return F.linear(self._norm(x, self.final_norm), self.lm_head)[:, 0].float()

    @torch.no_grad()
    def decode(self, tokens: torch.Tensor) -> torch.Tensor:
        """One step for ``tokens [B]``; returns logits ``[B, vocab]``."""
        b = tokens.shape[0]
        pos = self.length
        trig = self._trig(pos, 1)
        x = self.embed[tokens].unsqueeze(1)
        for layer, cache in zip(self.layers, self.caches):
            k, kr, v = torch.empty((3, b, self.h_kv, 1, 128), dtype=torch.float16, device=self.device)
            q, qr = self._qkv(layer, x, trig, k, kr, v)
            if self.cache_kind == "reskv":
                keys, values = cache.update(kr, v, {"raw_keys": k})
                if cache.compressed is not None:
                    att = attention(q.contiguous(), cache.compressed, position=pos, start_position=cache.start_position,
                                    inv_freq=self.inv_freq, scaling=self.scaling, recent=(qr, keys, values))
                else:
                    att = F.scaled_dot_product_attention(qr, keys, values, enable_gqa=True, scale=self.scaling)
            else:
                keys, values = cache.append(kr, v)
                att = F.scaled_dot_product_attention(qr, keys, values, enable_gqa=True, scale=self.scaling)
            self._add_projection(x, att.transpose(1, 2).reshape(b, 1, -1), layer["wo"])
            self._add_mlp(layer, x)
        self.length += 1
        return self._logits(x)

    @torch.no_grad()
    def generate(self, ids: torch.Tensor, new_tokens: int) -> torch.Tensor:
        """Greedy continuation ``[B, new_tokens]`` of the prompt ``ids [B, T]``."""
        logits = self.prefill(ids, reserve=new_tokens)
        out = [logits.argmax(-1)]
        for _ in range(new_tokens - 1):
            out.append(self.decode(out[-1]).argmax(-1))
        return torch.stack(out, dim=1)

    # -- CUDA-graph decode ------------------------------------------------------------------------
    # RESKV_CHECK_STATUS=1: every step is waited for, and a kernel's bounded wait that ran out (or a step state beyond its
    # buffers) raises instead of leaving wrong logits
    _check_status = os.environ.get("RESKV_CHECK_STATUS") == "1"

    def _raise_on_status(self):
        from .._extension import _stream, check

        linear = ctypes.c_uint32(0)
        check(self._native().reskv_skinny_linear_status(ctypes.addressof(linear), _stream(self.device)), launches=0)
        decode = self._workspace[:4].view(torch.int32).item() if self.cache_kind == "reskv" else 0
        if linear.value or decode:
            raise RuntimeError(f"decode step: device status 0x{linear.value:x} (linear layers), 0x{decode:x} (attention)")

    # A decode step is ~20 small launches per layer; at small batch the GPU waits for Python.  The
    # step is therefore captured once per "epoch" (the 64 steps between two group compressions, in
    # which the compressed segment is fixed) and replayed: query position and window length live in
    # a device-side step state that the append / decode kernels read and a final kernel advances.
    def _step_body(self, tok):
        from .._extension import (LAYOUT_COMPACT, LAYOUT_STRUCTURED, LAYOUT_TILED, LAYOUT_UNSTRUCTURED, _stream,
                                  bound_library, check)

        lib = bound_library(self.device)  # every launch below runs with the model's device current
        b = tok.shape[0]
        d = self.shape.hidden
        stream = _stream(self.device)
        state = self._state.data_ptr()
        reskv = self.cache_kind == "reskv"

        def half(*shape):
            return torch.empty(shape, dtype=torch.float16, device=self.device)

        def norm(x, weight):
            if not (_dense_half(x, (b, d), x.device) and _dense_half(weight, (d,), x.device)):
                return self._norm(x, weight)
            out = half(b, d)
            check(lib.reskv_rms_norm(x.data_ptr(), weight.data_ptr(), out.data_ptr(), b, d, float(self.shape.rms_eps), stream))
            return out

        def ptr(t):
            return None if t is None else t.data_ptr()

        def streams(x, weight, n, mode, norm_weight=None):
            """Whether the library's own weight stream, for few rows, takes the sizes, and the tensors as they are.  Asked
            while a step is captured only: a replay pays nothing for it."""
            k = x.shape[-1]
            return (lib.reskv_skinny_linear_fits(b, n, k, mode) and _dense_half(x, (b, k), x.device)
                    and _dense_half(weight, (2 * n if mode == 2 else n, k), x.device)
                    and (norm_weight is None or _dense_half(norm_weight, (k,), x.device)))

        def stream_weight(x, weight, mode, out, norm_weight=None):
            check(lib.reskv_skinny_linear(x.data_ptr(), ptr(norm_weight), float(self.shape.rms_eps), weight.data_ptr(),
                                          out.data_ptr(), b, out.shape[-1], x.shape[-1], mode, stream))
            return out

        def linear(x, weight, norm_weight):
            """norm(x) @ weight^T"""
            n = weight.shape[0]
            if streams(x, weight, n, 0, norm_weight):
                return stream_weight(x, weight, 0, half(b, n), norm_weight)
            return F.linear(norm(x, norm_weight), weight)

        def project(x, inp, weight):
            """x + inp @ weight^T, summed over the tensor-parallel group."""
            if self.tp == 1:
                if _dense_half(x, (b, d), inp.device) and streams(inp, weight, d, 1):
                    return stream_weight(inp, weight, 1, x)
                return x.addmm_(inp, weight.t())  # in place: no copy of x in front of the product
            return x + self._all_reduce(F.linear(inp, weight))

        # one step on: the new token's position, and (compressed cache) its place in the window -- it goes to slot
        # count - 1 and the attention of this step already includes it
        check(lib.reskv_step_advance(state, 1, 1 if reskv else 0, stream))
        x = self.embed[tok]
        for index, (layer, cache) in enumerate(zip(self.layers, self.caches)):
            qkv = linear(x, layer["wqkv"], layer["norm1"])
            q_rot = half(b * self.h_q, 128)
            if reskv:
                cap = cache.keys.shape[2]
                q_raw = half(b * self.h_q, 128)
                check(lib.reskv_rope_split(qkv.data_ptr(), b, self.h_q, self.h_kv, self.inv_freq.data_ptr(), state,
                                           q_raw.data_ptr(), q_rot.data_ptr(), None, None, cache.keys.data_ptr(),
                                           cache.raw_keys.data_ptr(), cache.values.data_ptr(), cap, stream))
                key, val = cache.compressed.key, cache.compressed.value
                plan = key.plan
                _, ki, kp, km, ks = key._native
                _, vi, vp, vm, vs = val._native
                kc, vc = self._centroids[index]
                layout = {"unstructured": LAYOUT_UNSTRUCTURED, "tiled": LAYOUT_TILED, "structured": LAYOUT_STRUCTURED,
                          "compact": LAYOUT_COMPACT}[plan.layout]
                att = half(b, self.h_q * 128)
                # token count and centroid tables are read from the step state / fixed-shape tables,
                # so the captured launch stays valid when a group is compressed between replays
                check(lib.reskv_decode_step(layout, plan.bits, plan.nnz, q_raw.data_ptr(), kc.data_ptr(), ki.data_ptr(),
                                            kp.data_ptr(), ptr(km), ptr(ks), vc.data_ptr(), vi.data_ptr(), vp.data_ptr(),
                                            ptr(vm), ptr(vs), b, self.h_kv, self.h_q, key.seq_len, key.token_stride,
                                            kc.shape[1], vc.shape[1], cache.start_position, float(self.shape.rope_theta),
                                            self.inv_freq.data_ptr(), float(self.scaling), 0, q_rot.data_ptr(),
                                            cache.keys.data_ptr(), cache.values.data_ptr(), cap, state,
                                            self._workspace.data_ptr(), self._workspace.numel(), att.data_ptr(), stream),
                      launches=2)
            elif _flash_kvcache is not None:
                k_rot, v_new = half(b, 1, self.h_kv, 128), half(b, 1, self.h_kv, 128)
                check(lib.reskv_rope_split(qkv.data_ptr(), b, self.h_q, self.h_kv, self.inv_freq.data_ptr(), state,
                                           None, q_rot.data_ptr(), k_rot.data_ptr(), v_new.data_ptr(), None, None, None,
                                           0, stream))
                att = _flash_kvcache(q_rot.view(b, 1, self.h_q, 128), cache.k, cache.v, k=k_rot, v=v_new,
                                     cache_seqlens=self._seqlens, softmax_scale=self.scaling, causal=True)
                att = att.reshape(b, self.h_q * 128)
            else:
                raise RuntimeError("graph decode of the dense baseline needs flash_attn")
            x = project(x, att, layer["wo"])
            act = half(b, self.ffn)
            if streams(x, layer["w_gate_up"], self.ffn, 2, layer["norm2"]):
                stream_weight(x, layer["w_gate_up"], 2, act, layer["norm2"])
            else:
                gate_up = F.linear(norm(x, layer["norm2"]), layer["w_gate_up"])
                check(lib.reskv_silu_mul(gate_up.data_ptr(), act.data_ptr(), b, self.ffn, stream))
            x = project(x, act, layer["w_down"])
        if not reskv:
            self._seqlens += 1
        vocab = self.lm_head.shape[0]
        if streams(x, self.lm_head, vocab, 3, self.final_norm):
            logits = torch.empty((b, vocab), dtype=torch.float32, device=self.device)
            return stream_weight(x, self.lm_head, 3, logits, self.final_norm)
        return F.linear(norm(x, self.final_norm), self.lm_head).float()

    @torch.no_grad()
    def begin_graph_decode(self, batch: int):
        """Prepare static buffers after ``prefill``; call once before ``decode_graph``."""
        from .._extension import library

        self._tok_in = torch.zeros(batch, dtype=torch.long, device=self.device)
        self._graph = self._logits_out = None
        if self.cache_kind == "reskv":
            self._state = torch.zeros(4, dtype=torch.int32, device=self.device)
            # centroid tables at their final shape (zero rows beyond the live count), one pair per layer
            rows = self.kernel_config.max_clusters
            self._centroids = [tuple(torch.zeros((batch * self.h_kv, rows, 128), dtype=torch.float16, device=self.device)
                                     for _ in range(2)) for _ in self.caches]
            self._sync_graph_inputs()
            # scratch for any compressed length up to 2^20 tokens with the library's own schedule
            need = library().reskv_decode_bitmap_fp16_workspace_bytes(batch, self.h_kv, self.h_q, 1 << 20, 0)
            self._workspace = torch.zeros(need, dtype=torch.uint8, device=self.device)
        else:
            if _flash_kvcache is None:
                raise RuntimeError("graph decode of the dense baseline needs flash_attn")
            self._state = torch.tensor([self.length - 1, 0], dtype=torch.int32, device=self.device)
            self._seqlens = torch.full((batch,), self.length, dtype=torch.int32, device=self.device)
            for c in self.caches:  # flash_attn_with_kvcache wants [B, T, H, D]
                c.k = c.k.transpose(1, 2).contiguous()
                c.v = c.v.transpose(1, 2).contiguous()

    def _sync_graph_inputs(self):
        """Refresh what a captured step reads: counts in the step state, centroid tables, and the
        addresses of the compressed buffers (a buffer that had to grow invalidates the graph)."""
        comp = self.caches[0].compressed
        self._state.copy_(torch.tensor([self.length - 1, self.caches[0].live, comp.seq_len if comp is not None else -1, 0],
                                       dtype=torch.int32))
        addresses = []
        for cache, (kc, vc) in zip(self.caches, self._centroids):
            if cache.compressed is None:
                raise RuntimeError("graph decode needs a compressed segment (prompt shorter than recent + group)")
            for table, tensor in ((kc, cache.compressed.key), (vc, cache.compressed.value)):
                native = tensor._native
                table[:, :native[0].shape[1]].copy_(native[0])
                addresses += [t.data_ptr() for t in native[1:] if t is not None] + [tensor.token_stride]
        if addresses != getattr(self, "_graph_addresses", None):
            self._graph_addresses = addresses
            self._graph = None

    def _capture_step(self):
        """Capture one decode step as a CUDA graph.

        ``torch.cuda.graph`` would collect garbage and empty the allocator's cache first, and everything a server
        allocates next would go back to ``cudaMalloc`` (72 of 114 ms for a prompt of 4 x 1024 tokens and 72 steps).  The
        step's temporaries come from one pool per model: the graph captured last stays alive, and with it the pool,
        until the next capture has taken the pool over."""
        side, main = _capture_stream(self.device), torch.cuda.current_stream(self.device)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            if self._tok_in.shape[0] not in self._warm:
                # once per batch size: a step outside capture (library handles, lazy inits), on a state that is restored
                reskv = self.cache_kind == "reskv"
                counts = self._state if reskv else self._seqlens
                saved, saved_state = counts.clone(), self._state.clone()
                self._step_body(self._tok_in)
                self._state.copy_(saved_state)
                if not reskv:
                    counts.copy_(saved)
                self._warm.add(self._tok_in.shape[0])
            graph = torch.cuda.CUDAGraph()
            with _collector_held():
                graph.capture_begin(pool=None if self._last_graph is None else self._last_graph.pool())
                try:
                    self._logits_out = self._step_body(self._tok_in)
                finally:
                    graph.capture_end()
        main.wait_stream(side)
        self._graph = self._last_graph = graph

    @torch.no_grad()
    def decode_graph(self, tokens: torch.Tensor) -> torch.Tensor:
        """Same result as ``decode`` but replaying a captured CUDA graph of the step."""
        if self.cache_kind == "reskv" and self.caches[0].live + 1 == self.caches[0].keys.shape[2]:
            # this token fills the window.  The eager step appends it and then compresses the oldest
            # group before attending (as the reference does); the group does not contain the new
            # token, so compressing it first and appending afterwards gives the same cache.  That is
            # done here, outside the graph; the graph then only needs the new counts.
            for cache in self.caches:
                cache._compress_oldest_group()
            self._sync_graph_inputs()
        self._tok_in.copy_(tokens)
        if self._graph is None:
            self._capture_step()
        self._graph.replay()
        if self._check_status:
            self._raise_on_status()
        self.length += 1
        if self.cache_kind == "reskv":
            for cache in self.caches:
                cache.live += 1
                cache.length += 1
        return self._logits_out

    def cache_bytes(self) -> int:
        total = 0
        for c in self.caches or []:
            if isinstance(c, _DenseLayerCache):
                total += c.k.nbytes + c.v.nbytes
            else:
                total += (c.compressed.nbytes if c.compressed is not None else 0)
                total += c.keys.nbytes + c.raw_keys.nbytes + c.values.nbytes
        return total
