"""Model modules (drop-in for the reference's ``dia/layers.py``).

Same class names, constructor signatures and state_dict keys / shapes as the reference
(``DenseGeneral`` dia/layers.py:17-66, ``MlpBlock`` :69-105, ``RotaryEmbedding`` :108-173,
``Attention`` :176-346, ``EncoderLayer`` :349-416, ``Encoder`` :419-462, ``DecoderLayer`` :465-584,
``Decoder`` :587-766, ``DiaModel`` :769-807), so reference checkpoints, ``prune`` masks on
``.weight`` and PEFT target names keep working.

What runs where
  * ``Decoder.decode_step`` and ``DecoderLayer.forward`` at T=1 - the autoregressive hot path - run
    entirely in the hand-written sm_100a kernels of ``csrc/`` through the C ABI (``engine.py``).
    There is no eager fallback for them: without a CUDA device they raise.
  * ``Encoder``, ``Decoder.precompute_cross_attn_cache`` and the prompt prefill (``Decoder.forward``)
    are once-per-utterance work.  A layer of these T > 1 passes is one native call (``_rows_layer``): its dense layers run on
    the tcgen05 / TMEM GEMMs of ``csrc/gemm_tcgen05.cu``, its attention on the kernels of ``csrc/prefill_kernels.cu`` and
    ``csrc/attention_split.cu``.  The results feed the decode kernels through the KV caches.
  * Pruned checkpoints: ``Decoder.engine()`` drops exactly-dead MLP neurons from the weight stream and streams a
    2:4 model compressed on ``mma.sp`` (``pruning_utils``).

Numerics: dense kernels may be stored bf16 (``compute_dtype``), but activations, residual stream,
norms, softmax and KV caches are always fp32.
"""

from __future__ import annotations

import contextlib
import math
import os
import weakref
from typing import Callable, Optional

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch import Tensor
from torch.nn import RMSNorm

try:  # hub mixin gives DiaModel.from_pretrained / save_pretrained exactly like the reference
    from huggingface_hub import PyTorchModelHubMixin
except Exception:  # pragma: no cover - hub not installed
    class PyTorchModelHubMixin:  # type: ignore
        def __init_subclass__(cls, **kw):
            super().__init_subclass__()

from . import _lib
from ._lib import RowsLayer
from .config import DiaConfig
from .state import DecoderInferenceState, EncoderInferenceState, KVCache


@contextlib.contextmanager
def _exact_fp32():
    """fp32 library GEMMs without TF32 (the K/V they produce are re-read by every decode step)."""
    if not torch.cuda.is_available():
        yield
        return
    a, b = torch.backends.cuda.matmul.allow_tf32, torch.backends.cudnn.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    torch.backends.cudnn.allow_tf32 = False
    try:
        yield
    finally:
        torch.backends.cuda.matmul.allow_tf32, torch.backends.cudnn.allow_tf32 = a, b


class DenseGeneral(nn.Module):
    """Bias-free generalised dense layer with a JAX-layout kernel ``in_shapes + out_features``."""

    def __init__(self, in_shapes: tuple[int, ...], out_features: tuple[int, ...], axis: tuple[int, ...] = (-1,),
                 weight_dtype: torch.dtype | None = None, device: torch.device | None = None):
        super().__init__()
        self.in_shapes, self.out_features, self.axis = in_shapes, out_features, axis
        self.kernel_shape = self.in_shapes + self.out_features
        self.weight = nn.Parameter(torch.empty(self.kernel_shape, dtype=weight_dtype, device=device))

    # the K-major bf16 copy the tcgen05 GEMM reads is keyed by (data_ptr, version): drop it whenever the parameter object
    # is replaced (torch.nn.utils.prune, load_state_dict(assign=True)) or moved (.to / .cpu / .cuda) - a new tensor can
    # land on the very address the old one had
    def __setattr__(self, name, value):
        if name in ("weight", "weight_orig", "weight_mask"):
            self._drop_copies()
        super().__setattr__(name, value)

    def __delattr__(self, name):
        if name in ("weight", "weight_orig", "weight_mask"):
            self._drop_copies()
        super().__delattr__(name)

    def _apply(self, fn, *a, **kw):
        self._drop_copies()
        return super()._apply(fn, *a, **kw)

    def _drop_copies(self) -> None:
        self.__dict__.pop("_b200_wt", None)
        self.__dict__.pop("_b200_half", None)

    def forward(self, inputs: Tensor) -> Tensor:
        """``tensordot(x, W)`` over ``axis`` (dia/layers.py:55-66).  On a CUDA device every call runs on the tcgen05
        GEMM of ``csrc/gemm_tcgen05.cu``; there is no library fallback on that device.  On the CPU (state-dict
        tooling, pruning, the CPU test suite) and under autograd (fine-tuning is outside this path) it is the
        reference's own tensordot."""
        n = len(self.axis)
        x_axes = tuple(a if a >= 0 else inputs.ndim + a for a in self.axis)
        w = self.weight
        if inputs.is_cuda and w.is_cuda and not (torch.is_grad_enabled() and (w.requires_grad or inputs.requires_grad)):
            return self._forward_tcgen05(inputs, x_axes)
        out = torch.tensordot(inputs.to(torch.float32), w.to(torch.float32), dims=(x_axes, tuple(range(n))))
        return out.to(inputs.dtype)

    # ---- sm_100a path (encoder, cross-attention K/V precompute, prompt prefill) ----------------------------------
    def kernel_weight_kmajor(self) -> Tensor:
        """The K-major bf16 copy ``[N, K]`` of the kernel the tcgen05 GEMM reads (made once per weight version)."""
        if not self._has_kmajor():
            make_kmajor_kernels([[self]])
        return self._b200_wt[1]

    def _has_kmajor(self) -> bool:
        cached = self.__dict__.get("_b200_wt")
        return cached is not None and cached[0] == self._weight_key()

    def kernel_weight_half(self) -> tuple[Tensor, Tensor] | None:
        """The fp16 copy that products of many rows read (made once per weight version), or None: fp16 cannot hold these weights, or the
        stream is being captured and there is no copy yet."""
        cached = self.__dict__.get("_b200_half")
        if cached is None or cached[0] != self._weight_key():
            if torch.cuda.is_current_stream_capturing():
                return None
            prepare_half_kernels([self])
            cached = self._b200_half
        return cached[1]

    def _weight_key(self):
        w = self.weight
        return (w.data_ptr(), w._version, w.dtype, w.device)

    def _forward_tcgen05(self, inputs: Tensor, x_axes: tuple[int, ...], norm_weight: Tensor | None = None,
                         eps: float = 1e-5, residual: Tensor | None = None) -> Tensor:
        """``x @ W`` on the tcgen05 tensor cores with the activations split into three bf16 terms or, for many rows, two fp16 terms (float32-operand
        accuracy).  ``norm_weight``: RMSNorm of the input rows fused into the split pass; ``residual``: added in the
        epilogue (the result aliases it)."""
        from . import engine as _engine
        n = len(x_axes)
        if x_axes != tuple(range(inputs.ndim - n, inputs.ndim)):
            raise NotImplementedError("DenseGeneral on sm_100a contracts the trailing axes only")
        K, N = math.prod(self.in_shapes), math.prod(self.out_features)
        M = inputs.numel() // K if K else 0
        lead = inputs.shape[: inputs.ndim - n]
        if M == 0:
            return torch.zeros((*lead, *self.out_features), dtype=torch.float32, device=inputs.device)
        if not _engine.dense_supported(M, N, K):
            raise NotImplementedError(f"dense layer [{M} x {K}] . [{K} x {N}] does not fit the tcgen05 tiling "
                                      f"(K must be a multiple of 64, N of 4)")
        if _engine.dense_half_rows(M, N, K, inputs.device):
            x, r = inputs.reshape(M, K), None if residual is None else residual.reshape(M, N)
            half = self.kernel_weight_half() if _plain(x, norm_weight, r) else None
            if half is not None:
                return _engine.dense_forward_half(x, half, norm_weight, eps, r).reshape(*lead, *self.out_features)
        y = _engine.dense_forward(inputs.reshape(M, K), self.kernel_weight_kmajor(), norm_weight=norm_weight, eps=eps,
                                  residual=None if residual is None else residual.reshape(M, N))
        return y.reshape(*lead, *self.out_features)


def _plain(*tensors: Tensor | None) -> bool:
    """float32, contiguous and 16-byte aligned."""
    return all(t is None or (t.dtype == torch.float32 and t.is_contiguous() and t.data_ptr() % 16 == 0) for t in tensors)


@torch.no_grad()
def make_kmajor_kernels(groups: list[list["DenseGeneral"]]) -> None:
    """K-major copies of these kernels, those of a group one behind the other (products of the same rows may then be one product).  Any stream may read a
    copy once it is kept, so they are waited for (but for a capture, whose graph makes them)."""
    from . import engine as _engine
    made = []
    for modules in groups:
        for m in modules:
            canonicalize_dense_kernel_(m)
        K, sizes = math.prod(modules[0].in_shapes), [math.prod(m.out_features) for m in modules]
        rows = torch.empty((sum(sizes), K), dtype=torch.bfloat16, device=modules[0].weight.device)
        made += [(m, _engine.dense_prepare_weight(m.weight.detach().reshape(K, out.shape[0]), out)) for m, out in zip(modules, rows.split(sizes))]
    if rows.is_cuda and not torch.cuda.is_current_stream_capturing():
        torch.cuda.current_stream(rows.device).synchronize()
    for m, wt in made:
        m._b200_wt = (m._weight_key(), wt)


@torch.no_grad()
def prepare_half_kernels(modules: list["DenseGeneral"]) -> None:
    """The fp16 copies of these kernels, with one look at whether they are exact for all of them."""
    from . import engine as _engine
    def missing(m):
        cached = m.__dict__.get("_b200_half")
        return cached is None or cached[0] != m._weight_key()

    todo = [m for m in modules if missing(m)]
    for m in todo:
        canonicalize_dense_kernel_(m)
    if not todo:
        return
    flags = torch.zeros((len(todo),), dtype=torch.int32, device=todo[0].weight.device)
    halves = [_engine.dense_prepare_half(m.weight.detach().reshape(math.prod(m.in_shapes), math.prod(m.out_features)), flags[i:i + 1])
              for i, m in enumerate(todo)]
    for m, half, inexact in zip(todo, halves, flags.tolist()):
        m._b200_half = (m._weight_key(), None if inexact else half)


_ROUNDING_WARNED = False


@torch.no_grad()
def canonicalize_dense_kernel_(m: "DenseGeneral") -> bool:
    """The sm_100a kernels stream DenseGeneral kernels as bf16 (activations, norms, softmax and caches stay fp32).
    A float16 kernel is widened to float32 first (exact); a kernel that is not bf16-representable - a real float32
    or float16 checkpoint - is rounded to bf16 ONCE, in place, with a warning, so that the encoder, the prompt
    prefill and the decode engine all see the very same numbers.  Returns True if values changed."""
    global _ROUNDING_WARNED
    w = m.weight
    if w.dtype == torch.bfloat16:
        return False
    if w.dtype == torch.float16:
        w.data = w.data.to(torch.float32)
    r = w.data.to(torch.bfloat16).to(torch.float32)
    if torch.equal(r, w.data):
        return False
    if not _ROUNDING_WARNED:
        import warnings
        warnings.warn("dia_tts_prune_b200: DenseGeneral kernels are not bf16-representable; rounding them to bf16 once "
                      "(the sm_100a path keeps weights in bf16 and everything else in fp32: logits differ from the "
                      "float32 reference by ~1e-2, as with the reference's own compute_dtype='bfloat16')", stacklevel=3)
        _ROUNDING_WARNED = True
    w.data.copy_(r)
    return True


def canonicalize_dense_kernels_(model: nn.Module) -> int:
    """:func:`canonicalize_dense_kernel_` over every DenseGeneral of ``model``; returns how many were rounded."""
    return sum(1 for m in model.modules() if isinstance(m, DenseGeneral) and canonicalize_dense_kernel_(m))


class MlpBlock(nn.Module):
    def __init__(self, embed_dim: int, intermediate_dim: int, compute_dtype: torch.dtype):
        super().__init__()
        self.dtype = compute_dtype
        self.wi_fused = DenseGeneral((embed_dim,), (2, intermediate_dim), axis=(-1,), weight_dtype=compute_dtype)
        self.wo = DenseGeneral((intermediate_dim,), (embed_dim,), axis=(-1,), weight_dtype=compute_dtype)

    def forward(self, x: Tensor) -> Tensor:
        gu = self.wi_fused(x)                               # [..., 2, F]: gate columns first, then up
        if x.is_cuda and not torch.is_grad_enabled():
            from . import engine as _k
            h = _k.silu_mul(gu.reshape(-1, 2, gu.shape[-1]))
            return self.wo(h.reshape(*x.shape[:-1], -1))
        return self.wo(F.silu(gu[..., 0, :].float()).to(x.dtype) * gu[..., 1, :])


class RotaryEmbedding(nn.Module):
    """Half-split RoPE, theta = position * max_timescale^(-2i/d) (intended semantics of
    dia/layers.py:126-173; the shipped forward has a shape bug)."""

    def __init__(self, embedding_dims: int, min_timescale: int = 1, max_timescale: int = 10000,
                 dtype: torch.dtype = torch.float32):
        super().__init__()
        if embedding_dims % 2:
            raise ValueError("Embedding dim must be even for RoPE.")
        self.embedding_dims, self.min_timescale, self.max_timescale = embedding_dims, min_timescale, max_timescale
        self.compute_dtype = dtype
        fraction = (2.0 * torch.arange(0, embedding_dims // 2)) / embedding_dims
        inv = 1.0 / (min_timescale * (max_timescale / min_timescale) ** fraction)
        self.register_buffer("inv_freq", inv.to(torch.float32), persistent=False)

    def forward(self, inputs: Tensor, position: Tensor) -> Tensor:
        theta = (position[..., None, None] * self.inv_freq.to(position.device)).to(torch.float32)   # [B,T,1,d/2]
        sin, cos = torch.sin(theta), torch.cos(theta)
        a, b = inputs.to(torch.float32).chunk(2, dim=-1)
        return torch.cat((a * cos - b * sin, a * sin + b * cos), dim=-1)


class Attention(nn.Module):
    """Library (fp32) attention used off the hot path: encoder, cross-KV precompute, prompt prefill."""

    def __init__(self, config: DiaConfig, q_embed_dim: int, kv_embed_dim: int, num_query_heads: int,
                 num_kv_heads: int, head_dim: int, compute_dtype: torch.dtype, is_cross_attn: bool = False,
                 out_embed_dim: int | None = None):
        super().__init__()
        if num_query_heads % num_kv_heads:
            raise ValueError(f"num_query_heads ({num_query_heads}) must be divisible by num_kv_heads ({num_kv_heads})")
        self.num_query_heads, self.num_kv_heads, self.head_dim = num_query_heads, num_kv_heads, head_dim
        self.is_cross_attn = is_cross_attn
        self.output_dim = out_embed_dim if out_embed_dim is not None else q_embed_dim
        self.projected_query_dim = num_query_heads * head_dim
        self.num_gqa_groups = num_query_heads // num_kv_heads
        self.compute_dtype = compute_dtype
        self.q_proj = DenseGeneral((q_embed_dim,), (num_query_heads, head_dim), axis=(-1,), weight_dtype=compute_dtype)
        self.k_proj = DenseGeneral((kv_embed_dim,), (num_kv_heads, head_dim), axis=(-1,), weight_dtype=compute_dtype)
        self.v_proj = DenseGeneral((kv_embed_dim,), (num_kv_heads, head_dim), axis=(-1,), weight_dtype=compute_dtype)
        self.o_proj = DenseGeneral((num_query_heads, head_dim), (self.output_dim,), axis=(-2, -1),
                                   weight_dtype=compute_dtype)
        self.rotary_emb = RotaryEmbedding(head_dim, config.model.rope_min_timescale, config.model.rope_max_timescale,
                                          dtype=compute_dtype)

    def forward(self, Xq: Tensor, Xkv: Tensor, q_positions: Tensor, kv_positions: Tensor | None = None,
                attn_mask: Tensor | None = None, cache: KVCache | None = None, prefill: bool = False,
                is_causal: bool = False) -> Tensor:
        if kv_positions is None:
            kv_positions = q_positions
        q = self.rotary_emb(self.q_proj(Xq.float()), q_positions).transpose(1, 2)          # [B, Hq, Tq, d]
        if self.is_cross_attn and cache is not None:
            # K/V were precomputed from the encoder output; the reference's per-step re-projection of
            # Xkv here is dead work (its result is discarded, dia/layers.py:274-275,284-287) and is omitted
            k, v = cache.k, cache.v
        else:
            k = self.rotary_emb(self.k_proj(Xkv.float()), kv_positions).transpose(1, 2)
            v = self.v_proj(Xkv.float()).transpose(1, 2)
            if cache is not None:
                k, v = cache.prefill(k, v) if prefill else cache.update(k, v)
        if self.num_gqa_groups > 1:
            k = k.repeat_interleave(self.num_gqa_groups, dim=1)
            v = v.repeat_interleave(self.num_gqa_groups, dim=1)
        out = F.scaled_dot_product_attention(q, k.float(), v.float(), attn_mask=attn_mask,
                                             is_causal=is_causal and not self.is_cross_attn, dropout_p=0.0)
        if attn_mask is not None and attn_mask.dtype == torch.bool:
            # a query with no allowed key contributes exact zeros (the reference's CPU SDPA behaviour,
            # made explicit here because GPU SDPA backends may return NaN there
            out = torch.where(attn_mask.any(dim=-1, keepdim=True), out, torch.zeros((), dtype=out.dtype, device=out.device))
        return self.o_proj(out.transpose(1, 2).contiguous()).to(Xq.dtype)


def _rows_kernels(D: int, attn: Attention, mlp: MlpBlock, cross: Attention | None) -> tuple[list[DenseGeneral], tuple[tuple[int, int], ...]]:
    """The dense kernels of a native layer call in its order, and the sizes ``(N, K)`` with which it reads them."""
    wo = mlp.wo
    F, Nq, Nk = wo.in_shapes[0], attn.num_query_heads * 128, attn.num_kv_heads * 128
    modules, sizes = [attn.q_proj, attn.k_proj, attn.v_proj, attn.o_proj, mlp.wi_fused, wo], ((Nq, D), (Nk, D), (Nk, D), (D, Nq), (2 * F, D), (D, F))
    if cross is not None:
        Nc = cross.num_query_heads * 128
        modules += (cross.q_proj, cross.o_proj)
        sizes += ((Nc, D), (D, Nc))
    return modules, sizes


def _kmajor_groups(modules: list[DenseGeneral], missing: list[DenseGeneral]) -> list[list[DenseGeneral]]:
    """How the missing K-major copies of a layer's kernels are made: q, k and v together, whichever of them is missing, unless one has a copy - that may be read
    by another stream or a captured graph, and stays while its weights do."""
    group = modules[:3] if any(m in missing for m in modules[:3]) and not any(m._has_kmajor() for m in modules[:3]) else []
    if len({math.prod(m.in_shapes) for m in group}) > 1:
        group = []                                                # (not products of the same rows)
    return ([group] if group else []) + [[m] for m in missing if m not in group]


def _prepare_for_rows(layers, M: int, D: int, device: torch.device) -> None:
    """The copies that calls of ``M`` rows read of all of these layers, with one look at them and one wait, where the last layer has none
    of its own yet."""
    from . import engine as _k
    def kernels_of(layer):
        return _rows_kernels(D, layer.self_attention, layer.mlp, getattr(layer, "cross_attention", None))

    modules, sizes = kernels_of(layers[-1])
    probe, two = modules[5], _k.dense_half_choice(M, sizes, device)[5]
    half = probe.__dict__.get("_b200_half")
    if (half is not None and half[0] == probe._weight_key() if two else probe._has_kmajor()) or torch.cuda.is_current_stream_capturing():
        return
    kernels = [kernels_of(layer) for layer in layers]
    choices = [_k.dense_half_choice(M, sizes, device) for _, sizes in kernels]
    prepare_half_kernels([m for (modules, _), choice in zip(kernels, choices) for m, two in zip(modules, choice) if two])
    groups = []
    for (modules, _), choice in zip(kernels, choices):
        groups += _kmajor_groups(modules, [m for m, two in zip(modules, choice) if not (two and m.kernel_weight_half() is not None) and not m._has_kmajor()])
    if groups:
        make_kmajor_kernels(groups)


def _rows_weights(a, M: int, attn: Attention, norm: RMSNorm, mlp: MlpBlock, norm_mlp: RMSNorm, cross: Attention | None, norm_cross: RMSNorm | None,
                  device) -> list:
    """Points the arguments of a native layer call of ``M`` rows at the layer's weights.  Returns what has to live until the call has been made.
    Nothing is kept from one call for the next but the copies that the kernels hold themselves: arguments kept per layer held copies that their
    kernels had dropped, and were made anew for every other number of rows (host time of a layer's
    arguments, us: 27 for any number of rows; kept ones 16 for the last number and 60 for another)."""
    from . import engine as _k
    D, keep = a.D, []
    a.F, a.heads, a.kv_heads = mlp.wo.in_shapes[0], attn.num_query_heads, attn.num_kv_heads
    modules, sizes = _rows_kernels(D, attn, mlp, cross)
    norms = [("norm_self", norm), ("norm_mlp", norm_mlp)]
    if cross is not None:
        a.cross_heads = cross.num_query_heads
        norms.append(("norm_cross", norm_cross))
    for name, n in norms:
        w = n.weight
        if w.numel() != D:
            raise ValueError("norm weight length must equal K")
        if w.dtype != torch.float32 or not w.is_contiguous():
            w = w.detach().to(torch.float32).contiguous()
        keep.append(w)
        setattr(a, name, w.data_ptr())
    copies, missing = [], []
    for m, two in zip(modules, _k.dense_half_choice(M, sizes, device)):
        h = m.kernel_weight_half() if two else None               # (the product's rows go as two fp16 terms)
        if h is None:
            c = m.__dict__.get("_b200_wt")
            if c is None or c[0] != m._weight_key():
                missing.append(m)
        copies.append(h)
    if missing:
        make_kmajor_kernels(_kmajor_groups(modules, missing))
    pointers = []
    for m, size, h in zip(modules, sizes, copies):
        wt = m._b200_wt[1] if h is None else h[0]
        if wt.shape != size:                                      # the native call takes its sizes from D, F and the heads
            raise NotImplementedError(f"a layer of width {D} on sm_100a has heads of 128 channels: dense kernel {tuple(m.kernel_shape)} where {size[::-1]} is read")
        keep.append(wt)
        if h is None:
            pointers += (wt.data_ptr(), 0, 0)
        else:
            keep.append(h)
            pointers += (0, wt.data_ptr(), h[1].data_ptr())
    _lib.set_kernels(a, pointers)
    return keep


def _check_caches(name: str, k: Tensor, v: Tensor, B: int, device: torch.device) -> None:
    """Keys and values as the kernels read them: ``[B, heads, slots, 128]``, float32, contiguous, on the rows' device."""
    for t in (k, v):
        if t.dim() != 4 or t.shape[0] != B or t.shape[3] != 128 or t.dtype != torch.float32 or not t.is_contiguous() or t.device != device:
            raise ValueError(f"{name} cache {tuple(t.shape)} {t.dtype} on {t.device}: contiguous float32 [{B}, heads, slots, 128] on {device} is read")
    if k.shape != v.shape:
        raise ValueError(f"{name} cache: keys {tuple(k.shape)}, values {tuple(v.shape)}")


def _rows_layer(x: Tensor, attn: Attention, norm: RMSNorm, mlp: MlpBlock, norm_mlp: RMSNorm, eps: float, positions: Callable[[], Tensor], tables,
                mode: int, n_valid: list[int] | None, k: Tensor, v: Tensor, cross: tuple | None = None, out: Tensor | None = None) -> Tensor:
    """One layer over ``x [B, T, D]`` (float32, contiguous) on our kernels, in one native call: RMSNorm in the split pass of the projections, RoPE with
    the scatter into the caches ``k``, ``v [B, heads, slots, 128]``, attention, residual adds in the epilogues, the gate in the split pass of
    the last product.  ``mode``: 0 causal, 1 pad-partitioned at ``n_valid``.  ``cross``: (attention, norm, cache, valid keys) of a cross-attention
    behind the self-attention.  The result is in ``out`` (``x`` itself, say) or a new tensor.  ``positions`` gives int32 ``[B * T]`` and is asked last: where
    they have to be made, their copy waits for the device, which then has the layer's launches to do at once."""
    from . import engine as _k
    B, T, D = x.shape
    y = torch.empty_like(x) if out is None else out
    if B * T == 0:
        return y
    if x.data_ptr() % 16:                                         # (a view of other memory)
        x = x.clone()
    ca, cn, cc, valid = cross if cross is not None else (None, None, None, None)
    _check_caches("self-attention", k, v, B, x.device)
    if k.shape[1] != attn.num_kv_heads or k.shape[2] < T:
        raise ValueError(f"self-attention cache {tuple(k.shape)} for {attn.num_kv_heads} key heads and {T} rows")
    if cc is not None:
        _check_caches("cross-attention", cc.k, cc.v, B, x.device)
        if not cc.k.shape[1] or ca.num_query_heads % cc.k.shape[1]:
            raise ValueError(f"cross-attention cache {tuple(cc.k.shape)} for {ca.num_query_heads} query heads")
    a = RowsLayer(D=D, eps=eps)
    keep = _rows_weights(a, B * T, attn, norm, mlp, norm_mlp, ca, cn, x.device)
    a.B, a.T, a.slots, a.mode, a.n_pos = B, T, k.shape[2], mode, tables[0].shape[0]
    a.x_in, a.x = x.data_ptr(), y.data_ptr()
    a.sin_table, a.cos_table, a.k_cache, a.v_cache = tables[0].data_ptr(), tables[1].data_ptr(), k.data_ptr(), v.data_ptr()
    if n_valid is not None:
        if len(n_valid) > min(B, 16):
            raise ValueError(f"{len(n_valid)} numbers of valid keys for a batch of {B} (16 at most)")
        a.n_valid[:len(n_valid)] = [int(n) for n in n_valid]      # (rows without one have none)
    if cc is not None:
        a.cross_kv_heads, a.cross_slots, a.cross_k, a.cross_v = cc.k.shape[1], cc.k.shape[2], cc.k.data_ptr(), cc.v.data_ptr()
        a.cross_valid[:B] = [int(n) for n in valid]
    pos = positions()
    if pos.numel() < B * T or pos.dtype != torch.int32 or pos.device != x.device:
        raise ValueError(f"{B * T} int32 positions are read")
    a.positions = pos.data_ptr()
    _k.rows_layer_forward(a, _k.rows_layer_work_bytes(a), x.device)
    del keep
    return y


class EncoderLayer(nn.Module):
    def __init__(self, config: DiaConfig, compute_dtype: torch.dtype):
        super().__init__()
        self.config, self.compute_dtype = config, compute_dtype
        e, eps = config.model.encoder, config.model.normalization_layer_epsilon
        self.pre_sa_norm = RMSNorm(e.n_embd, eps=eps)
        self.self_attention = Attention(config, e.n_embd, e.n_embd, e.n_head, e.n_head, e.head_dim, compute_dtype,
                                        is_cross_attn=False, out_embed_dim=e.n_embd)
        self.post_sa_norm = RMSNorm(e.n_embd, eps=eps)
        self.mlp = MlpBlock(e.n_embd, e.n_hidden, compute_dtype)

    def forward(self, x: Tensor, state: EncoderInferenceState) -> Tensor:
        if x.is_cuda and not torch.is_grad_enabled():
            from . import engine as _k
            eps = self.config.model.normalization_layer_epsilon
            B, T, _ = x.shape
            x = x.to(torch.float32).contiguous()

            def positions():
                pos = state.extras.get("pos_i32")
                if pos is None or pos.numel() != B * T:
                    pos = state.extras["pos_i32"] = _k.positions_i32(T, B, x.device)
                return pos

            kv = torch.empty((2, B, self.self_attention.num_kv_heads, T, 128), dtype=torch.float32, device=x.device)
            return _rows_layer(x, self.self_attention, self.pre_sa_norm, self.mlp, self.post_sa_norm, eps, positions,
                               _k.rope_tables_device(self.config, x.device), 1, _encoder_valid_lens(state), kv[0], kv[1])
        h = self.pre_sa_norm(x.float())
        x = x + self.self_attention(h, h, state.positions, state.positions, attn_mask=state.attn_mask)
        return x + self.mlp(self.post_sa_norm(x.float()))


class Encoder(nn.Module):
    def __init__(self, config: DiaConfig, compute_dtype: torch.dtype):
        super().__init__()
        self.config, self.compute_dtype = config, compute_dtype
        e = config.model.encoder
        self.embedding = nn.Embedding(config.model.src_vocab_size, e.n_embd)
        self.layers = nn.ModuleList([EncoderLayer(config, compute_dtype) for _ in range(e.n_layer)])
        self.norm = RMSNorm(e.n_embd, eps=config.model.normalization_layer_epsilon)

    def forward(self, x_ids: Tensor, state: EncoderInferenceState) -> Tensor:
        if x_ids.is_cuda and not torch.is_grad_enabled():
            from . import engine as _k
            B, T = x_ids.shape
            x = _k.embed_rows(self.embedding.weight, x_ids.reshape(-1).to(torch.int32).contiguous()).reshape(B, T, -1)
            if B * T and len(self.layers):
                _prepare_for_rows(self.layers, B * T, x.shape[2], x.device)
            for layer in self.layers:
                x = layer(x, state)
            return _k.rmsnorm_rows(x.reshape(B * T, -1), self.norm.weight,
                                   self.config.model.normalization_layer_epsilon).reshape(B, T, -1)
        with _exact_fp32():
            x = self.embedding(x_ids).float()
            for layer in self.layers:
                x = layer(x, state)
            return self.norm(x)


def _encoder_valid_lens(state: EncoderInferenceState) -> list[int]:
    """Valid text bytes per batch row (a prefix: pad = 0 never occurs inside utf-8 text); read back once per state."""
    lens = getattr(state, "valid_lens", None)
    if lens is None:
        pm = state.padding_mask
        lens = [int(v) for v in pm.sum(dim=-1).tolist()]
        for b, n in enumerate(lens):
            if not bool(pm[b, :n].all().item()):
                raise NotImplementedError("text with embedded pad bytes is not supported by the attention kernels")
        state.valid_lens = lens
    return lens


def _contract_dims(name: str) -> int:
    """Leading (input) axes of a decoder DenseGeneral kernel: 2 for the attention output projections
    ``[heads, head_dim, D]``, 1 for everything else."""
    return 2 if name.endswith("o_proj.weight") else 1


class DecoderLayer(nn.Module):
    def __init__(self, config: DiaConfig, compute_dtype: torch.dtype):
        super().__init__()
        self.config, self.compute_dtype = config, compute_dtype
        d, e, eps = config.model.decoder, config.model.encoder, config.model.normalization_layer_epsilon
        self.pre_sa_norm = RMSNorm(d.n_embd, eps=eps)
        self.pre_ca_norm = RMSNorm(d.n_embd, eps=eps)
        self.pre_mlp_norm = RMSNorm(d.n_embd, eps=eps)
        self.self_attention = Attention(config, d.n_embd, d.n_embd, d.gqa_query_heads, d.kv_heads, d.gqa_head_dim,
                                        compute_dtype, is_cross_attn=False, out_embed_dim=d.n_embd)
        self.cross_attention = Attention(config, d.n_embd, e.n_embd, d.cross_query_heads, d.cross_query_heads,
                                         d.cross_head_dim, compute_dtype, is_cross_attn=True, out_embed_dim=d.n_embd)
        self.mlp = MlpBlock(d.n_embd, d.n_hidden, compute_dtype)
        self._owner = None       # weakref to the Decoder, set by it
        self._index = -1

    def forward(self, x: Tensor, state: DecoderInferenceState, self_attn_cache: KVCache | None = None,
                cross_attn_cache: KVCache | None = None, prefill: bool = False) -> Tensor:
        if not prefill and x.shape[1] == 1:
            # hot path: the 8 fused stages of this layer in the persistent step kernel
            dec = self._owner() if self._owner is not None else None
            if dec is None:
                raise RuntimeError("DecoderLayer used for decoding outside a Decoder: no engine to run on")
            eng = dec._engine_for(state)
            if self_attn_cache is not state.self_attn_cache[self._index]:
                raise NotImplementedError("decode expects the layer's own cache from `state`")
            slot = self_attn_cache.current_idx
            y = eng.layer_step(self._index, x[:, 0, :], state.step_from, slot)
            self_attn_cache.current_idx = slot + 1
            return y[:, None, :].to(x.dtype)
        if x.is_cuda and not torch.is_grad_enabled():
            # prompt prefill (T > 1) on our kernels
            from . import engine as _k
            eps = self.config.model.normalization_layer_epsilon
            B, T, _ = x.shape
            tables = _k.rope_tables_device(self.config, x.device)

            def positions():
                pos = state.extras.get("prefill_pos")
                if pos is None or pos.numel() != B * T:
                    pos = state.extras["prefill_pos"] = _k.positions_i32(state.step_to - state.step_from, B, x.device, start=state.step_from)
                return pos

            if state.text_len is None:
                raise NotImplementedError("prefill needs DecoderInferenceState.text_len (valid text bytes)")
            x = x.to(torch.float32).contiguous()
            if self_attn_cache is not None:
                if not prefill:
                    raise NotImplementedError("T > 1 rows append through prefill only")
                k, v = self_attn_cache.k, self_attn_cache.v
                self_attn_cache.current_idx = T - 1                                        # KVCache.prefill (Appendix C Q2)
            else:
                k, v = torch.empty((2, B, self.self_attention.num_kv_heads, T, 128), dtype=torch.float32, device=x.device)
            if cross_attn_cache is None:
                raise NotImplementedError("cross-attention needs the precomputed K/V cache")
            return _rows_layer(x, self.self_attention, self.pre_sa_norm, self.mlp, self.pre_mlp_norm, eps, positions, tables, 0, None, k, v,
                               (self.cross_attention, self.pre_ca_norm, cross_attn_cache, [0] * (B - 1) + [state.text_len]),
                               out=x if x.data_ptr() % 16 == 0 else None)
        # CPU (state-dict tooling and the CPU test suite): the reference's own formulation
        h = self.pre_sa_norm(x.float())
        x = x + self.self_attention(h, h, state.dec_positions, state.dec_positions, attn_mask=None,
                                    cache=self_attn_cache, prefill=prefill, is_causal=prefill)
        h = self.pre_ca_norm(x.float())
        x = x + self.cross_attention(h, state.enc_out, state.dec_positions, state.enc_positions,
                                     attn_mask=state.dec_cross_attn_mask, cache=cross_attn_cache)
        return x + self.mlp(self.pre_mlp_norm(x.float()))


class Decoder(nn.Module):
    def __init__(self, config: DiaConfig, compute_dtype: torch.dtype):
        super().__init__()
        self.config, self.compute_dtype = config, compute_dtype
        d = config.model.decoder
        self.num_channels, self.num_layers = config.data.channels, d.n_layer
        self.embeddings = nn.ModuleList([nn.Embedding(config.model.tgt_vocab_size, d.n_embd)
                                         for _ in range(self.num_channels)])
        self.layers = nn.ModuleList([DecoderLayer(config, compute_dtype) for _ in range(self.num_layers)])
        self.norm = RMSNorm(d.n_embd, eps=config.model.normalization_layer_epsilon)
        self.logits_dense = DenseGeneral((d.n_embd,), (self.num_channels, config.model.tgt_vocab_size), axis=(-1,),
                                         weight_dtype=compute_dtype)
        for i, layer in enumerate(self.layers):
            layer._owner, layer._index = weakref.ref(self), i
        self._engine = None
        self._engine_sig = None
        self.compact_pruned_mlp = True      # drop exactly-dead MLP neurons from the engine's weight stream
        # drop all-zero input rows of the other kernels (K-row compaction); DIA_NO_ROW_COMPACTION=1 is the A/B switch of bench.py
        self.compact_pruned_rows = os.environ.get("DIA_NO_ROW_COMPACTION", "0") != "1"
        self.use_sparse24 = True            # stream 2:4 checkpoints compressed (mma.sp) when every kernel qualifies
        self.register_load_state_dict_post_hook(lambda m, k: m.invalidate_engine())

    # ---- engine management -------------------------------------------------------------------------
    def invalidate_engine(self) -> None:
        """Drop the repacked device copy of the weights (call after modifying parameters in place)."""
        self._engine_sig = None

    def _apply(self, fn, *a, **kw):                      # .to() / .cuda() / .float() move or retype parameters
        self._engine_sig = None
        return super()._apply(fn, *a, **kw)

    def _weights_signature(self):
        w = self.logits_dense.weight
        return (w.device, w.dtype, w.data_ptr(), sum(p._version for p in self.parameters()))

    def engine(self):
        """The bound ``DecodeEngine`` (weights repacked on first use and after any change)."""
        from .engine import DecodeEngine, decoder_tensor_names
        dev = self.logits_dense.weight.device
        if dev.type != "cuda":
            raise RuntimeError("the Dia decode path needs the model on a CUDA device (sm_100a); no CPU fallback")
        sig = self._weights_signature()
        if self._engine is not None and self._engine_sig == sig and self._engine.device == dev:
            return self._engine
        # (re)pack: a checkpoint whose MLP was structurally pruned (zero hidden neurons) gets a narrower engine
        from .pruning_utils import compact_mlp, is_2to4, plan_mlp_compaction
        from .synthetic import is_dense_kernel
        import torch.nn.utils.prune as _prune
        if any(_prune.is_pruned(m) for m in self.modules() if isinstance(m, DenseGeneral)):
            raise RuntimeError("pruning masks are still attached (parameters are named weight_orig): call "
                               "pruning_utils.make_pruning_permanent(model) before decoding")
        canonicalize_dense_kernels_(self)
        sig = self._weights_signature()
        sd = dict(self.named_parameters())
        tensors = {n: sd[n].detach() for n in decoder_tensor_names(self.config)}
        d = self.config.model.decoder
        plan = plan_mlp_compaction(tensors, d.n_layer, d.n_hidden) if self.compact_pruned_mlp else None
        width = plan[0] if plan is not None else d.n_hidden
        if plan is not None:
            tensors = compact_mlp(tensors, plan)
        # a 2:4 checkpoint (every dense kernel) streams compressed and runs on mma.sp
        sparse = bool(self.use_sparse24) and all(is_2to4(t, _contract_dims(n)) for n, t in tensors.items()
                                                 if is_dense_kernel(n))
        # `--prune-dim 0` checkpoints: all-zero INPUT rows of the other kernels are dropped as well (K-row compaction)
        from .pruning_utils import compact_rows, plan_row_compaction
        rplan = plan_row_compaction(tensors, d.n_layer) if (self.compact_pruned_rows and not sparse) else {}
        maps = {}
        if rplan:
            tensors, maps = compact_rows(tensors, rplan)
        k_rows = {fam: w for fam, (w, _) in rplan.items()}
        if self._engine is None or self._engine.device != dev or self._engine.n_hidden != width or \
                self._engine.sparse24 != sparse or self._engine.k_rows != k_rows:
            if self._engine is not None:
                self._engine.close()
            self._engine = DecodeEngine(self.config, dev, n_hidden=width, sparse24=sparse, k_rows=k_rows)
        self._engine.load_weights(tensors)
        if maps:
            self._engine.set_row_maps(maps)
        self._engine_sig = sig
        return self._engine

    def batch_engine(self, max_utterances: int = 8):
        """The ``BatchDecodeEngine`` (N utterances per launch on the tcgen05 step kernel), repacked like :meth:`engine`."""
        from .engine import BatchDecodeEngine, decoder_tensor_names
        dev = self.logits_dense.weight.device
        if dev.type != "cuda":
            raise RuntimeError("the Dia decode path needs the model on a CUDA device (sm_100a); no CPU fallback")
        sig = (self._weights_signature(), int(max_utterances))
        if getattr(self, "_bengine", None) is not None and self._bengine_sig == sig and self._bengine.device == dev:
            return self._bengine
        import torch.nn.utils.prune as _prune
        if any(_prune.is_pruned(m) for m in self.modules() if isinstance(m, DenseGeneral)):
            raise RuntimeError("pruning masks are still attached: call pruning_utils.make_pruning_permanent(model) first")
        canonicalize_dense_kernels_(self)
        sig = (self._weights_signature(), int(max_utterances))
        from .pruning_utils import compact_mlp, plan_mlp_compaction
        sd = dict(self.named_parameters())
        tensors = {n: sd[n].detach() for n in decoder_tensor_names(self.config)}
        d = self.config.model.decoder
        plan = plan_mlp_compaction(tensors, d.n_layer, d.n_hidden) if self.compact_pruned_mlp else None
        width = plan[0] if plan is not None else d.n_hidden
        if plan is not None:
            tensors = compact_mlp(tensors, plan)
        old = getattr(self, "_bengine", None)
        if old is None or old.device != dev or old.n_hidden != width or old.max_utterances != int(max_utterances):
            if old is not None:
                old.close()
            self._bengine = BatchDecodeEngine(self.config, dev, max_utterances=int(max_utterances), n_hidden=width)
        self._bengine.load_weights(tensors)
        self._bengine_sig = sig
        return self._bengine

    def _engine_for(self, state: DecoderInferenceState):
        eng = self.engine()
        if state.text_len is None:
            row = state.dec_cross_attn_mask[1].reshape(-1)
            n = int(row.sum().item())
            if bool(state.dec_cross_attn_mask[0].any().item()) or not bool(row[:n].all().item()):
                raise NotImplementedError("cross-attention mask must be (all-pad row 0, valid-prefix row 1)")
            state.text_len = n
        key = tuple(c.k.data_ptr() for c in state.self_attn_cache) + \
            tuple(c.k.data_ptr() for c in state.cross_attn_cache) + (state.text_len,)
        if eng.bound_key() != key:
            for c in state.cross_attn_cache:            # the kernels need contiguous fp32 [2,H,S,128]
                if c.k.dtype != torch.float32 or not c.k.is_contiguous():
                    c.k = c.k.to(torch.float32).contiguous()
                if c.v.dtype != torch.float32 or not c.v.is_contiguous():
                    c.v = c.v.to(torch.float32).contiguous()
            eng.bind(state.self_attn_cache, state.cross_attn_cache, state.text_len)
        return eng

    # ---- once per utterance ---------------------------------------------------------------------------
    def precompute_cross_attn_cache(self, enc_out: Tensor, enc_positions: Tensor) -> list[KVCache]:
        out: list[KVCache] = []
        if enc_out.is_cuda and not torch.is_grad_enabled():
            from . import engine as _k
            B, S, _ = enc_out.shape
            x = enc_out.to(torch.float32).contiguous()
            tables, pos = _k.rope_tables_device(self.config, x.device), _k.positions_i32(S, B, x.device)
            for layer in self.layers:
                ca = layer.cross_attention
                H = ca.num_kv_heads
                k = torch.empty((B, H, S, 128), dtype=torch.float32, device=x.device)
                v = torch.empty_like(k)
                _k.rope_rows(ca.k_proj._forward_tcgen05(x, (2,)).reshape(B * S, H * 128), pos, B, S, H, tables, cache=k)
                _k.rope_rows(ca.v_proj._forward_tcgen05(x, (2,)).reshape(B * S, H * 128), None, B, S, H, tables,
                             rotate=False, cache=v)
                out.append(KVCache.from_kv(k, v))
            return out
        with torch.no_grad(), _exact_fp32():
            x = enc_out.float()
            for layer in self.layers:
                ca = layer.cross_attention
                k = ca.rotary_emb(ca.k_proj(x), enc_positions).transpose(1, 2).contiguous()
                v = ca.v_proj(x).transpose(1, 2).contiguous()
                out.append(KVCache.from_kv(k, v))
        return out

    def precompute_cross_attn_cache_live(self, enc_live: Tensor, text_length: int) -> list[KVCache]:
        """Same caches as ``precompute_cross_attn_cache`` for the entries that are ever observed.  ``enc_live`` is
        the encoder output of the valid text bytes of the conditional row, ``[1, n, E]``.  The reference projects
        all 2 x text_length encoder positions in every layer, but the unconditional row is fully masked and so are
        the pad positions of the conditional row; here those entries are zeros and only ``n`` rows are projected."""
        out: list[KVCache] = []
        n = enc_live.shape[1]
        if enc_live.is_cuda and not torch.is_grad_enabled():
            from . import engine as _k
            x = enc_live.to(torch.float32).contiguous()
            tables, pos_i = _k.rope_tables_device(self.config, x.device), _k.positions_i32(n, 1, x.device)
            for layer in self.layers:
                ca = layer.cross_attention
                H = ca.num_kv_heads
                k = torch.zeros((2, H, text_length, 128), dtype=torch.float32, device=x.device)
                v = torch.zeros_like(k)
                _k.rope_rows(ca.k_proj._forward_tcgen05(x, (2,)).reshape(n, H * 128), pos_i, 1, n, H, tables, cache=k[1:])
                _k.rope_rows(ca.v_proj._forward_tcgen05(x, (2,)).reshape(n, H * 128), None, 1, n, H, tables,
                             rotate=False, cache=v[1:])
                out.append(KVCache.from_kv(k, v))
            return out
        pos = torch.arange(n, dtype=torch.float32, device=enc_live.device)[None, :]
        with torch.no_grad(), _exact_fp32():
            x = enc_live.float()
            for layer in self.layers:
                ca = layer.cross_attention
                k_live = ca.rotary_emb(ca.k_proj(x), pos).transpose(1, 2)           # [1, H, n, d]
                v_live = ca.v_proj(x).transpose(1, 2)
                k = torch.zeros((2, k_live.shape[1], text_length, k_live.shape[3]), dtype=k_live.dtype, device=x.device)
                v = torch.zeros_like(k)
                k[1, :, :n] = k_live[0]
                v[1, :, :n] = v_live[0]
                out.append(KVCache.from_kv(k, v))
        return out

    # ---- the hot path -------------------------------------------------------------------------------------
    def decode_step(self, tgt_ids_Bx1xC: Tensor, state: DecoderInferenceState) -> Tensor:
        B, T, C = tgt_ids_Bx1xC.shape
        assert T == 1, "decode_step expects T=1"
        assert C == self.num_channels, "Input channels mismatch"
        assert B == 2, "decode_step expects the CFG batch of 2"
        eng = self._engine_for(state)
        slot = state.self_attn_cache[0].current_idx
        logits = eng.decode_step(tgt_ids_Bx1xC.reshape(2, C), state.step_from, slot)
        for c in state.self_attn_cache:
            c.current_idx = slot + 1
        return logits[:, None, :, :]

    def forward(self, tgt_ids_BxTxC: Tensor, state: DecoderInferenceState, want_logits: bool = True) -> Tensor:
        """Prompt prefill / teacher-forced pass over T positions (dia/layers.py:722-766).  ``want_logits=False`` skips
        the logits head, whose output ``Dia._prepare_generation`` discards (dia/model.py:420-421)."""
        B, T, C = tgt_ids_BxTxC.shape
        assert C == self.num_channels, "Input channels mismatch"
        if tgt_ids_BxTxC.is_cuda and not torch.is_grad_enabled():
            # own kernels end to end: embedding gather-sum, 18 x (fused-norm GEMMs, RoPE + cache scatter, fp32 attention,
            # gate, residual epilogues), final norm fused into the logits GEMM
            x = self.engine().embed_sum(tgt_ids_BxTxC.reshape(B * T, C)).reshape(B, T, -1)
            if B * T and len(self.layers):
                _prepare_for_rows(self.layers, B * T, x.shape[2], x.device)
            state.extras.pop("prefill_pos", None)
            for i, layer in enumerate(self.layers):
                x = layer(x, state, self_attn_cache=state.self_attn_cache[i],
                          cross_attn_cache=state.cross_attn_cache[i], prefill=True)
            if not want_logits:
                return None
            return self.logits_dense._forward_tcgen05(x, (2,), norm_weight=self.norm.weight,
                                                      eps=self.config.model.normalization_layer_epsilon)
        with _exact_fp32():
            x = None
            for i, emb in enumerate(self.embeddings):
                e = emb(tgt_ids_BxTxC[..., i]).float()
                x = e if x is None else x + e
            for i, layer in enumerate(self.layers):
                x = layer(x, state, self_attn_cache=state.self_attn_cache[i],
                          cross_attn_cache=state.cross_attn_cache[i], prefill=True)
            return self.logits_dense(self.norm(x.float())).to(torch.float32)


class DiaModel(nn.Module, PyTorchModelHubMixin, repo_url="https://github.com/nari-labs/dia",
               pipeline_tag="text-to-speech", license="apache-2.0",
               coders={DiaConfig: (lambda c: c.model_dump(), lambda d: DiaConfig.model_validate(d))}):
    def __init__(self, config: DiaConfig, compute_dtype: Optional[torch.dtype] = None):
        super().__init__()
        self.config = config
        if compute_dtype is None:
            compute_dtype = {"bfloat16": torch.bfloat16, "float16": torch.float16}.get(
                getattr(config.model, "weight_dtype", "float32"), torch.float32)
            print(f"Inferred compute_dtype: {compute_dtype} from config")
        self.encoder = Encoder(config, compute_dtype)
        self.decoder = Decoder(config, compute_dtype)
