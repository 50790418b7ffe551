"""The contractions of the decoder, out = x @ W^T, each with its epilogue fused.

Which kernel runs is decided here, by dtype and shape:
  float32   the kernels of `gemm_f32` (FFMA for a few tokens; beyond, three bfloat16 parts per operand on the
            tensor cores, which together are the operand: sums as close to 64 bits as the FFMA kernel's) when rows are
            whole 16-byte pieces and sums not short (`_in_parts`), else the FFMA kernel (`gemm_simt`);
  bfloat16  the tcgen05 kernel (`gemm_tcgen05`) when the shape meets its alignment rule,
            else the FFMA kernel on bf16 operands.  Either way accumulation is float32.
"""
from __future__ import annotations

import torch

from . import ops, tcgen05
from .attention import _sm_count


class Weight:
    """A weight matrix [out, in] (row-major over `in`, as quant.rs:45-50 holds it) plus
    whatever a kernel wants to keep beside it (tensor-map handles)."""

    __slots__ = ("t", "n", "k", "tc")

    def __init__(self, t: torch.Tensor):
        self.t = t.contiguous()
        self.n, self.k = self.t.shape
        self.tc = None


def _use_tensor_cores(x: torch.Tensor, w: Weight) -> bool:
    if x.dtype != torch.bfloat16:
        return False
    return tcgen05.supports(x, w)


# Sums of fewer than 128 terms are left to the FFMA kernel, and up to 256 products of more than 32 rows whose tiles of 64 x 64 it
# does in one round: it has them sooner, because a block of the tensor cores' kernel is 64 steps of K long and costs 4.5 to 9 us to
# start.  (us, FFMA / tensor cores.  N = 512: 17 rows of K = 96 5.9 / 6.4, of 128 7.3 / 6.4; 64 rows of 128 7.6 / 8.4, of 160 9.2 / 10.3,
# of 256 13.8 / 7.3, which is the first to be cut over a cluster; 333 rows of 128 7.7 / 11.8, of 192 10.7 / 13.7, of 256 13.8 / 9.9.
# Two rounds, N = 4,096: 333 rows of 128 16.3 / 12.5.)
F32_PARTS_MIN_K, F32_PARTS_ALWAYS_K = 128, 256


def _in_parts(m: int, n: int, k: int) -> bool:
    if k < F32_PARTS_MIN_K or k >= F32_PARTS_ALWAYS_K:
        return k >= F32_PARTS_MIN_K
    return m <= 32 or -(-m // 64) * -(-n // 64) > _sm_count()


def _plain(x, w: Weight, out, mode, w2: Weight | None = None, ctx=None, **constants):
    """The product without bfloat16 tensor cores."""
    t2 = w2.t if w2 is not None else None
    m = x.shape[0]
    if not (ops.gemm_f32_supports(x, w.t, t2) and (m <= 16 or _in_parts(m, w.n, w.k))):
        return ops.gemm_simt(x, w.t, out, mode, w2=t2, **constants)
    if ctx is not None and ops.gemm_f32_takes_wide(m, w.n, w.k):
        constants["parts"] = ctx.buffer("f32_parts", ops.gemm_f32_wide_scratch(m, w.k), torch.bfloat16)
    return ops.gemm_f32(x, w.t, out, mode, w2=t2, **constants)


on_tensor_cores = _use_tensor_cores      # for callers that choose their path by it


def project(x, w: Weight, out, ctx, bias=None):
    """out<run dtype> = x W^T + bias."""
    if _use_tensor_cores(x, w):
        return tcgen05.gemm(x, w, out, ops.EPI_STORE, ctx, bias=bias)
    return _plain(x, w, out, ops.EPI_STORE, ctx=ctx, bias=bias)


def logits(x, w: Weight, out, ctx, silu_cols=None):
    """out<float32> = x W^T; with silu_cols (float32 [1] on the device) the first so many columns through silu."""
    if silu_cols is not None:
        if _use_tensor_cores(x, w):
            return tcgen05.gemm(x, w, out, ops.EPI_SILU_F32, ctx, silu_cols=silu_cols)
        return _plain(x, w, out, ops.EPI_SILU_F32, ctx=ctx, silu_cols=silu_cols)
    if _use_tensor_cores(x, w):
        return tcgen05.gemm(x, w, out, ops.EPI_STORE_F32, ctx)
    return _plain(x, w, out, ops.EPI_STORE_F32, ctx=ctx)


def into_residual(x, w: Weight, residual, ctx):
    """residual<float32> += x W^T."""
    if _use_tensor_cores(x, w):
        return tcgen05.gemm(x, w, residual, ops.EPI_RESIDUAL, ctx)
    return _plain(x, w, residual, ops.EPI_RESIDUAL, ctx=ctx)


def gated(x, w_gate: Weight, w_up: Weight, out, ctx, form=None):
    """out<run dtype> = silu(x Wg^T) * (x Wu^T); with `form` (`ops.gate_form`: float32 [5] on the device: alpha,
    limit, shift, cubic, mult) out = mult g' sigmoid(alpha g' (1 + cubic g'^2)) (u' + shift), g' = min(x Wg^T, limit),
    u' = clamp(x Wu^T, -limit, limit)."""
    if _use_tensor_cores(x, w_gate):
        return tcgen05.gemm(x, w_gate, out, ops.EPI_SILU_MUL, ctx, w2=w_up, gate_form=form)
    return _plain(x, w_gate, out, ops.EPI_SILU_MUL, w_up, ctx=ctx, gate_form=form)


def activated(x, w: Weight, out, ctx, form):
    """out<run dtype> = act(x W^T), an activation with its four constants `form` (float32 on the device: `ops.xielu`'s
    two learned numbers through `ops.whole_act_form`, or `ops.RELU_SQUARED_FORM`), applied to the float32 accumulators in the product's epilogue."""
    if _use_tensor_cores(x, w):
        return tcgen05.gemm(x, w, out, ops.EPI_ACT, ctx, act_form=form)
    return _plain(x, w, out, ops.EPI_ACT, ctx=ctx, act_form=form)


def accumulate_split(x, w: Weight, acc, ctx) -> bool:
    """acc<float32> += x W^T with K split over enough CTAs to fill the GPU, if the tensor-core
    kernel takes the shape (returns False otherwise and does nothing).  For small steps whose
    output has too few tiles to keep every SM streaming weights."""
    if not _use_tensor_cores(x, w):
        return False
    tcgen05.gemm(x, w, acc, ops.EPI_RESIDUAL, ctx)
    return True


# Up to this many tokens a projection that has to leave its result in the run dtype is worth cutting
# over K into float32 accumulators (measured on a 3584-wide model: a whole 256-token step 1.4% faster,
# a 512-token step 2% slower)
SPLIT_MAX_TOKENS = 256


def wants_split(x, w: Weight) -> bool:
    """True for a small step whose projection would otherwise leave most SMs idle."""
    if not _use_tensor_cores(x, w) or x.shape[0] > SPLIT_MAX_TOKENS:
        return False
    return tcgen05.pick_split(x.shape[0], w.n, w.k) > 1
