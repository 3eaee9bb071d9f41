"""Matrix products y = x W^T.

The reference's engine uses a library for every linear layer (nn.Linear, i.e.
cuBLAS: src/dli/model/llama.py:72-74,95,190,305).  Here a product goes to one of the
engine's own tcgen05 kernels where the rules below say that it beats the library:
few tokens (csrc/skinny_gemm.cu), some (few_gemm.cu), many with their elementwise step
(dense_gemm.cu), float32 (float_gemm.cu); the others stay with the library.  The
float32 path is true 32-bit: TF32 and reduced-precision accumulation are switched
off for the process when this module is imported, and checked at every call.
"""

from __future__ import annotations

import torch

from . import ops
from .attention import sm_count

torch.backends.cuda.matmul.allow_tf32 = False
torch.backends.cudnn.allow_tf32 = False
torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
torch.backends.cuda.matmul.allow_fp16_reduced_precision_reduction = False


# Up to this many tokens a layer's bfloat16 products go to the engine's decode product, which
# there beats the library on three of the four shapes and fuses the next elementwise step;
# measured on B200 at Llama-3.2-1B sizes, the library's kernels beat it from about 12 tokens on
# (steps of 9 tokens and more: few_max_tokens).
# The head's product (float32 logits straight from the accumulator) stays with it up to 64.
SKINNY_MAX_TOKENS = 8
SKINNY_MAX_TOKENS_HEAD = 64


def decode_product(x: torch.Tensor, max_tokens: int = SKINNY_MAX_TOKENS) -> bool:
    """Whether a product with these activations goes to the engine's own decode kernel."""
    return x.dtype == torch.bfloat16 and x.shape[0] <= max_tokens and ops.skinny_gemm_supported(x.shape[0], x.shape[1])


# Up to this many tokens the decode product also finishes the next elementwise step (rotary and
# cache write, SiLU * up) in its epilogue; with more tokens per CTA the separate kernels, which
# spread that work over the whole GPU, are faster.
FUSED_EPILOGUE_MAX_TOKENS = 8


def fused_epilogue(x: torch.Tensor) -> bool:
    return decode_product(x) and x.shape[0] <= FUSED_EPILOGUE_MAX_TOKENS


# From this many tokens two of a layer's bfloat16 products go to the engine's tcgen05 product for many tokens, which
# does the elementwise step behind the product in its epilogue.  Measured on B200 at Llama-3.2-1B sizes (us, this
# product against the library's product plus the kernel it saves; 512 / 2,048 / 8,192 tokens): gate|up with SiLU * up
# 39/38, 102/116, 383/427: always.  q|k|v with rotary and cache write 26/37, 39/37, 87/98: when its tiles fill their
# waves (2,048 tokens are 96 tiles on 74 pairs of SMs).  The plain product takes 1.00 of the library's time for gate|up
# at 2,048 tokens, 0.96-1.07 for o and down, which stay with the library: with the residual addition and the norm's
# sums in the epilogue they were slower than the library's product and the norm kernel (the epilogue read and wrote
# the float32 residual a row per thread), so that epilogue was taken out again.
DENSE_MIN_TOKENS = 512
DENSE_TILE = (256, 256)  # tokens x features of a tile, which a pair of SMs computes
WAVE_FILL_MIN = 0.8


def _dense_tiles(tokens: int, features: int) -> int:
    return -(-tokens // DENSE_TILE[0]) * -(-features // DENSE_TILE[1])


def _dense_candidate(x, features: int) -> bool:
    return x.dtype == torch.bfloat16 and x.shape[0] >= DENSE_MIN_TOKENS and ops.dense_gemm_supported(x.shape[1], features)


def dense_product(x, features: int, epilogue: str) -> bool:
    """Whether the product of these activations with a [features, K] weight, followed by ``epilogue`` ("swiglu", "act": a
    plain feed-forward's activation, or "rotary"), goes to the engine's product for many tokens."""
    if not _dense_candidate(x, features):
        return False
    tiles, pairs = _dense_tiles(x.shape[0], features), max(1, sm_count() // 2)
    if epilogue in ("swiglu", "act"):  # the activation of a feed-forward rides for nothing under the next tile's products
        return True
    if epilogue == "rotary":
        return tiles <= pairs or tiles / (-(-tiles // pairs) * pairs) >= WAVE_FILL_MIN
    raise ValueError(f"unknown epilogue {epilogue!r}")


# Steps of more tokens than the decode product takes go to the engine's product for some tokens (csrc/few_gemm.cu) where it beats the library.  Measured with cold weights
# between a norm and an activation (us, library / own), and in chains of whole layers (norm, layer, norm, ..: own minus library, a layer).
# As a rule up to 24 tokens: at 9 and 24 of them 2,048 features of K 2,048 9.3/7.4 and 9.6/8.1, 10,304 of 2,048 14.3/12.3 and 14.5/12.8, 4,096 of 1,024 8.5/7.3 and
# 8.7/7.7; layers of 2,048 with 16 tokens: the products in front -2.1 (grouped-query), -0.7 (latent), -1.2 (Mamba-2), behind -2.0, -1.7, -1.9.
#   * Long sums with few features, up to 64: at 33 and 64 tokens 2,048 of 8,192 15.4/12.4 and 15.7/12.2, 1,024 of 4,096 10.3/6.7 and 10.3/7.9.  4,096 of 4,096 only up to 40:
#     the product behind a layer of 4,096, at 32 / 48 / 64 tokens: grouped-query -3.0 / -1.9 / -0.2, differential -2.0 / -0.7 / -0.3, latent -0.6 / -0.3 / +1.9,
#     matrix memory 0.0 / +1.7 / +2.0.
#   * Where two CTAs share K (few_splits) they stay behind: 6,176 of 2,048 in front of a gated delta rule -0.4 / +1.1 / +1.9 at 12 / 16 / 20 tokens, 8,192 of 2,048 of a
#     matrix memory +0.4 at 12; of 4,096, 6,144 to 8,480 features: -0.3 to -2.6 at 16 tokens, -0.3 to +1.0 at 20 and 24.
#   * Small products up to 16: 1,024 of 1,024 behind a gated delta rule 0.0 / +0.7 / +0.7 at 16 / 20 / 24 tokens.
#   * A CTA has an SM, so a tile more than SMs is a second wave: 18,944 features (148 tiles) of 2,048 19.7/18.7, 19,072 19.7/23.7, 24,576 24.0/25.4, 28,672 (three quarters of
#     two waves) 27.2/26.4, of 1,024 16.9/17.5.
# gate|up with SiLU * up up to 96: 16,384 of 2,048 at 9 / 64 / 96 tokens 16.4/13.1, 16.7/15.4, 18.2/16.6; but 11,264 of 8,192 (88 CTAs, each all of K) at 96 42.0/44.3, and
# in a second wave 28,672 of 4,096 at 9 / 64 / 96 44.2/41.3, 48.0/48.2, 54.6/55.9, of 1,024 at 64 18.7/19.9, 57,344 of 4,096 at 24 / 48 86.5/84.6, 87.4/91.5.
FEW_MAX_TOKENS, FEW_MAX_TOKENS_SWIGLU, FEW_MAX_TOKENS_SHORT_K = 64, 96, 24
FEW_MIN_SIZE, FEW_LONG_K, FEW_MAX_FEATURES = 1024, 4096, 4224  # least K and features; from which K on, and up to which width, more than 24 tokens go there
FEW_WAVE_FILL = 0.75


def few_splits(features: int, K: int) -> int:
    """CTAs that share a tile's K: the most for which clusters of them still fit the GPU at once (of a B200's 148 SMs, clusters of four fill 132, of eight 112)
    and each has four steps of 128."""
    tiles, steps = -(-features // 128), -(-K // 128)
    return next((s for s, places in ((8, 112), (4, 132), (2, 148)) if tiles * s <= places and steps >= 4 * s), 1)


def few_max_tokens(features: int, K: int, swiglu: bool = False) -> int:
    """The most tokens whose product with a [features, K] weight goes to the engine's product for some tokens (0: none)."""
    tiles, sms, splits = -(-features // 128), sm_count(), few_splits(features, K)
    waves = -(-tiles // sms)
    if waves > 1:
        if tiles < FEW_WAVE_FILL * waves * sms or (K < 2048 and not swiglu):
            return 0
        return FEW_MAX_TOKENS if swiglu and waves == 2 and K >= 2048 else FEW_MAX_TOKENS_SHORT_K
    if swiglu:
        return FEW_MAX_TOKENS_SWIGLU if splits > 1 or K < 4096 or tiles >= FEW_WAVE_FILL * sms else FEW_MAX_TOKENS
    if K >= FEW_LONG_K and features <= FEW_MAX_FEATURES:
        return FEW_MAX_TOKENS if features <= 3200 or K >= 8192 else 40
    if K < 2048 and features <= 3200:
        return 16
    if splits == 2 and 2048 <= K < 8192:
        return 16 if K >= 3072 or features <= 5400 else 12 if features <= 7168 else 0
    return FEW_MAX_TOKENS_SHORT_K


def few_product(x: torch.Tensor, weight: torch.Tensor, swiglu: bool = False) -> bool:
    """Whether the product of these activations with a [features, K] weight goes to the engine's product for some tokens."""
    if not SKINNY_MAX_TOKENS < x.shape[0] <= FEW_MAX_TOKENS_SWIGLU or not ops.few_gemm_supported(x, weight) or min(weight.shape) < FEW_MIN_SIZE or (swiglu and weight.shape[0] % 128):
        return False
    return x.shape[0] <= few_max_tokens(*weight.shape, swiglu)


def project(x, weight: torch.Tensor, out_dtype: torch.dtype | None = None, max_tokens: int = SKINNY_MAX_TOKENS) -> torch.Tensor:
    """y = x W^T for a step's tokens, in x's dtype or in ``out_dtype`` (float32 for logits).  x may be
    ops.ScaledRows (rows that still lack their norm's factor): those only exist for token counts that
    the decode kernel serves, which applies the factor."""
    # TMA reads the decode product's activations: rows back to back from a 16-byte boundary (a column slice of wider rows is
    # neither, and a slice of a single row, though "contiguous", may start off the boundary): those stay with the library
    if isinstance(x, ops.ScaledRows) or (decode_product(x, max_tokens) and x.is_contiguous() and x.data_ptr() % 16 == 0):
        return ops.skinny_gemm(x, weight, out_dtype or x.dtype)
    if out_dtype == torch.float32 and x.dtype != torch.float32:
        return logits_product(x, weight)
    y = linear(x, weight)
    return y if out_dtype in (None, y.dtype) else y.to(out_dtype)


def project_bias(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None) -> torch.Tensor:
    """y = x W^T + b: the bias joins the float32 sums before the one rounding (the library's product with its bias
    epilogue, at every token count); without a bias it is ``project``."""
    if bias is None:
        return project(x, weight)
    return linear_bias(x, weight, bias)


def linear_bias(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    _need_device(x, "linear_bias")
    if torch.backends.cuda.matmul.allow_tf32:
        raise RuntimeError("linear_bias: TF32 was switched on; the float32 path must stay true 32-bit")
    return torch.addmm(bias, x, weight.t())


def last_product(x: torch.Tensor, weight: torch.Tensor, defer: bool):
    """The product that ends a mixer or feed-forward: x W^T, or — if the part's owner allowed it and
    the decode kernel with its fused epilogues will serve these tokens — the product left
    uncomputed for the norm behind it (parts.base.PendingProduct)."""
    if defer and fused_epilogue(x):
        from ..parts.base import PendingProduct

        return PendingProduct(x, weight)
    return project(x, weight)


# From this many tokens and this inner size on a float32 product goes to the engine's own kernel on the tensor cores (csrc/float_gemm.cu: three
# bfloat16 terms a number, true float32 results).  Library / own, us: 2,048 x 2,048, 1 / 4 / 8 / 100 / 512 tokens 12/21, 32/23, 32/22, 57/27, 94/45; 8,192 x 2,048
# 23/35, 37/35, 57/35, 94/49, 315/137; K 192, 8 / 512 tokens 12/12, 18/14; K 64 8/10 up to 200 tokens.  From 17 tokens on every size of K 256 and more gains, 4 to 128,256 features
# (64 features of K 2,048 at 24 tokens 33/12, of K 256 6.8/6.0; a few of K 256 lose up to 0.8 of 7).  Up to 16 the library has kernels of its own for small products: 512
# features of K 256 3.6/5.9, of K 384 4.5/7.3, of K 512 8.2/7.0; 320 of K 768 6.6/7.3, 384 8.8/7.1; and for few features with long sums, which the own one puts on one cluster a tile: 64 of K
# 4,096 12.8/12.3, of 8,192 13.4/19.5, 256 of 8,192 19.4/25.8 (but 32 of 4,096 39/12); at 8 also for the widest, 32,768 of 4,096 167/174, 16,384 of 8,192 201/172.
FLOAT_MIN_TOKENS, FLOAT_MIN_K = 8, 256
FLOAT_FEW_TOKENS, FLOAT_FEW_MIN_SIZE = 16, 1 << 18  # (size: numbers of a weight)


def float_product(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether x [.., n, in] times weight [.., out, in] transposed goes to the engine's float32 product."""
    if not (x.dtype == torch.float32 and x.is_cuda and x.dim() in (2, 3) and x.shape[-2] >= FLOAT_MIN_TOKENS and x.shape[-1] >= FLOAT_MIN_K
            and ops.float_gemm_supported(x, weight)):
        return False
    return x.shape[-2] > FLOAT_FEW_TOKENS or _float_few(x.shape[-2], weight.numel() // x.shape[-1], x.shape[-1])


def _float_few(tokens: int, features: int, K: int) -> bool:
    """Whether a float32 product of FLOAT_MIN_TOKENS to FLOAT_FEW_TOKENS tokens goes there."""
    if K < 1024:
        return features * K >= FLOAT_FEW_MIN_SIZE
    if K <= 2048:
        return True
    return features <= 24576 or tokens >= 12 if features > 256 else features <= 32 and K <= 6144


def linear(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """x [n, in] times weight [out, in] transposed; float32 accumulation in both dtypes."""
    if not x.is_cuda:
        raise RuntimeError("linear: the engine has no CPU path")
    if torch.backends.cuda.matmul.allow_tf32:
        raise RuntimeError("linear: TF32 was switched on; the float32 path must stay true 32-bit")
    if out is None:  # (a step that is launched kernel by kernel waits for the host: what most products need not ask is asked first)
        if x.dtype == torch.float32:
            if float_product(x, weight):
                return ops.float_gemm(x, weight)
        elif x.shape[0] <= FEW_MAX_TOKENS_SWIGLU and few_product(x, weight):
            return ops.few_gemm(x, weight, few_splits(*weight.shape))
    return torch.matmul(x, weight.t(), out=out)


def _need_device(x: torch.Tensor, what: str) -> None:
    if not x.is_cuda:
        raise RuntimeError(f"{what}: the engine has no CPU path")


HEADS_MATVEC_MAX_TOKENS = 8  # up to this many tokens a gated per-head product goes to the engine's own small kernel


def heads_product(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, gate: torch.Tensor | None = None) -> torch.Tensor:
    """out[t, a, :] = x[t, a, :] @ weight[a]: one product per head a (x [n, heads, in] and out [n, heads, features]
    may be column slices of wider rows; weight [heads, in, features] contiguous), float32 accumulation; with ``gate``
    [n, heads * features] the result is multiplied by sigmoid(gate).  The library's strided-batched product, and the
    gate kernel behind it; for a decode step's few tokens a gated product is one kernel of the engine instead (measured
    in replayed graphs at 8 tokens, 16 heads, 192 x 128: 4.6 us against 2.4 + 5.0; without a gate the library's 2.5 us
    stand)."""
    _need_device(x, "heads_product")
    if torch.backends.cuda.matmul.allow_tf32:
        raise RuntimeError("heads_product: TF32 was switched on; the float32 path must stay true 32-bit")
    n, heads, features = out.shape
    if gate is not None and n <= HEADS_MATVEC_MAX_TOKENS and ops.heads_matvec_supported(x.shape[2], features):
        ops.heads_matvec(out, x, weight, gate)
        return out
    torch.bmm(x.transpose(0, 1), weight, out=out.transpose(0, 1))
    if gate is not None:
        ops.sigmoid_gate(out.view(n, heads * features), gate)
    return out


def batched_project(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """out[b] = x[b] @ weight[b] for x [batch, n, in] and weight [batch, in, features] (several products of one shape whose
    inputs differ, in one call of the library's batched product); float32 accumulation."""
    _need_device(x, "batched_project")
    if torch.backends.cuda.matmul.allow_tf32:
        raise RuntimeError("batched_project: TF32 was switched on; the float32 path must stay true 32-bit")
    if float_product(x, weight.transpose(1, 2)):
        return ops.float_gemm(x, weight.transpose(1, 2))
    return torch.bmm(x, weight)


def logits_product(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """x [n, in] (bfloat16 or float32) times weight [out, in] transposed, the float32 sums returned as they are."""
    _need_device(x, "logits_product")
    if x.dtype == torch.float32:
        return linear(x, weight)
    return torch.mm(x, weight.t(), out_dtype=torch.float32)
