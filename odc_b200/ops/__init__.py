"""Differentiable ops of the decoder.

On CUDA every op runs this package's own sm_100a kernels through the native extension (and
raises if the extension is missing); on CPU the plain PyTorch statements in
:mod:`odc_b200.ops.reference` run instead, which is what the CPU/gloo tests use.

``ODC_GEMM=cublas`` and ``ODC_ATTN=flash`` switch the two largest kernels to library calls; they
exist to measure the hand-written kernels against the libraries, not as a fallback.
"""
from __future__ import annotations

import math
import os
from typing import Optional

import torch

from . import reference as ref

_C = None   # the native extension, loaded by the first op on a CUDA tensor


def _ext():
    global _C
    if _C is None:
        from .. import _ext as loader
        _C = loader.load()
    return _C


def kernel_launches() -> int:
    """Number of this package's kernels launched by the ops so far (for benchmark accounting)."""
    return _C.kernel_launches() if _C is not None else 0


def _count(n: int = 1):
    _ext().count_launches(n)


def check_status() -> None:
    """Raise if a kernel of this package gave up on a bounded wait since the last check (one small D2H copy + sync).

    The FSDP integrations and the reduction service read the same per-device word at every once-per-minibatch
    synchronisation; code that uses the ops on their own calls this where it would otherwise trust the results.
    """
    from ..runtime.status import check_status_word
    word = _ext().kernel_status()
    host = word.cpu()
    if int(host[0]) != 0:
        _ext().clear_kernel_status()
        check_status_word(int(host[0]), int(host[1]), int(host[2]))


def gemm_backend() -> str:
    return os.environ.get("ODC_GEMM", "tcgen05")


def attn_backend() -> str:
    return os.environ.get("ODC_ATTN", "native")


# ------------------------------------------------------------------------------------------
# GEMM.  layouts (all operands row-major):
#   "nt": C[M,N] = A[M,K] @ B[N,K]^T      (forward  y = x W^T)
#   "nn": C[M,N] = A[M,K] @ B[K,N]        (dgrad    dx = dy W)
#   "tn": C[M,N] = A[K,M]^T @ B[K,N]      (wgrad    dW = dy^T x)
# ------------------------------------------------------------------------------------------
def gemm(a: torch.Tensor, b: torch.Tensor, layout: str = "nt", out: Optional[torch.Tensor] = None,
         bias: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None,
         accumulate: bool = False, residual: Optional[torch.Tensor] = None) -> torch.Tensor:
    if layout == "nt":
        M, N = a.shape[0], b.shape[0]
    elif layout == "nn":
        M, N = a.shape[0], b.shape[1]
    elif layout == "tn":
        M, N = a.shape[1], b.shape[1]
    else:
        raise ValueError(layout)
    if out is None:
        out = torch.empty(M, N, dtype=out_dtype or a.dtype, device=a.device)
        assert not accumulate
    if not a.is_cuda or gemm_backend() == "cublas":
        A = a.t() if layout == "tn" else a
        B = b.t() if layout == "nt" else b
        r = (A.float() @ B.float()) if not a.is_cuda else (A @ B)
        if bias is not None:
            r = r + bias
        if residual is not None:
            r = r + residual
        if accumulate:
            out += r.to(out.dtype)
        else:
            out.copy_(r)
        return out
    _ext().gemm(a, b, out, layout, bias, accumulate, residual)
    _count()
    return out


def linear(x, w, bias=None, residual=None):
    """``x @ w.T (+ bias) (+ residual)``; on CUDA bias and residual are fused into the GEMM epilogue."""
    if not x.is_cuda:
        y = ref.linear(x, w, bias)
        return y if residual is None else y + residual
    return _ext().linear(x, w, bias, residual)


# ------------------------------------------------------------------------------------------
def rms_norm(x, weight, eps: float = 1e-6):
    if not x.is_cuda:
        return ref.rms_norm(x, weight, eps)
    return _ext().rms_norm(x, weight, eps)


def rms_norm_residual(x, weight, eps: float = 1e-6):
    """``(rms_norm(x, weight), x)`` for pre-norm blocks: feed the second value to the block's residual add.

    The second output's gradient and the normalised branch's gradient meet again in backward, where ONE kernel forms
    ``d rms_norm + d residual`` (autograd would otherwise add the two with a separate pass over the activation)."""
    if not x.is_cuda:
        return ref.rms_norm(x, weight, eps), x
    return _ext().rms_norm_residual(x, weight, eps)


# ------------------------------------------------------------------------------------------
def rope_qkv(qkv, position_ids, n_q: int, n_kv: int, head_dim: int, theta: float,
             inv_freq: Optional[torch.Tensor] = None):
    """Rotate the q and k parts of a fused qkv activation; v passes through.

    ``inv_freq`` (rescaled rotary frequencies, ``ops.reference.rope_inv_freq``) selects the PyTorch statements on
    any device: the kernel derives its frequencies from ``theta`` alone.
    """
    if not qkv.is_cuda or inv_freq is not None:
        T = qkv.shape[0]
        q, k, v = qkv.split([n_q * head_dim, n_kv * head_dim, n_kv * head_dim], dim=-1)
        q = ref.rope(q.reshape(T, n_q, head_dim), position_ids, theta, inv_freq=inv_freq).reshape(T, -1)
        k = ref.rope(k.reshape(T, n_kv, head_dim), position_ids, theta, inv_freq=inv_freq).reshape(T, -1)
        return torch.cat([q, k, v], dim=-1)
    return _ext().rope(qkv, position_ids, n_q, n_kv, head_dim, theta)


# ------------------------------------------------------------------------------------------
def swiglu(gate_up):
    if not gate_up.is_cuda:
        return ref.swiglu(gate_up)
    return _ext().swiglu(gate_up)


def linear_swiglu(x, w):
    """``swiglu(linear(x, w))`` for ``w = [gate; up]``; on CUDA the activation is formed in the GEMM epilogue."""
    if not x.is_cuda:
        return ref.swiglu(ref.linear(x, w, None))
    return _ext().linear_swiglu(x, w)


def mlp(x, w_gate_up, w_down, residual=None):
    """``linear(linear_swiglu(x, w_gate_up), w_down, residual=residual)`` as one function: on CUDA the gradient of the
    projection is formed in the epilogue of the product with ``w_down``."""
    if not x.is_cuda:
        return linear(linear_swiglu(x, w_gate_up), w_down, residual=residual)
    return _ext().mlp(x, w_gate_up, w_down, residual)


def decoder_layer(x, position_ids, cu_seqlens, max_seqlen: int, n_q: int, n_kv: int, head_dim: int, theta: float, attn_eps: float,
                  mlp_eps: float, attn_norm, wqkv, bqkv, wo, mlp_norm, w_gate_up, w_down):
    """A pre-norm decoder layer (RMSNorm, rotary causal attention, RMSNorm, SwiGLU) on a CUDA tensor as one function; None where
    its weights are not plain bf16 matrices that all want a gradient, or none of them: then it has to be put together from
    the ops above."""
    return _ext().decoder_layer(x, position_ids, cu_seqlens, max_seqlen, n_q, n_kv, head_dim, theta, attn_eps, mlp_eps, attn_norm,
                                wqkv, bqkv, wo, mlp_norm, w_gate_up, w_down)


# ------------------------------------------------------------------------------------------
def varlen_attention_qkv(qkv, n_q: int, n_kv: int, head_dim: int, cu_seqlens, max_seqlen: int, causal: bool = True,
                         scale: Optional[float] = None):
    """Causal attention on a fused qkv activation ``[T, (Hq+2Hkv)*D]``; returns ``[T, Hq, D]``."""
    scale = scale if scale is not None else 1.0 / math.sqrt(head_dim)
    if qkv.is_cuda and attn_backend() == "native":
        return _ext().attention_qkv(qkv, n_q, n_kv, head_dim, cu_seqlens, max_seqlen, causal, scale)
    T, nq, nk = qkv.shape[0], n_q * head_dim, n_kv * head_dim
    q = qkv[:, :nq].view(T, n_q, head_dim)
    k = qkv[:, nq:nq + nk].view(T, n_kv, head_dim)
    v = qkv[:, nq + nk:].view(T, n_kv, head_dim)
    return varlen_attention(q, k, v, cu_seqlens, max_seqlen, causal, scale)


def varlen_attention(q, k, v, cu_seqlens, max_seqlen: int, causal: bool = True, scale: Optional[float] = None):
    """Causal attention over packed sequences; q ``[T,Hq,D]``, k/v ``[T,Hkv,D]`` (strided views allowed)."""
    scale = scale if scale is not None else 1.0 / math.sqrt(q.shape[-1])
    if not q.is_cuda:
        return ref.varlen_attention(q, k, v, cu_seqlens, causal, scale)
    if attn_backend() == "flash":
        from flash_attn import flash_attn_varlen_func
        return flash_attn_varlen_func(q, k, v, cu_seqlens, cu_seqlens, max_seqlen, max_seqlen,
                                      softmax_scale=scale, causal=causal)
    return _ext().attention(q, k, v, cu_seqlens, max_seqlen, causal, scale)


# ------------------------------------------------------------------------------------------
def linear_cross_entropy(h, w, labels, loss_scale=None, ignore_index: int = -100, chunk: int = 4096):
    """Summed (optionally per-token weighted) cross-entropy of ``h @ w.T`` against ``labels``.

    On CUDA the loss and both gradients are formed in one pass over token chunks; ``[T, vocab]`` logits never exist."""
    if not h.is_cuda:
        return ref.linear_cross_entropy(h, w, labels, loss_scale, ignore_index, chunk)
    return _ext().linear_cross_entropy(h, w, labels, loss_scale, ignore_index, chunk)


def linear_token_logprobs(h, w, ids, temperature: float = 1.0, ignore_index: int = -100, chunk: int = 4096):
    """``log_softmax(h @ w.T / temperature)[t, ids[t]]`` as fp32, for ``h`` of shape ``[T, H]`` or ``[B, S, H]``.

    Positions whose id equals ``ignore_index`` give 0 and no gradient.
    """
    shape = ids.shape
    h2 = h.reshape(-1, h.shape[-1])
    flat = ids.reshape(-1).to(torch.int64)
    if not h.is_cuda:
        return ref.linear_token_logprobs(h2, w, flat, temperature, ignore_index, chunk).view(shape)
    if temperature == 0 and flat.numel():
        raise ZeroDivisionError("temperature of zero")
    return _ext().linear_token_logprobs(h2, w, flat, float(temperature), ignore_index, chunk).view(shape)


class LinearTokenLogProbs(torch.nn.Module):
    """Module form: ``forward(hidden_states, vocab_weights, input_ids, temperature) -> (log_probs, None)``.

    The second value is the place of the entropy the reference's module leaves unset as well
    (examples/llm_training/lm_head.py:193-214).
    """

    def __init__(self, chunk_size: int = 4096):
        super().__init__()
        self.chunk_size = chunk_size

    def forward(self, hidden_states, vocab_weights, input_ids, temperature: float = 1.0):
        return linear_token_logprobs(hidden_states, vocab_weights, input_ids, temperature, chunk=self.chunk_size), None


# ------------------------------------------------------------------------------------------
def fused_adamw_(p32, g, m, v, p_lowp, lr, beta1, beta2, eps, weight_decay, step, grad_scale=1.0):
    """One AdamW step on a flat fp32 shard; also refreshes the low-precision copy that peers gather."""
    if not p32.is_cuda:
        ref.adamw_step(p32, g, m, v, lr, beta1, beta2, eps, weight_decay, step, grad_scale)
        if p_lowp is not None:
            p_lowp.copy_(p32)
        return
    _ext().adamw_step(p32, g, m, v, p_lowp, lr, beta1, beta2, eps, weight_decay, step, grad_scale)
    _count()
