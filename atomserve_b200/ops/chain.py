"""The projections between one layer's attention and the next one's, for few tokens, as one kernel (csrc/decode_chain.cu)."""

from __future__ import annotations

import ctypes
import functools
import os

import torch

from atomserve_b200.ops.library import KernelLibraryError, check, lib, ptr, require_cuda, stream
from atomserve_b200.ops.linear import gemm_status, own_kernels

# ATOMSERVE_B200_CHAIN=0: every product and norm as a kernel of its own (for comparison)
CHAIN = os.environ.get("ATOMSERVE_B200_CHAIN", "1") != "0"


@functools.lru_cache(maxsize=1)
def chain_limits() -> tuple[int, int]:
    """(most tokens, the multiple that every product's K has to be)."""
    tokens, k_multiple = ctypes.c_int(), ctypes.c_int()
    lib().asb_decode_chain_limits(ctypes.byref(tokens), ctypes.byref(k_multiple))
    return tokens.value, k_multiple.value


def decode_chain_takes(x: torch.Tensor, *weights: torch.Tensor) -> bool:
    """Whether `decode_chain` runs for this residual stream and these weights: matrices (the output, gated and down projections,
    and any that follow) and norms' gains, or for the stream with some weights. Its loads are of 16 bytes; what is laid out
    otherwise, the separate kernels take."""
    if not CHAIN or not own_kernels() or x.dtype != torch.bfloat16 or not x.is_cuda:
        return False
    tokens, k_multiple = chain_limits()
    if not 0 < x.shape[0] <= tokens or not x.is_contiguous() or x.data_ptr() % 16:
        return False
    for w in weights:
        size = w.shape
        if len(size) == 2:
            fits = w.dtype == torch.bfloat16 and size[0] % 2 == 0 and size[1] % k_multiple == 0
        else:
            fits = len(size) == 1 and w.dtype == torch.float32
        if not fits or not w.is_contiguous() or w.data_ptr() % 16:
            return False
    return True


def decode_chain(
    attn: torch.Tensor,
    o_proj: torch.Tensor,
    x: torch.Tensor,
    gain: torch.Tensor,
    eps: float,
    gate_up: torch.Tensor,
    down: torch.Tensor,
    arrived: torch.Tensor,
    next_gain: torch.Tensor | None = None,
    next_eps: float = 0.0,
    next_proj: torch.Tensor | None = None,
) -> tuple[torch.Tensor, torch.Tensor | None]:
    """(x2, N'(x2) . next_proj^T) with x1 = attn . o_proj^T + x and x2 = (silu(g) * u) . down^T + x1, g and u the two
    halves of N(x1) . gate_up^T, whose rows alternate gate_i, up_i (`interleave_gate_up`); the second is None without
    next_proj. All bfloat16, each stored value (x1, the gated values, x2, the last product) rounded once, sums, norms and the
    activation in float32 (a norm's input times its gain is rounded as the product's operand, its factor multiplies the sums).

    `arrived`: four int32 zeros on the device that belong to this call (the kernel's blocks count themselves in there).
    The matrices are read before the stream's previous kernel has completed: they must not be what it writes."""
    require_cuda(attn, o_proj, x, gain, gate_up, down, arrived, next_gain, next_proj)
    T, hidden = x.shape
    if next_proj is not None and (next_proj.shape[1] != hidden or next_gain is None):
        raise KernelLibraryError("decode_chain: the last product reads the normed stream")
    if not decode_chain_takes(x, o_proj, gate_up, down, gain, *([next_proj, next_gain] if next_proj is not None else [])):
        raise KernelLibraryError("decode_chain: tokens, types or sizes that the kernel does not take")
    ff = down.shape[1]
    if attn.shape != (T, o_proj.shape[1]) or o_proj.shape[0] != hidden or gate_up.shape != (2 * ff, hidden) or down.shape[0] != hidden:
        raise KernelLibraryError("decode_chain: the matrices' sizes do not follow from one another")
    if attn.dtype != x.dtype or not attn.is_contiguous() or not x.is_contiguous():
        raise KernelLibraryError("decode_chain: attn and x must be contiguous bfloat16")
    for g in (gain, next_gain):
        if g is not None and (g.dtype != torch.float32 or g.shape != (hidden,) or not g.is_contiguous()):
            raise KernelLibraryError(f"decode_chain: gains are contiguous float32 [{hidden}]")
    if arrived.dtype != torch.int32 or arrived.numel() != 4 or not arrived.is_contiguous():
        raise KernelLibraryError("decode_chain: arrived is four int32 zeros")
    x1, x2 = torch.empty_like(x), torch.empty_like(x)
    act = torch.empty(T, ff, device=x.device, dtype=x.dtype)
    out = torch.empty(T, next_proj.shape[0], device=x.device, dtype=x.dtype) if next_proj is not None else None
    squares = torch.empty(2 * T * lib().asb_decode_chain_blocks(), device=x.device, dtype=torch.float32)
    check(lib().asb_decode_chain(
        ptr(attn), ptr(o_proj), ptr(x), ptr(x1), ptr(gain), float(eps), ptr(gate_up), ptr(act), ptr(down), ptr(x2), ptr(next_gain),
        float(next_eps), ptr(next_proj), ptr(out), ptr(squares), ptr(arrived), T, hidden, o_proj.shape[1], ff,
        0 if next_proj is None else next_proj.shape[0], ptr(gemm_status(x.device)), stream()))  # fmt: skip
    return x2, out
