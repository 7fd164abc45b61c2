"""Wrapper of the tcgen05 / TMA matrix product (bfloat16 operands, f32 accumulation in tensor memory)."""
from __future__ import annotations

from ctypes import c_float, c_int, c_int64, c_void_p
from typing import Optional

import torch

from .lib import KernelError, check, num_sms, ptr, require_cuda, stream_handle
from .ops import _fn, gate_constants

DECODE_MAX_TOKENS = 64          # up to here the operands are swapped (weight rows fill the tile)
MAX_SPLITS = 8                  # the portable cluster size

# Per device: the status word the tcgen05 kernels set when a bounded wait runs out.
_STATE = {}


def _state(device):
    st = _STATE.get(device)
    if st is None:
        st = {"status": torch.zeros(1, dtype=torch.int32, device=device)}
        _STATE[device] = st
    return st


def _device(device=None) -> torch.device:
    device = torch.device(device if device is not None else torch.cuda.current_device())
    if device.type == "cuda" and device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    return device


def device_status(device=None) -> int:
    """The status word of the kernels with bounded waits (0 = fine).  Reading it synchronizes."""
    st = _STATE.get(_device(device))
    return int(st["status"].item()) if st else 0


# what a kernel was waiting for when it gave up (the code it left in the status word)
STATUS_MEANING = {
    1: "matrix product: the TMA producer waited for a free shared-memory stage",
    2: "matrix product: the MMA thread waited for an operand tile (or a free accumulator)",
    3: "matrix product: the epilogue warps waited for the accumulator",
    11: "prompt attention: the TMA producer waited for a free K/V stage",
    12: "prompt attention: the MMA thread waited for the Q or the first K tiles",
    13: "prompt attention: the MMA thread waited for the softmax warps' P tile",
    14: "prompt attention: the MMA thread waited for a K or V tile",
    15: "prompt attention: the softmax warps waited for a score tile or for P V to finish",
    16: "prompt attention: the softmax warps waited for the last P V before writing the output",
    21: "decode attention: the TMA producer waited for a free stage",
    22: "decode attention: the compute warps waited for a key/value tile",
    31: "attention over expanded latents: a TMA producer waited for a free K or V stage",
    32: "attention over expanded latents: the MMA thread waited for the Q or the first K tiles",
    33: "attention over expanded latents: the MMA thread waited for the softmax warps' P tile",
    34: "attention over expanded latents: the MMA thread waited for a K or V tile",
    35: "attention over expanded latents: the softmax warps waited for a score tile",
    36: "attention over expanded latents: the softmax warps waited for the last P V before writing the output",
    37: "attention over expanded latents: the step's portions pass the rows or row tiles its launch was made for",
    41: "32-bit product: the splitting warps waited for a free stage",
    42: "32-bit product: an MMA thread waited for a split stage or a free accumulator",
    43: "32-bit product: the summing warps waited for a stage's sums",
    44: "32-bit product: the TMA producer waited for a free stage",
    45: "32-bit product: the splitting warps waited for an operand tile",
    46: "routed products: the TMA producer waited for a free stage",
    47: "routed products: a warp waited for the experts' weights",
    51: "state-space chunks: the sums waited for their operands or their MMAs",
    52: "state-space chunks: the outputs waited for their operands or their MMAs",
    53: "state-space chunks: the step has more portions than its launch was made for",
}


def describe_status(code: int) -> str:
    return STATUS_MEANING.get(int(code), "unknown code")


def check_status(device=None) -> None:
    """Raise if a kernel gave up one of its bounded waits, or met a step beyond its launch's bounds.  The word stays set (every later check raises too)
    until ``reset_status``: after such a fault the step's results are not to be trusted."""
    code = device_status(device)
    if code:
        what = "met a step beyond its launch's bounds" if code in (37, 53) else "gave up a bounded wait and returned early"
        raise KernelError(f"a kernel {what} (status {code}: "
                          f"{describe_status(code)}); the results of that step are invalid")


def reset_status(device=None) -> int:
    """Clear the status word; returns the code it held."""
    st = _STATE.get(_device(device))
    if st is None:
        return 0
    code = int(st["status"].item())
    st["status"].zero_()
    return code


def wait_probe(polls: int = 1000, device=None) -> int:
    """Launch one CTA that allocates tensor memory and waits, with the products' own bounded wait cut down to
    ``polls`` polls, on an mbarrier nobody arrives at; it must give up, record code 2 in the status word, free its
    tensor memory and return.  Returns the status word after it (reading synchronizes).  For tests of the
    failure path; nothing in the engine calls it."""
    device = _device(device)
    st = _state(device)
    lib, f = _fn("gemm_tc", "dinfer_gemm_tc_wait_probe", [c_void_p, c_int, c_void_p])
    with torch.cuda.device(device):
        check(lib, f(ptr(st["status"]), int(polls), stream_handle()), "gemm_tc_wait_probe")
    return device_status(device)


def supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    """bfloat16 operands whose rows TMA can address: K and the row strides multiples of 8 elements."""
    return (x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.dim() == 2 and w.dim() == 2
            and x.shape[1] % 8 == 0 and x.stride(1) == 1 and w.stride(1) == 1
            and x.stride(0) % 8 == 0 and w.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def decode_splits(tokens: int, N: int, K: int) -> int:
    """K splits of the decode orientation: one wave of CTAs (three fit an SM up to 16 tokens, two
    beyond), at least four 64-wide K blocks per CTA (at eight, one row of 1024 x 2048 took 4.8 us, now 3.9;
    4096 x 1024 5.1 and 4.2, 6144 x 1024 5.6 and 4.9, 1024 x 3072 4.9 and 4.6), at most ``MAX_SPLITS`` (the CTAs of a tile are
    one thread-block cluster)."""
    tiles = (N + 127) // 128
    k_blocks = (K + 63) // 64
    sms = num_sms()
    # a tile's CTAs are one cluster and a cluster stays inside a part of the chip, so not every slot can be filled:
    # 384 CTAs in clusters of 8 run as one wave of 3 an SM, 392 do not, nor do 432 in clusters of 3
    slots = 3 * sms - 58 if tokens <= 16 else 2 * sms - 16
    return max(1, min(slots // tiles, k_blocks // 4, MAX_SPLITS))


# the gates the product's epilogue knows; the clamped gate comes with its constants (see ops.gate_constants)
GATES = {False: 0, None: 0, True: 1, "silu": 1, "gelu_tanh": 2, "clamped_swish": 3}
# the activations it knows without a gate; an xIELU comes as ("xielu", a_pos, a_neg)
UNARY = {None: 0, "relu2": 1, "silu": 2, "gelu_tanh": 3, "relu": 4, "xielu": 5}


def gemm_tc(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor, splits: Optional[int] = None,
            gated=False, residual: Optional[torch.Tensor] = None, norm_weight: Optional[torch.Tensor] = None,
            sums: Optional[torch.Tensor] = None, row_scale=None, activation=None) -> torch.Tensor:
    """out[tokens, N] = x[tokens, K] @ w[N, K]^T.  out: bfloat16 or float32, last axis contiguous.

    ``gated`` (any number of rows; True or "silu", "gelu_tanh", or a clamped gate with its constants): the rows of w are (gate, up) pairs, out is
    [tokens, N / 2], out[t, j] = g(x w_2j) * (x w_2j+1) with that g.
    ``activation`` (any number of rows; no gate, no residual): a key of ``UNARY`` or ("xielu", a_pos, a_neg), applied to
    the result.
    Epilogues of the decode orientation (at most ``DECODE_MAX_TOKENS`` rows):
      ``residual`` [tokens, N] f32 with ``norm_weight`` [N] and ``sums`` [parts, stride >= tokens] f32
        (``parts = residual_parts(...)``): the product is added into the residual, out gets the new
        residual times the norm weight, ``sums[p, t]`` the squares of row t summed over part p;
      ``row_scale = (sums, parts, size, eps)``: out[t] *= rsqrt(sum_p sums[p, t] / size + eps).
    """
    require_cuda(x, w, out)
    if not supported(x, w):
        raise KernelError("gemm_tc: bfloat16 operands with K and row strides multiples of 8 and 16-byte aligned bases")
    tokens, K = x.shape
    N = w.shape[0]
    gated, gate_a, gate_b = gate_constants(gated)
    if gated not in GATES:
        raise KernelError(f"gemm_tc: unknown gate {gated!r}")
    if (residual is not None or row_scale is not None) and tokens > DECODE_MAX_TOKENS:
        raise KernelError("gemm_tc: the norm epilogues take at most 64 rows")
    unary, a_pos, a_neg = activation if isinstance(activation, (tuple, list)) else (activation, gate_a, gate_b)
    if unary not in UNARY or (unary == "xielu") != isinstance(activation, (tuple, list)) or (unary and (gated or residual is not None)):
        raise KernelError(f"gemm_tc: activation {activation!r}: one of {', '.join(str(k) for k in UNARY)}, without a gate or a residual")
    if gated and (N % 2 or residual is not None):
        raise KernelError("gemm_tc: the gated epilogue needs an even number of weight rows and no residual")
    if w.shape[1] != K or out.shape != (tokens, N // 2 if gated else N) or out.stride(1) != 1 \
            or out.dtype not in (torch.bfloat16, torch.float32):
        raise KernelError(f"gemm_tc: shapes x{tuple(x.shape)} w{tuple(w.shape)} out{tuple(out.shape)} do not agree")
    st = _state(x.device)
    if tokens <= DECODE_MAX_TOKENS:
        splits = decode_splits(tokens, N, K) if splits is None else max(1, min(int(splits), MAX_SPLITS))
    else:
        splits = 1
    r_ptr = nw_ptr = so_ptr = si_ptr = None
    ldr = nw_f32 = parts = stride = 0
    inv_size = eps = 0.0
    if residual is not None:
        require_cuda(residual, norm_weight, sums)
        if (residual.dtype != torch.float32 or residual.shape != (tokens, N) or residual.stride(1) != 1
                or norm_weight.shape != (N,) or not norm_weight.is_contiguous()
                or norm_weight.dtype not in (torch.bfloat16, torch.float32)
                or sums.dtype != torch.float32 or sums.dim() != 2 or sums.stride(1) != 1 or sums.shape[1] < tokens
                or sums.shape[0] < residual_parts(tokens, N, K, splits)):
            raise KernelError("gemm_tc: residual [tokens, N] f32, norm_weight [N], sums [parts, >= tokens] f32")
        r_ptr, ldr, nw_ptr, nw_f32 = ptr(residual), residual.stride(0), ptr(norm_weight), int(norm_weight.dtype == torch.float32)
        so_ptr, stride = ptr(sums), sums.stride(0)
    if row_scale is not None:
        s_in, parts, size, eps = row_scale
        require_cuda(s_in)
        if s_in.dtype != torch.float32 or s_in.dim() != 2 or s_in.stride(1) != 1 or s_in.shape[1] < tokens \
                or not (0 < parts <= s_in.shape[0]):
            raise KernelError("gemm_tc: row_scale sums [parts, >= tokens] f32")
        if residual is not None and s_in.stride(0) != stride:
            raise KernelError("gemm_tc: the sums read and written must have one row stride")
        si_ptr, stride, inv_size = ptr(s_in), s_in.stride(0), 1.0 / float(size)
    lib, f = _fn("gemm_tc", "dinfer_gemm_tc_all",
                 [c_void_p, c_int64, c_void_p, c_int64, c_void_p, c_int64, c_int, c_int, c_int, c_int, c_int, c_int,
                  c_int, c_float, c_float,
                  c_void_p, c_int64, c_void_p, c_int, c_void_p, c_void_p, c_int, c_int, c_float, c_float,
                  c_void_p, c_void_p])
    check(lib, f(ptr(x), x.stride(0), ptr(w), w.stride(0), ptr(out), out.stride(0), int(out.dtype == torch.float32),
                 tokens, N, K, int(splits), GATES[gated], UNARY[unary], float(a_pos), float(a_neg), r_ptr, ldr, nw_ptr, nw_f32, so_ptr, si_ptr, int(parts),
                 int(stride), float(inv_size), float(eps), ptr(st["status"]), stream_handle()), "gemm_tc")
    return out


# the longest input of a lone token's product (shared memory)
GEMV_MAX_K = 12 * 1024 - 16


def gemv_supported(w: torch.Tensor) -> bool:
    """A matrix whose product with one bfloat16 row ``gemv`` takes."""
    return (w.dtype == torch.bfloat16 and w.dim() == 2 and w.shape[1] % 8 == 0 and w.shape[1] <= GEMV_MAX_K and w.stride(1) == 1
            and w.stride(0) % 8 == 0 and w.data_ptr() % 16 == 0)


def gemv_norms(residual: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor) -> bool:
    """Whether ``gemv`` can make its input from these: 16-byte loads of each.  (The norm's own kernel takes any address.)"""
    return (residual.dtype == torch.float32 and residual.is_contiguous() and residual.data_ptr() % 16 == 0
            and (delta is None or (delta.dtype == torch.bfloat16 and delta.is_contiguous() and delta.data_ptr() % 16 == 0))
            and weight.dtype in (torch.bfloat16, torch.float32) and weight.is_contiguous() and weight.data_ptr() % 16 == 0)


def gemv(x: Optional[torch.Tensor], w: torch.Tensor, out: torch.Tensor, gated: bool = False, norm=None) -> torch.Tensor:
    """out[1, N] = x[1, K] @ w[N, K]^T for one row in bfloat16; ``gated``: the rows of w are (gate, up) pairs and out [1, N / 2]
    gets silu(gate) * up.  With ``norm = (residual [1, K] f32, delta [1, K] bfloat16 or None, residual_out [1, K] f32 or None,
    weight [K], eps)`` the input is the RMSNorm of residual + delta (rounded to bfloat16), and residual_out, another buffer
    than residual, gets the sum."""
    require_cuda(w, out)
    K, N = w.shape[1], w.shape[0]
    if not gemv_supported(w) or tuple(out.shape) != (1, N // 2 if gated else N) or out.stride(1) != 1 or (gated and N % 2) \
            or out.dtype not in (torch.bfloat16, torch.float32):
        raise KernelError(f"gemv: w{tuple(w.shape)} bfloat16 rows of 16-byte pieces, out{tuple(out.shape)} bfloat16 or float32")
    residual = delta = residual_out = weight = None
    eps = 0.0
    if norm is None:
        if x.dtype != torch.bfloat16 or tuple(x.shape) != (1, K) or x.stride(1) != 1 or x.data_ptr() % 16:
            raise KernelError("gemv: x bfloat16 [1, K], 16-byte aligned")
    else:
        residual, delta, residual_out, weight, eps = norm
        x = None
        if any(t is not None and tuple(t.shape) != (1, K) for t in (residual, delta, residual_out)) or weight.numel() != K \
                or not gemv_norms(residual, delta, weight) or (residual_out is not None and not gemv_norms(residual_out, None, weight)):
            raise KernelError("gemv: residual and residual_out float32 [1, K], delta bfloat16 [1, K], the norm's weight [K], 16-byte aligned")
        if delta is not None and (residual_out is None or residual_out.data_ptr() == residual.data_ptr()):
            raise KernelError("gemv: with a delta another buffer for the new residual")
    lib, f = _fn("gemv", "dinfer_gemv", [c_void_p, c_void_p, c_int64, c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_void_p,
                                         c_void_p, c_void_p, c_int, c_float, c_void_p])
    check(lib, f(ptr(x), ptr(w), w.stride(0), ptr(out), int(out.dtype == torch.float32), N, K, int(bool(gated)), ptr(residual),
                 ptr(delta), ptr(residual_out), ptr(weight), int(weight is not None and weight.dtype == torch.float32), float(eps),
                 stream_handle()), "gemv")
    return out


def residual_parts(tokens: int, N: int, K: int, splits: Optional[int] = None) -> int:
    """Rows of the ``sums`` the residual epilogue writes for these sizes."""
    if splits is None:
        splits = decode_splits(tokens, N, K)
    lib, f = _fn("gemm_tc", "dinfer_gemm_tc_parts", [c_int, c_int, c_int, c_int])
    return int(f(tokens, N, K, int(splits)))

