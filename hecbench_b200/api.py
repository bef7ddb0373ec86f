"""Host-side mirror of the reference launchers, on torch CUDA tensors.

Each function keeps the name, argument order and in/out convention of the
HeCBench launcher it stands in for (file:line given per function; paths
relative to the HeCBench source tree) and forwards to the C ABI of libhq.so on
the current torch CUDA stream (lib.host, a native extension: for a decode-time
mat-vec the host side of the call would otherwise take longer than the kernel).
Arguments are validated there and here the way the C ABI validates them; errors
surface as HqError / TypeError, never as a silent fallback.
"""
from __future__ import annotations

from typing import Optional, Sequence

import torch

from ._lib import load_library

NF4_HIGH_NIBBLE_FIRST = 0
NF4_WEIGHTS_RESIDENT = 2
NF4_LOW_NIBBLE_FIRST = 1


# --------------------------------------------------------------------------
# quant3MatMul
# --------------------------------------------------------------------------

def vecquant3matmul(vec, mat, mul, scales, zeros, height: int, width: int) -> None:
    """vecquant3matmul<float> (quant3MatMul-cuda/kernels.h:171-190).

    mul[c] += sum_k (scales[c]*q[k][c] - zeros[c]) * vec[k]; `mul` is
    accumulated into, exactly like the reference (the caller zeroes it)."""
    load_library().host.hq_q3_gemv_f32(vec, mat, mul, scales, zeros, height, width)


def vecquant3matmul_faster(vec, mat, mul, scales, zeros, height: int, width: int) -> None:
    """vecquant3matmul_faster (quant3MatMul-cuda/kernels.h:193-217): fp16 input."""
    load_library().host.hq_q3_gemv_f16in(vec, mat, mul, scales, zeros, height, width)


def vecquant3_dequant(mat, scales, zeros, height: int, width: int,
                      dtype: torch.dtype = torch.float32) -> torch.Tensor:
    """Dequantised weights W[K][width] by the fp32 rule (kernels.h:43) or the
    fp16 rule (kernels.h:121-122,137)."""
    host = load_library().host
    fn = {torch.float32: host.hq_q3_dequant_f32, torch.float16: host.hq_q3_dequant_f16}[dtype]
    W = host.empty(mat, dtype, height * 32 // 3, width)
    fn(mat, scales, zeros, W, height, width)
    return W


# --------------------------------------------------------------------------
# quantBnB
# --------------------------------------------------------------------------

def kQuantize(code, A, out, n: int) -> None:
    """kQuantize<256,256><<<grid,block>>>(code, A, out, n)
    (quantBnB-cuda/main.cu:90-130,176)."""
    if n > A.numel() or n > out.numel():
        raise ValueError("n exceeds the buffers")
    load_library().host.hq_bnb_quantize_u8(code, A, out, n)


def dequantize_nf4(B, absmax, lut16, n: int, blocksize: int = 64,
                   nibble_order: int = NF4_HIGH_NIBBLE_FIRST,
                   out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """NF4 blockwise dequantize to fp16 (no counterpart in the reference tree):
    out[e] = half_rn(lut16[code_e] * absmax[e // blocksize])."""
    host = load_library().host
    if out is None:
        out = host.empty(B, torch.float16, n)
    host.hq_nf4_dequant_f16(B, absmax, lut16, out, n, blocksize, nibble_order)
    return out


def gemv_nf4(A, B, absmax, lut16, N: int, K: int, blocksize: int = 64,
             nibble_order: int = NF4_HIGH_NIBBLE_FIRST,
             out: Optional[torch.Tensor] = None, weights_resident: bool = False) -> torch.Tensor:
    """NF4 4-bit GEMV (no counterpart in the reference tree):
    out[n] = half(sum_k A[k] * lut16[code[n][k]] * absmax[(n*K+k)//blocksize]).
    weights_resident: B, absmax and lut16 are not written by earlier work in the
    stream, so the kernel may fetch them while the preceding kernel is finishing."""
    host = load_library().host
    if out is None:
        out = host.empty(B, torch.float16, N)
    host.hq_nf4_gemv_f16(A, B, absmax, lut16, out, N, K, blocksize,
                         nibble_order | (NF4_WEIGHTS_RESIDENT if weights_resident else 0))
    return out


# --------------------------------------------------------------------------
# quantVLLM: per-token int8 activation quantization
# --------------------------------------------------------------------------

_VLLM_DTYPE = {torch.float16: 0, torch.bfloat16: 1, torch.float32: 2}


def _vllm_input(input, hidden_size: int, num_tokens: int) -> int:
    if not isinstance(input, torch.Tensor) or not input.is_cuda:
        raise TypeError("input: must be a CUDA tensor (there is no CPU path)")
    if input.dtype not in _VLLM_DTYPE:
        raise TypeError(f"input: expected float16, bfloat16 or float32, got {input.dtype}")
    if not input.is_contiguous() or input.numel() != hidden_size * num_tokens:
        raise TypeError("input: must be contiguous [num_tokens][hidden_size]")
    return _VLLM_DTYPE[input.dtype]


def static_scaled_int8_quant(output, input, hidden_size: int, num_tokens: int, scale: float,
                             azp: int = 0) -> None:
    """static_scaled_int8_quant<scalar_t>(output, input, hidden_size, num_tokens,
    scale, azp) (quantVLLM-cuda/main.cu:137-153): azp == 0 selects the form
    without zero point, as in the reference."""
    code = _vllm_input(input, hidden_size, num_tokens)
    if output.numel() != input.numel():
        raise ValueError("output and input differ in size")
    load_library().host.hq_vllm_static_scaled_int8_quant(output, input, code, hidden_size,
                                                         num_tokens, float(scale), int(azp))


def dynamic_scaled_int8_quant(output, input, hidden_size: int, num_tokens: int, scales,
                              azp=None) -> None:
    """dynamic_scaled_int8_quant<scalar_t>(output, input, hidden_size, num_tokens,
    scales, azp) (quantVLLM-cuda/main.cu:155-172): scales float32[num_tokens]
    and, when azp (int32[num_tokens]) is given, the per-token zero points are
    written too."""
    code = _vllm_input(input, hidden_size, num_tokens)
    if output.numel() != input.numel() or scales.numel() < num_tokens:
        raise ValueError("output / scales are too small")
    if azp is not None and azp.numel() < num_tokens:
        raise ValueError("azp is too small")
    load_library().host.hq_vllm_dynamic_scaled_int8_quant(output, input, code, hidden_size,
                                                          num_tokens, scales, azp)


# --------------------------------------------------------------------------
# gemv: uniform int8 / int4 weight-only mat-vec
# --------------------------------------------------------------------------

def _gemv_out(host, mat, vec, n: int, out):
    rows = mat.shape[0]
    if vec.numel() != n:
        raise ValueError(f"vec has {vec.numel()} elements, a row of mat {n}")
    if out is None:
        out = host.empty(mat, torch.float16, rows)
    elif out.numel() < rows:
        raise ValueError("out is too small")
    return rows, out


def gemv_fp16(mat, vec, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """gemv_fp16 behind solve_gemv_with_params (gemv-cuda/kernels.h:64-123,
    gemv.cu:61-81): mat fp16 [rows][n], vec fp16 [n] -> fp16 [rows]."""
    host = load_library().host
    n = mat.shape[1]
    rows, out = _gemv_out(host, mat, vec, n, out)
    host.hq_gemv_f16(mat, vec, out, rows, n)
    return out


def gemv_int8_quantized(mat, vec, scale: float, zero_point: float,
                        out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """gemv_quantized_int8 behind solve_gemv_int8_quantized_with_params
    (gemv-cuda/kernels.h:127-200, gemv.cu:38-59): mat int8 [rows][n]; scale and
    zero_point are rounded to fp16 as the reference launcher does."""
    host = load_library().host
    n = mat.shape[1]
    rows, out = _gemv_out(host, mat, vec, n, out)
    host.hq_gemv_int8_f16(mat, vec, out, rows, n, scale, zero_point)
    return out


def gemv_int4_quantized(mat, vec, scale: float, zero_point: float,
                        out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """gemv_quantized_int4 behind solve_gemv_int4_quantized_with_params
    (gemv-cuda/kernels.h:205-307, gemv.cu:15-36): mat uint8 [rows][n/2], element
    2j in the low nibble of byte j (uint4_2, kernels.h:9-32)."""
    host = load_library().host
    n = 2 * mat.shape[1]
    rows, out = _gemv_out(host, mat, vec, n, out)
    host.hq_gemv_int4_f16(mat, vec, out, rows, n, scale, zero_point)
    return out


# --------------------------------------------------------------------------
# quantization parameters and packers
# --------------------------------------------------------------------------

def zero_point(x_min, x_max, qmin: int, qmax: int, size: int, preserve_sparsity: bool, scale,
               zero_point_out) -> None:
    """zero_point<<<...>>>(x_min, x_max, qmin, qmax, size, preserve_sparsity, scale,
    zero_point) (zeropoint-cuda/main.cu:10-18): fp32 scale and int32 zero point of
    every channel from its minimum and maximum."""
    if min(x_min.numel(), x_max.numel(), scale.numel(), zero_point_out.numel()) < size:
        raise ValueError("a tensor is shorter than size")
    load_library().host.hq_zero_point(x_min, x_max, int(qmin), int(qmax), int(size),
                                      int(bool(preserve_sparsity)), scale, zero_point_out)


def quantize_q3(W, mat=None, scales=None, zeros=None):
    """Round-to-nearest 3-bit quantizer and packer (per-column min / max, the layout
    of quant3MatMul-cuda/kernels.h:41-87; no counterpart in the reference tree):
    W[K][N] float16 / bfloat16 / float32 -> (mat int32[K*3/32][N], scales float32[N],
    zeros float32[N]) as vecquant3matmul consumes them."""
    lib = load_library()
    code = _VLLM_DTYPE.get(W.dtype)
    if code is None:
        raise TypeError("W must be float16, bfloat16 or float32")
    if W.dim() != 2 or not W.is_cuda or not W.is_contiguous():
        raise ValueError("W must be a contiguous 2-D CUDA tensor")
    K, N = W.shape
    host = lib.host
    if mat is None:
        mat = host.empty(W, torch.int32, K * 3 // 32, N)
    if scales is None:
        scales = host.empty(W, torch.float32, N)
    if zeros is None:
        zeros = host.empty(W, torch.float32, N)
    nbytes = int(lib.hq_q3_quantize_workspace_bytes(N))
    ws = host.empty(W, torch.uint8, max(nbytes, 4))
    host.hq_q3_quantize(W, code, K, N, mat, scales, zeros, ws, nbytes)
    return mat, scales, zeros


def quantize_bcq(W, nb: int = 3, group_size: int = 128, bias: bool = True):
    """Greedy binary-coding quantizer (no counterpart in the reference tree): W[K][M]
    float16 / bfloat16 / float32 -> (bW int32[K/32][nb][M] sign planes, alpha
    float16[K/group_size][nb][M], q_bias float16[K/group_size][M] or None), the
    arrays nQWeight_fp16 takes."""
    host = load_library().host
    code = _VLLM_DTYPE.get(W.dtype)
    if code is None:
        raise TypeError("W must be float16, bfloat16 or float32")
    if W.dim() != 2 or not W.is_cuda or not W.is_contiguous():
        raise ValueError("W must be a contiguous 2-D CUDA tensor")
    K, M = W.shape
    G = K // group_size
    bW = host.empty(W, torch.int32, K // 32, nb, M)
    alpha = host.empty(W, torch.float16, G, nb, M)
    qb = host.empty(W, torch.float16, G, M) if bias else None
    host.hq_lutgemm_quantize(W, code, K, M, nb, group_size, bW, alpha, qb)
    return bW, alpha, qb


def quantize_nf4(W, lut16, blocksize: int = 64, nibble_order: int = NF4_HIGH_NIBBLE_FIRST,
                 B=None, absmax=None):
    """Blockwise 4-bit quantizer (the inverse of dequantize_nf4; no counterpart in
    the reference tree): W float16 / bfloat16 / float32 -> (B uint8[n / 2], absmax
    float32[n / blocksize]); code = the nearest of the 16 ascending levels lut16 to
    w / absmax, a tie going to the lower level."""
    host = load_library().host
    code = _VLLM_DTYPE.get(W.dtype)
    if code is None:
        raise TypeError("W must be float16, bfloat16 or float32")
    if not W.is_cuda or not W.is_contiguous():
        raise ValueError("W must be a contiguous CUDA tensor")
    n = W.numel()
    if B is None:
        B = host.empty(W, torch.uint8, n // 2)
    if absmax is None:
        absmax = host.empty(W, torch.float32, n // blocksize)
    host.hq_nf4_quantize(W, code, n, blocksize, lut16, nibble_order, B, absmax)
    return B, absmax


_MX_DTYPE = {torch.float16: 0, torch.bfloat16: 1}


def _mx_code(t) -> int:
    if t.dtype not in _MX_DTYPE:
        raise TypeError("MXFP4 takes float16 or bfloat16 tensors")
    if not t.is_cuda or not t.is_contiguous():
        raise ValueError("tensors must be contiguous CUDA tensors")
    return _MX_DTYPE[t.dtype]


def mxfp4(y, a, numel: int) -> None:
    """mxfp4<T>(y, a, numel, ...) (mxfp4-cuda/main.cu:152-176, without its timing
    loop): y = a quantized to MXFP4 and back, groups of 32, T = float16 or
    bfloat16."""
    code = _mx_code(a)
    if y.dtype != a.dtype or min(y.numel(), a.numel()) < numel:
        raise ValueError("y and a must have the same type and numel elements")
    load_library().host.hq_mxfp4_qdq(a, y, int(numel), code)


def mxfp4_quantize(a, codes=None, scales=None):
    """Packed MXFP4 of a float16 / bfloat16 tensor: (codes uint8[numel / 2], element
    2j in the low nibble; scales uint8[numel / 32], E8M0)."""
    host = load_library().host
    code = _mx_code(a)
    n = a.numel()
    if codes is None:
        codes = host.empty(a, torch.uint8, n // 2)
    if scales is None:
        scales = host.empty(a, torch.uint8, n // 32)
    host.hq_mxfp4_quantize(a, codes, scales, n, code)
    return codes, scales


def mxfp4_dequantize(codes, scales, dtype=torch.float16, out=None):
    """Values of a packed MXFP4 tensor in float16 or bfloat16."""
    host = load_library().host
    n = codes.numel() * 2
    if out is None:
        out = host.empty(codes, dtype, n)
    host.hq_mxfp4_dequantize(codes, scales, out, n, _mx_code(out))
    return out


# --------------------------------------------------------------------------
# RMSNorm -> mat-vec -> gated activation, fused
# --------------------------------------------------------------------------

ACT_NONE, ACT_SWIGLU, ACT_GEGLU = 0, 1, 2


def gemv_fused(fmt: str, x, mat, rows_out: int, *, gamma=None, eps: float = 1e-5, act: int = ACT_NONE,
               scale: float = 1.0, zero_point: float = 0.0, absmax=None, lut16=None,
               blocksize: int = 64, nibble_order: int = 0, weights_resident: bool = False,
               out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One launch for the entry of a decode-time MLP: RMSNorm of x (skipped when
    gamma is None; rmsnorm-cuda/reference.h:4-25), the weight-only mat-vec in
    format fmt ("f16", "int8", "int4", "nf4"; layouts and parameters as gemv_fp16,
    gemv_int8_quantized, gemv_int4_quantized, gemv_nf4) and, with act = ACT_SWIGLU
    or ACT_GEGLU, the gated activation of row pairs: mat then has 2 * rows_out
    rows, row 2m the value row and row 2m + 1 the gate row of output m
    (geglu-cuda/reference.h:8-16, swish-cuda/reference.h:4).  weights_resident
    (NF4): as in gemv_nf4, the weights may be fetched while the preceding kernel
    of the stream drains."""
    host = load_library().host
    n = x.numel()
    if out is None:
        out = host.empty(x, torch.float16, rows_out)
    if fmt == "f16":
        host.hq_gemv_fused_f16(x, gamma, eps, mat, out, rows_out, n, act)
    elif fmt == "int8":
        host.hq_gemv_fused_int8_f16(x, gamma, eps, mat, out, rows_out, n, scale, zero_point, act)
    elif fmt == "int4":
        host.hq_gemv_fused_int4_f16(x, gamma, eps, mat, out, rows_out, n, scale, zero_point, act)
    elif fmt == "nf4":
        host.hq_gemv_fused_nf4_f16(x, gamma, eps, mat, absmax, lut16, out, rows_out, n, blocksize,
                                   nibble_order | (NF4_WEIGHTS_RESIDENT if weights_resident else 0),
                                   act)
    else:
        raise ValueError(f"unknown format {fmt!r}")
    return out


# --------------------------------------------------------------------------
# lut-gemm
# --------------------------------------------------------------------------

def _stream_scratch(host, cache: dict, key, nbytes: int, like: torch.Tensor) -> torch.Tensor:
    """The zero-initialised scratch of `cache` for `key`, which names the device and
    current stream of `like`: calls on different streams may overlap on the GPU and
    must not share partial sums and counters.  Scratch that is first needed while the
    stream is being captured is not kept: its clearing belongs to that graph, so an
    eager call or another graph would find it uncleared."""
    ws = cache.get(key)
    if ws is None:
        ws = torch.zeros(nbytes, dtype=torch.uint8, device=like.device)
        if not host.capturing(like):
            cache[key] = ws
    return ws


class nQWeight_fp16:
    """Mirror of class nQWeight_fp16 (lut-gemm-cuda/nQWeight_fp16.h:22-45,
    nQWeight_fp16.cu:22-53): holds the bit-plane weights, fp16 alphas and the
    optional fp16 q_bias on the device.  `parsing` takes the same host-side
    arrays (uint32 bit planes [K/32][nb][M], fp32 alpha [groups][nb][M], fp32
    q_bias [groups][M] or None) and converts alpha / q_bias to fp16."""

    def __init__(self, bW=None, A=None, row: int = 0, col: int = 0, num_bits: int = 0,
                 is_row_wise_quantize: bool = False, num_alpha_groups: int = 1, q_bias=None,
                 device="cuda"):
        self.bWeight = self.alpha = self.q_bias = None
        self.num_groups = self.group_size = self.mSize = self.kSize = self.nb = 0
        self.is_row_wise_quantize = False
        self._ws = {}
        if bW is not None:
            self.parsing(bW, A, row, col, num_bits, is_row_wise_quantize, num_alpha_groups,
                         q_bias, device)

    def parsing(self, bW, A, row: int, col: int, num_bits: int, is_row_wise_quantize: bool,
                num_alpha_groups: int = 1, q_bias=None, device="cuda") -> None:
        self.num_groups = num_alpha_groups
        self.nb = num_bits
        self.is_row_wise_quantize = is_row_wise_quantize
        self.mSize, self.kSize = (row, col) if is_row_wise_quantize else (col, row)
        # the reference computes group_size before kSize is set
        # (nQWeight_fp16.cu:25); its launcher uses kSize/num_groups (mv_fp16.h:235)
        self.group_size = self.kSize // num_alpha_groups
        dev = torch.device(device)
        bW_t = torch.as_tensor(bW)
        if bW_t.dtype == torch.uint32:
            bW_t = bW_t.view(torch.int32)
        self.bWeight = bW_t.to(torch.int32).reshape(-1).contiguous().to(dev)
        self.alpha = torch.as_tensor(A, dtype=torch.float32).reshape(-1).to(torch.float16).to(dev)
        self.q_bias = None if q_bias is None else \
            torch.as_tensor(q_bias, dtype=torch.float32).reshape(-1).to(torch.float16).to(dev)
        need_w = self.kSize * self.mSize * self.nb // 32
        if self.bWeight.numel() != need_w:
            raise ValueError("bW has the wrong number of words")
        if self.alpha.numel() != self.num_groups * self.mSize * self.nb:
            raise ValueError("alpha has the wrong number of elements")

    def workspace(self) -> torch.Tensor:
        """Zero-initialised fp32 scratch the kernel accumulates K tiles into, one per
        device and current stream; it is left zero by every call."""
        lib = load_library()
        return _stream_scratch(lib.host, self._ws, (lib.host.place(self.bWeight), self.mSize),
                               lib.hq_lutgemm_workspace_bytes(self.mSize), self.bWeight)


def matmul(output, input, nqW: nQWeight_fp16, m: int = 1, algo: int = 0) -> None:
    """matmul(void* output, void* input, nQWeight_fp16& nqW, int m, int algo)
    (lut-gemm-cuda/kernels.cu:27-31): overwrites output[0:mSize] with the
    mat-vec of one input row (like the reference, only batch 1 is computed)."""
    ws = nqW.workspace()
    load_library().host.hq_lutgemm_nqmv(output, input, nqW.bWeight, nqW.alpha, nqW.q_bias,
                                        nqW.mSize, nqW.kSize, nqW.nb, nqW.group_size, ws,
                                        ws.numel())


# --------------------------------------------------------------------------
# quantAQLM
# --------------------------------------------------------------------------

def code1x16_matvec(A, B, C_out, codebook, prob_m: int, prob_k: int,
                    codebook_a_sizes: Sequence[int], codebook_stride: int,
                    scales: Optional[torch.Tensor] = None) -> None:
    """code1x16_matvec (quantAQLM-cuda/main.cu:113-141).  A = codes (int16 or
    uint16, [prob_m][prob_k/8]), B = input half[prob_k], C_out = half[prob_m]
    (overwritten), codebook half[..][65536][8]; `scales` is an extension.
    prob_k <= 8192.  codebook_a_sizes: up to four numbers, those left out count as 0;
    row m takes the codebook as many strides in as there are values <= m among the
    first three."""
    if A.dtype not in (torch.int16, torch.uint16):
        raise TypeError("A: expected int16/uint16 codes")
    sizes = codebook_a_sizes
    if not isinstance(sizes, (list, tuple)):
        sizes = list(sizes)
    if len(sizes) < 3:
        # a limit of 0 moves every row on: the codebook that the rows reach must be there
        last = sum(int(v) < prob_m for v in [*sizes, 0, 0, 0][:3])
        if (last * codebook_stride + 65536) * 8 > codebook.numel():
            raise ValueError("codebook_a_sizes: rows beyond the last codebook")
    load_library().host.hq_aqlm_1x16_matvec(A, B, C_out, codebook, prob_m, prob_k, sizes,
                                            codebook_stride, scales)


def code2x8_matvec(A, B, C_out, codebooks, prob_m: int, prob_k: int,
                   scales: Optional[torch.Tensor] = None) -> None:
    """AQLM 2x8 mat-vec (no counterpart in the reference tree).  A = uint8 codes
    [prob_m][prob_k/8][2], codebooks half[2][256][8]."""
    load_library().host.hq_aqlm_2x8_matvec(A, B, C_out, codebooks, prob_m, prob_k, scales)


# --------------------------------------------------------------------------
# batched dequant-GEMM (tensor cores)
# --------------------------------------------------------------------------

_qgemm_ws = {}


def _qgemm_workspace(lib, X, Mb: int, N: int):
    """Split-K scratch (fp32 partial sums and tile counters), one per (device, stream,
    Mb, N)."""
    ws = _stream_scratch(lib.host, _qgemm_ws, (lib.host.place(X), Mb, N),
                         lib.hq_qgemm_workspace_bytes(Mb, N), X)
    return ws, ws.numel()


def qgemm_reset_workspaces() -> None:
    """Re-zero every cached split-K scratch on its device.  Call this after a
    batched product reported status 1 (a bounded in-kernel wait ran out): such a
    call may leave partial sums and tile counters behind, and the kernels rely on
    finding the scratch zero."""
    for ws in _qgemm_ws.values():
        ws.zero_()


def qgemm_q3(X, mat, scales, zeros, N: int, K: int, group_size: int = 128,
             out: Optional[torch.Tensor] = None,
             status: Optional[torch.Tensor] = None, split_k: bool = True,
             peers=None) -> Optional[torch.Tensor]:
    """Y[Mb][N] = X[Mb][K] @ dequant(mat) for the GPTQ 3-bit layout with per-group
    fp16 scales / zeros [K/group_size][N] (no counterpart in the reference tree).
    `status` (int32[1], optional) receives 1 if a bounded in-kernel wait ran out;
    call qgemm_reset_workspaces() before the next product in that case.
    With split_k a zero-initialised scratch matrix is kept per (device, stream, Mb, N);
    the parts of K meet in it in a fixed order for wide layers only (hq.h), so
    split_k=False is the way to the same bits on every call for any shape.
    peers = (pointer_table, offset_elements, world): store every finished tile into
    the output slice of every GPU of the node instead of `out` (hq_qgemm_q3_f16_peers);
    returns None in that form."""
    lib = load_library()
    host = lib.host
    Mb = X.shape[0]
    ws, ws_bytes = _qgemm_workspace(lib, X, Mb, N) if split_k else (None, 0)
    if peers is not None:
        table, offset, world = peers
        host.hq_qgemm_q3_f16_peers(X, mat, scales, zeros, int(table), int(offset), int(world), Mb,
                                   N, K, group_size, ws, ws_bytes, status)
        return None
    if out is None:
        out = host.empty(X, torch.float16, Mb, N)
    host.hq_qgemm_q3_f16(X, mat, scales, zeros, out, Mb, N, K, group_size, ws, ws_bytes, status)
    return out


def qgemm_nf4(X, B, absmax, lut16, N: int, K: int, blocksize: int = 64, nibble_order: int = 0,
              out: Optional[torch.Tensor] = None, status: Optional[torch.Tensor] = None,
              split_k: bool = True, peers=None) -> Optional[torch.Tensor]:
    """Y[Mb][N] = X[Mb][K] @ W with W[k][n] the NF4 weight that dequantize_nf4
    gives for element n*K + k of B (uint8[N*K/2], absmax per `blocksize`
    elements); same conventions as gemv_nf4, same workspace, status and `peers`
    rules as qgemm_q3 (no counterpart in the reference tree).  Fastest with blocks of
    64, K a multiple of 128 and absmax on 16 bytes, as a fresh tensor is (hq.h)."""
    lib = load_library()
    host = lib.host
    Mb = X.shape[0]
    ws, ws_bytes = _qgemm_workspace(lib, X, Mb, N) if split_k else (None, 0)
    if peers is not None:
        table, offset, world = peers
        host.hq_qgemm_nf4_f16_peers(X, B, absmax, lut16, int(table), int(offset), int(world), Mb,
                                    N, K, blocksize, nibble_order, ws, ws_bytes, status)
        return None
    if out is None:
        out = host.empty(X, torch.float16, Mb, N)
    host.hq_qgemm_nf4_f16(X, B, absmax, lut16, out, Mb, N, K, blocksize, nibble_order, ws,
                          ws_bytes, status)
    return out
