"""Tensor-level wrappers over the C ABI: PyTorch supplies device memory and streams only.

Types and shapes are checked here; allocating outputs and workspace and making the call is one native call for the entry points
that a forward or a step makes many of (csrc/host_ops.cpp; us per call from Python, before / now: fused norm 22.9 / 13.1,
quantizer 21.0 / 11.6, both orientations 28.4 / 15.8, column mean 15.2 / 8.3, vector product 9.7 / 5.3, product 9.9 / 6.8, of
which the launches take 3 to 6).  Every function needs CUDA tensors and the built library; nothing here computes on the CPU.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from . import cabi

_DTYPES = {torch.bfloat16: cabi.DTYPE_BF16, torch.float32: cabi.DTYPE_F32}

# Kernels of this library launched since import, by entry point (two per quantizer call: the
# streaming pass and the scale pass; a memset in front of them is not a kernel).  The quantizers and the column
# mean have one-launch forms for small inputs; those calls are counted as two all the same.
LAUNCHES = {"quantize": 0, "rmsnorm_quantize": 0, "dequantize": 0, "col_mean": 0, "gemv": 0, "gemm": 0, "lowrank_bwd": 0, "decoder": 0}


def launch_count() -> int:
    return sum(LAUNCHES.values())


def _dtype_code(t: torch.Tensor, what: str) -> int:
    try:
        return _DTYPES[t.dtype]
    except KeyError:
        raise TypeError(f"{what} must be bfloat16 or float32, got {t.dtype}") from None


def _need_cuda(t: torch.Tensor, what: str) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{what} must be a CUDA tensor: the NVFP4 path has no CPU fallback")


# torch.cuda.current_device() without its checks: a CUDA tensor exists.  (A torch without CUDA has the checked one only.)
_current_device = getattr(torch._C, "_cuda_getDevice", torch.cuda.current_device)


def _stream() -> int:
    return torch._C._cuda_getCurrentRawStream(_current_device())


class _on_device:
    """Makes `dev` current for the calls inside; free when it already is (the common case)."""
    __slots__ = ("guard",)

    def __init__(self, dev: torch.device):
        self.guard = None if dev.index == _current_device() else torch.cuda.device(dev)

    def __enter__(self):
        if self.guard is not None:
            self.guard.__enter__()

    def __exit__(self, *exc):
        if self.guard is not None:
            self.guard.__exit__(*exc)


_STREAMS = {}          # (stream id, device index, device type) -> torch.cuda.Stream: handles only, rebuilt when dropped


def _stream_object(key) -> "torch.cuda.Stream":
    st = _STREAMS.get(key)
    if st is None:
        if len(_STREAMS) >= 256:
            _STREAMS.clear()
        st = _STREAMS[key] = torch.cuda.Stream(stream_id=key[0], device_index=key[1], device_type=key[2])
    return st


def current_stream(dev: torch.device) -> "torch.cuda.Stream":
    """torch.cuda.current_stream(dev) for a device with an index, without building a new handle on every call."""
    return _stream_object(torch._C._cuda_getCurrentStream(_current_device() if dev.index is None else dev.index))


class on_stream:
    """torch.cuda.stream(st) at a tenth of its cost where st's device is the current one (elsewhere: the same)."""
    __slots__ = ("st", "prev", "full")

    def __init__(self, st: "torch.cuda.Stream"):
        self.st = st

    def __enter__(self):
        st = self.st
        self.full = None
        if st.device_index != _current_device():
            self.full = torch.cuda.stream(st)
            self.full.__enter__()
            return
        self.prev = torch._C._cuda_getCurrentStream(st.device_index)
        torch._C._cuda_setStream(stream_id=st.stream_id, device_index=st.device_index, device_type=st.device_type)

    def __exit__(self, *exc):
        if self.full is not None:
            self.full.__exit__(*exc)
            return
        prev = self.prev
        torch._C._cuda_setStream(stream_id=prev[0], device_index=prev[1], device_type=prev[2])


def recorded_event(st: "torch.cuda.Stream") -> "torch.cuda.Event":
    ev = torch.cuda.Event()
    ev.record(st)
    return ev


def _sf_bytes(R: int, Cc: int, sf_layout: int) -> int:
    """metis_nvfp4_sf_bytes: one byte per 16 elements, or whole tiles of 128 rows x 256 elements."""
    if sf_layout == cabi.SF_MMA:
        return ((R + 127) // 128) * ((Cc + 255) // 256) * 2048
    if sf_layout == cabi.SF_ROWMAJOR:
        return R * (Cc // 16)
    return cabi.lib().metis_nvfp4_sf_bytes(R, Cc, sf_layout)


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _rows2d(x: torch.Tensor) -> torch.Tensor:
    """View x as [rows, cols] with unit stride along cols (copy only if it has to)."""
    if x.dim() == 2 and x.is_contiguous() and x.stride(0) == x.shape[1]:      # (a single row may have any stride)
        return x
    x2 = x.reshape(-1, x.shape[-1])
    if x2.stride(-1) != 1 or (x2.shape[0] > 1 and x2.stride(0) < x2.shape[1]):
        x2 = x2.contiguous()
    return x2


@dataclass
class NVFP4Tensor:
    """A quantized [R, C] matrix: packed e2m1 codes, E4M3 block scales, fp32 unit.

    `row_vec` (fp32 [C]) is the mean that was subtracted before quantization; the represented
    matrix is value(codes, scales, unit) + 1 * row_vec (bitlinear.py:330-332).  For a
    transposed quantization of x [M, K] with column means, `col_vec` (fp32 [R]) holds them
    instead: the represented matrix is value + col_vec * 1^T.
    """
    codes: torch.Tensor          # uint8 [R, C/2]
    scales: torch.Tensor         # uint8, flat
    unit: torch.Tensor           # float32 [1]
    shape: tuple
    sf_layout: int
    row_vec: Optional[torch.Tensor] = None
    col_vec: Optional[torch.Tensor] = None
    token_sums: Optional[torch.Tensor] = None     # fp32 [R]: sums of the rows' quantized values, when the quantizer formed them

    @property
    def device(self):
        return self.codes.device

    def dequantize(self, dtype: torch.dtype = torch.float32, add_mean: bool = True) -> torch.Tensor:
        return nvfp4_dequantize(self, dtype, add_mean=add_mean)


def col_mean(x: torch.Tensor) -> torch.Tensor:
    """Column means of x viewed as [rows, cols], fp32 (input_flat.mean(dim=0), bitlinear.py:326)."""
    _need_cuda(x, "x")
    x2 = _rows2d(x)
    with _on_device(x2.device):
        rc, mean = cabi.host().col_mean(x2, _dtype_code(x2, "x"), _stream())
    if rc:
        cabi.check(rc, "metis_col_mean")
    LAUNCHES["col_mean"] += 2
    return mean


def _hadamard_flags(sign_mask: Optional[int]) -> int:
    """Flag bits that make the transposed quantizer rotate its blocks: sign_mask has bit i set where position
    i of every block of 16 is negated before the Hadamard butterfly; None: no rotation."""
    if sign_mask is None:
        return 0
    if not 0 <= sign_mask < 1 << 16:
        raise ValueError("sign_mask holds one bit per position of a block of 16")
    return cabi.Q_HADAMARD | (sign_mask << 16)


def _sr_flags(stochastic: bool, sr_bits: int) -> int:
    if sr_bits not in (8, 16):
        raise ValueError(f"sr_bits must be 8 (hardware conversion) or 16 (software), not {sr_bits}")
    return cabi.Q_SR16 if stochastic and sr_bits == 16 else 0


def _mean_row(mean: torch.Tensor, cols: int) -> torch.Tensor:
    _need_cuda(mean, "mean")
    if mean.dim() != 1 or mean.dtype != torch.float32 or not mean.is_contiguous():
        mean = mean.reshape(-1).to(torch.float32).contiguous()
    assert mean.numel() == cols
    return mean


def nvfp4_quantize(x: torch.Tensor, *, transpose: bool = False, stochastic: bool = False, seed: int = 0,
                   offset: int = 0, sf_layout: int = cabi.SF_MMA,
                   mean: Optional[torch.Tensor] = None,
                   offset_counter: Optional[torch.Tensor] = None,
                   hadamard_signs: Optional[int] = None, sr_bits: int = 8) -> NVFP4Tensor:
    """Quantize x (viewed as [rows, cols]) or, with transpose=True, its transpose.
    sr_bits: random bits per element of the stochastic rounding, 8 (the hardware conversion) or 16 (software).

    `mean` (fp32 [cols]) is subtracted from every row of x first.  Stochastic rounding draws
    Philox(seed; element, offset); with `offset_counter` (int64 [1] on x's device) the offset is that
    counter's value and the call increments it, so the call can sit in a CUDA graph that is replayed."""
    _need_cuda(x, "x")
    x2 = _rows2d(x)
    rows, cols = x2.shape
    R, Cc = (cols, rows) if transpose else (rows, cols)
    if Cc % 16 != 0 or R == 0:
        raise ValueError(f"NVFP4 block shape (1, 16) does not divide tensor shape {(R, Cc)}")
    flags = (cabi.Q_TRANSPOSE if transpose else 0) | (cabi.Q_STOCHASTIC if stochastic else 0) | _hadamard_flags(hadamard_signs)
    flags |= _sr_flags(stochastic, sr_bits)
    dev = x2.device
    if stochastic and offset_counter is not None:
        if offset_counter.dtype != torch.int64 or offset_counter.device != dev or offset_counter.numel() != 1:
            raise ValueError("offset_counter must be an int64 tensor with one element on the device of x")
        flags |= cabi.Q_OFFSET_ON_DEVICE
        offset = offset_counter.data_ptr()
    if mean is not None:
        mean = _mean_row(mean, cols)
    with _on_device(dev):
        rc, codes, scales, unit = cabi.host().quantize(x2, _dtype_code(x2, "x"), transpose, flags, seed & (2**64 - 1), offset & (2**64 - 1), sf_layout,
                                                       _sf_bytes(R, Cc, sf_layout), cabi.QUANTIZE_EXTRA_WORKSPACE, mean, _stream())
    if rc:
        cabi.check(rc, "metis_nvfp4_quantize")
    LAUNCHES["quantize"] += 2
    q = NVFP4Tensor(codes, scales, unit, (R, Cc), sf_layout)
    if mean is not None:
        if transpose:
            q.col_vec = mean
        else:
            q.row_vec = mean
    return q


def nvfp4_quantize_dual(x: torch.Tensor, *, stochastic: bool = False, seed: int = 0, offset: int = 0,
                        sf_layout: int = cabi.SF_MMA, mean: Optional[torch.Tensor] = None,
                        offset_counter: Optional[torch.Tensor] = None, hadamard_signs: Optional[int] = None,
                        token_sums: bool = False, defer: Optional[str] = None, sr_bits: int = 8):
    """Both quantizations of x viewed as [rows, cols] from one pass over it: (Q of x, Q of x^T), each
    bit-identical to the separate call (round to nearest).  rows and cols must be multiples of 16.
    With token_sums the second result carries `token_sums` (fp32 [cols]), the sums of its rows' quantized
    values, formed by the scale pass (where the shape allows it: rows a multiple of 64, no rotation).
    defer = "rowmajor" or "transposed": the scale pass of that output (its scales, unit, token sums) is left
    out; a third value is returned, a function that launches it on the stream that is current when it is
    called (the caller orders that stream after this call and its consumers after that launch)."""
    _need_cuda(x, "x")
    x2 = _rows2d(x)
    rows, cols = x2.shape
    if rows % 16 != 0 or cols % 16 != 0 or rows == 0:
        raise ValueError(f"NVFP4 block shape (1, 16) does not divide both dimensions of tensor shape {(rows, cols)}")
    flags = (cabi.Q_STOCHASTIC if stochastic else 0) | _hadamard_flags(hadamard_signs)      # rotation: the transposed output only
    flags |= _sr_flags(stochastic, sr_bits)
    if defer not in (None, "rowmajor", "transposed"):
        raise ValueError(f"defer must be 'rowmajor' or 'transposed', not {defer!r}")
    deferred = {None: 0, "rowmajor": cabi.Q_DEFER_ROWMAJOR, "transposed": cabi.Q_DEFER_TRANSPOSED}[defer]
    flags |= deferred
    dev = x2.device
    if stochastic and offset_counter is not None:
        if offset_counter.dtype != torch.int64 or offset_counter.device != dev or offset_counter.numel() != 1:
            raise ValueError("offset_counter must be an int64 tensor with one element on the device of x")
        flags |= cabi.Q_OFFSET_ON_DEVICE
        offset = offset_counter.data_ptr()
    if mean is not None:
        mean = _mean_row(mean, cols)
    host = cabi.host()
    with _on_device(dev):
        rc, codes, scales, unit, codes_t, scales_t, unit_t, sums, ws = host.quantize_dual(
            x2, _dtype_code(x2, "x"), flags, seed & (2**64 - 1), offset & (2**64 - 1), sf_layout, _sf_bytes(rows, cols, sf_layout),
            _sf_bytes(cols, rows, sf_layout), mean, token_sums and rows % 64 == 0 and hadamard_signs is None, _stream())
    if rc:
        cabi.check(rc, "metis_nvfp4_quantize_dual")
    LAUNCHES["quantize"] += 2
    q = NVFP4Tensor(codes, scales, unit, (rows, cols), sf_layout)
    qt = NVFP4Tensor(codes_t, scales_t, unit_t, (cols, rows), sf_layout)
    if mean is not None:
        q.row_vec = mean
        qt.col_vec = mean
    qt.token_sums = sums
    if defer is None:
        return q, qt

    def finish():
        with _on_device(dev):
            # the buffers were allocated on the quantizing call's stream and are now also used on this one
            cur = torch._C._cuda_getCurrentStream(dev.index)
            rc2, = host.quantize_dual_finish(rows, cols, deferred, sf_layout, scales, unit, codes_t, scales_t, unit_t, sums, ws, _stream(), *cur)
        if rc2:
            cabi.check(rc2, "metis_nvfp4_quantize_dual_finish")
        LAUNCHES["quantize"] += 1
    return q, qt, finish


def rmsnorm_nvfp4_quantize(x: torch.Tensor, gamma: torch.Tensor, eps: float = 1e-6, *,
                           sf_layout: int = cabi.SF_MMA, return_norm: bool = False):
    """Fused RMSNorm -> NVFP4 quantization of x viewed as [rows, cols] (llama.py:23-31 then
    quant.py:6-36).  Returns the NVFP4Tensor, and the normalised tensor too if asked."""
    _need_cuda(x, "x")
    _need_cuda(gamma, "gamma")
    x2 = _rows2d(x)
    rows, cols = x2.shape
    if cols % 16 != 0 or rows == 0:
        raise ValueError(f"NVFP4 block shape (1, 16) does not divide tensor shape {(rows, cols)}")
    gamma = gamma.contiguous()
    assert gamma.numel() == cols
    dtype, gamma_dtype = _dtype_code(x2, "x"), _dtype_code(gamma, "gamma")
    norm_dtype = -1
    if return_norm:
        norm_dtype = cabi.DTYPE_BF16 if dtype == gamma_dtype == cabi.DTYPE_BF16 else cabi.DTYPE_F32
    with _on_device(x2.device):
        rc, codes, scales, unit, norm = cabi.host().rmsnorm_quantize(x2, dtype, gamma, gamma_dtype, float(eps), sf_layout, _sf_bytes(rows, cols, sf_layout),
                                                                     cabi.QUANTIZE_EXTRA_WORKSPACE, norm_dtype, _stream())
    if rc:
        cabi.check(rc, "metis_rmsnorm_nvfp4_quantize")
    LAUNCHES["rmsnorm_quantize"] += 2
    q = NVFP4Tensor(codes, scales, unit, (rows, cols), sf_layout)
    return (q, norm.reshape(x.shape)) if return_norm else q


def rmsnorm_mean(x: torch.Tensor, gamma: torch.Tensor, eps: float = 1e-6, *, want_rstd: bool = True):
    """RMSNorm of x viewed as [rows, cols] with the column mean of its output from the same pass:
    (y shaped like x, mean fp32 [cols], rstd fp32 [rows] or None).  First pass of the mean-centred
    activation path; nvfp4_quantize[_dual](y, mean=mean) is the second."""
    _need_cuda(x, "x")
    _need_cuda(gamma, "gamma")
    x2 = _rows2d(x)
    rows, cols = x2.shape
    if cols % 16 != 0 or rows == 0:
        raise ValueError(f"NVFP4 block shape (1, 16) does not divide tensor shape {(rows, cols)}")
    gamma = gamma.contiguous()
    assert gamma.numel() == cols
    L = cabi.lib()
    dev = x2.device
    with _on_device(dev):
        out_dtype = torch.bfloat16 if (x2.dtype == torch.bfloat16 and gamma.dtype == torch.bfloat16) else torch.float32
        y = torch.empty((rows, cols), dtype=out_dtype, device=dev)
        mean = torch.empty(cols, dtype=torch.float32, device=dev)
        rstd = torch.empty(rows, dtype=torch.float32, device=dev) if want_rstd else None
        ws = torch.empty(max(16, L.metis_rmsnorm_mean_workspace_bytes(rows, cols)), dtype=torch.uint8, device=dev)
        rc = L.metis_rmsnorm_mean(x2.data_ptr(), _dtype_code(x2, "x"), rows, cols, x2.stride(0), gamma.data_ptr(),
                                  _dtype_code(gamma, "gamma"), float(eps), y.data_ptr(), _ptr(rstd), mean.data_ptr(),
                                  ws.data_ptr(), ws.numel(), _stream())
    cabi.check(rc, "metis_rmsnorm_mean")
    LAUNCHES["rmsnorm_quantize"] += 2
    return y.reshape(x.shape), mean, rstd


def nvfp4_dequantize(q: NVFP4Tensor, dtype: torch.dtype = torch.float32, add_mean: bool = True,
                     unit: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Dense [R, C] tensor of q.  `unit` (fp32 [1], device) replaces q's own unit, e.g. to express the
    values in another product's accumulator units."""
    R, Cc = q.shape
    L = cabi.lib()
    with _on_device(q.device):
        out = torch.empty((R, Cc), dtype=dtype, device=q.device)
        rv = q.row_vec if add_mean else None
        rc = L.metis_nvfp4_dequantize(q.codes.data_ptr(), q.scales.data_ptr(), (q.unit if unit is None else unit).data_ptr(), q.sf_layout, R, Cc,
                                      _ptr(rv), out.data_ptr(), _DTYPES[dtype], out.stride(0), _stream())
    cabi.check(rc, "metis_nvfp4_dequantize")
    LAUNCHES["dequantize"] += 1
    if add_mean and q.col_vec is not None:
        out += q.col_vec.to(dtype)[:, None]
    return out


def _unit_ptr(unit: torch.Tensor, dev: torch.device) -> int:
    if unit.dtype != torch.float32 or unit.numel() != 1 or unit.device != dev:
        raise ValueError(f"a unit is one fp32 value on {dev}, not {unit.numel()} of {unit.dtype} on {unit.device}")
    return unit.data_ptr()


def nvfp4_dequantize_ratio(q: NVFP4Tensor, dtype: torch.dtype, unit0, unit1, over0, over1) -> torch.Tensor:
    """Dense [R, C] tensor of q with (unit0 * unit1) / (over0 * over1) in place of its unit (device fp32 [1] each); the
    mean vectors of q are left out."""
    R, Cc = q.shape
    units = [_unit_ptr(t, q.device) for t in (unit0, unit1, over0, over1)]
    with _on_device(q.device):
        out = torch.empty((R, Cc), dtype=dtype, device=q.device)
        rc = cabi.lib().metis_nvfp4_dequantize_ratio(q.codes.data_ptr(), q.scales.data_ptr(), *units, q.sf_layout, R, Cc,
                                                     out.data_ptr(), _DTYPES[dtype], out.stride(0), _stream())
    cabi.check(rc, "metis_nvfp4_dequantize_ratio")
    LAUNCHES["dequantize"] += 1
    return out


def nvfp4_gemv(q: NVFP4Tensor, v: Optional[torch.Tensor] = None) -> torch.Tensor:
    """out[r] = sum_c v[c] * value(q)[r, c] (v None: row sums), fp32; the mean vectors of q are ignored."""
    R, Cc = q.shape
    if v is not None:
        if v.dim() != 1 or v.dtype != torch.float32 or not v.is_contiguous():
            v = v.reshape(-1).to(torch.float32).contiguous()
        assert v.numel() == Cc
    with _on_device(q.device):
        rc, out = cabi.host().gemv(q.codes, q.scales, q.unit, q.sf_layout, R, Cc, v, _stream())
    if rc:
        cabi.check(rc, "metis_nvfp4_gemv")
    LAUNCHES["gemv"] += 1
    return out


def lowrank_scale(yv: torch.Tensor, s: torch.Tensor, unit_a: torch.Tensor, unit_b: torch.Tensor) -> torch.Tensor:
    """bf16( (yv * s).float() / (unit_a * unit_b) ) for bf16 yv [M, r]: torch.mul(self.s, y) of the
    low-rank branch, in the accumulator units of the GEMM whose side product it feeds (one kernel)."""
    _need_cuda(yv, "yv")
    if yv.dtype != torch.bfloat16 or yv.dim() != 2 or yv.stride(1) != 1:
        raise TypeError("yv must be a bf16 matrix with contiguous rows")
    if s.dtype not in (torch.bfloat16, torch.float32):
        s = s.float()
    s = s.reshape(-1).contiguous()
    M, r = yv.shape
    assert s.numel() == r and s.device == yv.device
    with _on_device(yv.device):
        rc, out = cabi.host().lowrank_scale(yv, s, _dtype_code(s, "s"), unit_a, unit_b, _stream())
    if rc:
        cabi.check(rc, "metis_lowrank_scale")
    LAUNCHES["gemv"] += 1
    return out


def lowrank_factors(yv: torch.Tensor, s: torch.Tensor, unit_a: torch.Tensor, unit_b: torch.Tensor, u: torch.Tensor, parts: int):
    """(yv * s) / (unit_a * unit_b) [M, r] and u [N, r] as bf16 operands of the side product, for fp32 yv and u: rounded (parts = 1)
    or split into head and tail (parts = 3: [Th Tl Th] and [Uh Uh Ul], [M, 3r] and [N, 3r])."""
    _need_cuda(yv, "yv")
    _need_cuda(u, "u")
    for name, t in (("yv", yv), ("u", u)):
        if t.dtype != torch.float32 or t.dim() != 2 or t.stride(1) != 1 or (t.shape[0] > 1 and t.stride(0) < t.shape[1]):
            raise TypeError(f"{name} must be an fp32 matrix with contiguous rows")
    if s.dtype not in (torch.bfloat16, torch.float32):
        s = s.float()
    s = s.reshape(-1).contiguous()
    assert s.numel() == yv.shape[1] == u.shape[1] and s.device == yv.device == u.device
    _unit_ptr(unit_a, yv.device)
    _unit_ptr(unit_b, yv.device)
    with _on_device(yv.device):
        rc, t, u_out = cabi.host().lowrank_factors(yv, s, _dtype_code(s, "s"), unit_a, unit_b, u, parts, _stream())
    if rc:
        cabi.check(rc, "metis_lowrank_factors")
    LAUNCHES["gemv"] += 1
    return t, u_out


def _fp32_vector(t: torch.Tensor, n: int) -> torch.Tensor:
    if t.dim() != 1 or t.dtype != torch.float32 or not t.is_contiguous():
        t = t.reshape(-1).to(torch.float32).contiguous()
    assert t.numel() == n and t.is_cuda
    return t


def nvfp4_gemm(a: NVFP4Tensor, b: NVFP4Tensor, *, lowrank=None, rank1=(), c: Optional[torch.Tensor] = None,
               out_dtype: torch.dtype = torch.bfloat16, alpha: float = 1.0,
               status: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
               sm_limit: int = 0, scaled=None, rows_ready: Optional["torch.cuda.Event"] = None, _debug: int = 0):
    """D = alpha*ua*ub * (A @ B^T + T @ U^T) + sum_i cvec_i (x) rvec_i (+ c), see metis_nvfp4_gemm.

    a: [M, K], b: [N, K] (both METIS_SF_MMA).  lowrank = (T [M, r] bf16, U [N, r] bf16), already in
    accumulator units.  rank1 = up to two (cvec or None, rvec) pairs of fp32 vectors.
    Only the packed parts of a and b enter the product; their mean vectors do not.
    sm_limit > 0 caps the SMs this launch occupies (room for a collective's kernel beside it).
    scaled = (s, unit_a, unit_b), for a bf16 D: returns (D, lowrank_scale(D, s, unit_a, unit_b)); the second value costs
    no launch of its own where the product is split along K.
    rows_ready: an event recorded on another stream behind the launches that write the row vectors of rank1; the product's
    stream waits for it as late as it can (a product split along K only in front of the launch that adds its splits)."""
    M, K = a.shape
    N, K2 = b.shape
    if K != K2:
        raise ValueError(f"inner dimensions differ: {K} vs {K2}")
    if a.sf_layout != cabi.SF_MMA or b.sf_layout != cabi.SF_MMA:
        raise ValueError("GEMM operands need METIS_SF_MMA scales")
    dev = a.device
    T = U = None
    if lowrank is not None:
        T, U = lowrank
        if T.dtype != torch.bfloat16 or U.dtype != torch.bfloat16:
            raise TypeError("low-rank factors must be bfloat16")
        T, U = _rows2d(T), _rows2d(U)
        if T.shape[0] != M or U.shape[0] != N or T.shape[1] != U.shape[1]:
            raise ValueError(f"low-rank shapes {tuple(T.shape)} / {tuple(U.shape)} do not fit [{M}, r] / [{N}, r]")
    if len(rank1) > 2:
        raise ValueError("at most two rank-1 terms")
    vectors = [None, None, None, None]                    # cvec0, rvec0, cvec1, rvec1
    for i, (cv, rv) in enumerate(rank1):
        vectors[2 * i + 1] = _fp32_vector(rv, N)
        if cv is not None:
            vectors[2 * i] = _fp32_vector(cv, M)
    if out is not None:
        assert out.shape == (M, N) and out.dtype == out_dtype and out.stride(1) == 1
    if c is not None:
        assert c.shape == (M, N) and c.dtype == out_dtype and c.stride(1) == 1 and c.is_cuda
    s = unit_a = unit_b = None
    s_dtype = 0
    if scaled is not None:
        s, unit_a, unit_b = scaled
        if s.dtype not in (torch.bfloat16, torch.float32):
            s = s.float()
        s = s.reshape(-1).contiguous()
        assert s.numel() == N and s.device == dev
        s_dtype = _dtype_code(s, "s")
        _unit_ptr(unit_a, dev)
        _unit_ptr(unit_b, dev)
    with _on_device(dev):
        rc, out, t, ws_bytes = cabi.host().gemm(M, N, K, float(alpha), a.codes, a.scales, a.unit, b.codes, b.scales, b.unit, T, U, *vectors, c, out,
                                                _DTYPES[out_dtype], int(_debug), int(sm_limit), status, 0 if rows_ready is None else rows_ready.cuda_event,
                                                s, s_dtype, unit_a, unit_b, _stream())
    if rc:
        cabi.check(rc, "metis_nvfp4_gemm")
    LAUNCHES["gemm"] += 2 if ws_bytes > 0 or scaled is not None else 1       # the sum of the splits, or the scaling
    return out if scaled is None else (out, t)


def _bf16_rows(t: torch.Tensor, what: str) -> torch.Tensor:
    _need_cuda(t, what)
    if t.dtype != torch.bfloat16 or t.dim() != 2:
        raise TypeError(f"{what} must be a bf16 matrix")
    if t.stride(1) != 1 or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


def bf16_panel_gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn_major: bool = False, b_mn_major: bool = False,
                    status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """D = A_op B_op^T in bf16 on the tensor core, fp32 out, at most 256 columns.  a is [Mg, Kg], or
    [Kg, Mg] with a_mn_major; b is [Ng, Kg], or [Kg, Ng] with b_mn_major."""
    a, b = _bf16_rows(a, "a"), _bf16_rows(b, "b")
    Mg, Kg = (a.shape[1], a.shape[0]) if a_mn_major else a.shape
    Ng, Kb = (b.shape[1], b.shape[0]) if b_mn_major else b.shape
    if Kg != Kb:
        raise ValueError(f"inner dimensions differ: {Kg} vs {Kb}")
    L = cabi.lib()
    with _on_device(a.device):
        out = torch.empty((Mg, Ng), dtype=torch.float32, device=a.device)
        ws = torch.empty(max(16, L.metis_bf16_panel_gemm_workspace_bytes(Mg, Ng, Kg)), dtype=torch.uint8, device=a.device)
        rc = L.metis_bf16_panel_gemm(a.data_ptr(), int(a_mn_major), a.stride(0), b.data_ptr(), int(b_mn_major), b.stride(0),
                                     Mg, Ng, Kg, out.data_ptr(), out.stride(0), ws.data_ptr(), ws.numel(), _ptr(status), _stream())
    cabi.check(rc, "metis_bf16_panel_gemm")
    LAUNCHES["lowrank_bwd"] += 2
    return out


def lowrank_dts(g: torch.Tensor, u: torch.Tensor, yv: torch.Tensor, s: torch.Tensor, status: Optional[torch.Tensor] = None,
                *, ds_dtype: torch.dtype = torch.float32, want_mean: bool = False):
    """(d_yv, ds) of the low-rank branch from one pass over g [M, N]: d_ts = bf16(g @ u), d_yv = bf16(d_ts * s),
    ds = sum over rows of bf16(d_ts * yv), summed in fp32 and returned in ds_dtype.  u [N, r], yv [M, r] bf16; s [r]
    bf16 or fp32.  want_mean: a third value, the column mean of d_yv (fp32 [r])."""
    g, u, yv = _bf16_rows(g, "g"), _bf16_rows(u, "u"), _bf16_rows(yv, "yv")
    M, N = g.shape
    r = u.shape[1]
    if u.shape[0] != N or yv.shape != (M, r) or s.numel() != r:
        raise ValueError(f"shapes do not fit: g {tuple(g.shape)}, u {tuple(u.shape)}, yv {tuple(yv.shape)}, s {tuple(s.shape)}")
    if s.dtype not in (torch.bfloat16, torch.float32):
        s = s.float()
    s = s.reshape(-1).contiguous()
    L = cabi.lib()
    with _on_device(g.device):
        d_yv = torch.empty((M, r), dtype=torch.bfloat16, device=g.device)
        ds = torch.empty(r, dtype=ds_dtype, device=g.device)
        mean = torch.empty(r, dtype=torch.float32, device=g.device) if want_mean else None
        ws = torch.empty(L.metis_lowrank_dts_workspace_bytes(M, N, r), dtype=torch.uint8, device=g.device)
        rc = L.metis_lowrank_dts_mean(g.data_ptr(), g.stride(0), M, N, u.data_ptr(), u.stride(0), r, yv.data_ptr(), yv.stride(0),
                                      s.data_ptr(), _dtype_code(s, "s"), d_yv.data_ptr(), d_yv.stride(0), ds.data_ptr(),
                                      _DTYPES[ds_dtype], _ptr(mean), ws.data_ptr(), ws.numel(), _ptr(status), _stream())
    cabi.check(rc, "metis_lowrank_dts_mean")
    # the product, the sum of its splits where it has more than one, the sums over the CTAs
    one_split = M * ((r + 63) // 64 * 64) * 4
    LAUNCHES["lowrank_bwd"] += 2 if L.metis_bf16_panel_gemm_workspace_bytes(M, r, N) == one_split else 3
    return (d_yv, ds, mean) if want_mean else (d_yv, ds)


def lowrank_du(g: torch.Tensor, ts: torch.Tensor, out_dtype: torch.dtype = torch.bfloat16,
               status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """dU = g^T @ ts [N, r] for g [M, N] and ts [M, r] (bf16), one pass over g, no transposed copies."""
    g, ts = _bf16_rows(g, "g"), _bf16_rows(ts, "ts")
    M, N = g.shape
    r = ts.shape[1]
    if ts.shape[0] != M:
        raise ValueError(f"shapes do not fit: g {tuple(g.shape)}, ts {tuple(ts.shape)}")
    L = cabi.lib()
    with _on_device(g.device):
        out = torch.empty((N, r), dtype=out_dtype, device=g.device)
        ws = torch.empty(L.metis_lowrank_du_workspace_bytes(M, N, r), dtype=torch.uint8, device=g.device)
        rc = L.metis_lowrank_du(g.data_ptr(), g.stride(0), M, N, ts.data_ptr(), ts.stride(0), r, out.data_ptr(), _DTYPES[out_dtype],
                                out.stride(0), ws.data_ptr(), ws.numel(), _ptr(status), _stream())
    cabi.check(rc, "metis_lowrank_du")
    LAUNCHES["lowrank_bwd"] += 2
    return out


def _same_device(first: torch.Tensor, **others) -> None:
    for name, t in others.items():
        if t.device != first.device:
            raise ValueError(f"{name} is on {t.device}, not on {first.device}")


def _dense(t: torch.Tensor, alignment: int) -> torch.Tensor:
    """t with contiguous elements on an aligned address (copied only if it has to be)."""
    t = t.contiguous()
    return t if t.data_ptr() % alignment == 0 else t.clone()


def rope_pair(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """Rotary embedding (rotate-half convention) of q [B, T, Hq, D] and k [B, T, Hk, D], bf16 and contiguous, in one
    launch, with every rounding of `x * cos + cat(-x2, x1) * sin` on bf16 tensors.  cos, sin: bf16, T rows of D elements
    (any leading ones).  Returns tensors shaped like q and k.  No autograd."""
    for name, t in (("q", q), ("k", k), ("cos", cos), ("sin", sin)):
        _need_cuda(t, name)
        if t.dtype != torch.bfloat16:
            raise TypeError(f"{name} must be bfloat16")
    B, T, Hq, D = q.shape
    Hk = k.shape[2]
    if k.shape != (B, T, Hk, D) or cos.numel() != T * D or sin.numel() != T * D:
        raise ValueError(f"shapes do not fit: q {tuple(q.shape)}, k {tuple(k.shape)}, cos {tuple(cos.shape)}, sin {tuple(sin.shape)}")
    _same_device(q, k=k, cos=cos, sin=sin)
    q, k, cos, sin = (_dense(t, 8) for t in (q, k, cos, sin))
    with _on_device(q.device):
        qo, ko = torch.empty_like(q), torch.empty_like(k)
        rc = cabi.lib().metis_rope_pair(q.data_ptr(), k.data_ptr(), cos.data_ptr(), sin.data_ptr(), qo.data_ptr(), ko.data_ptr(),
                                        B * T, T, Hq, Hk, D, _stream())
    cabi.check(rc, "metis_rope_pair")
    LAUNCHES["decoder"] += 1
    return qo, ko


def silu_mul(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """silu(gate) * up for bf16 tensors of one shape, with the rounding of silu's output, in one launch.  No autograd."""
    _need_cuda(gate, "gate")
    _need_cuda(up, "up")
    if gate.dtype != torch.bfloat16 or up.dtype != torch.bfloat16 or gate.shape != up.shape:
        raise TypeError("gate and up must be bfloat16 tensors of one shape")
    _same_device(gate, up=up)
    gate, up = _dense(gate, 16), _dense(up, 16)
    with _on_device(gate.device):
        out = torch.empty_like(gate)
        rc = cabi.lib().metis_silu_mul(gate.data_ptr(), up.data_ptr(), out.data_ptr(), gate.numel(), _stream())
    cabi.check(rc, "metis_silu_mul")
    LAUNCHES["decoder"] += 1
    return out
