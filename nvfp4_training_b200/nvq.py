"""Drop-in for the reference's `nvq` module (llm-1b/nvq.py): NVFP4 quantizers with swizzled
E4M3 scales and the block-scaled FP4 GEMM, same names, arguments, tensor layouts and assertions,
running on the sm_100a C-ABI library instead of NVRTC kernels + cuBLASLt.

Differences a caller can observe, all inside the stated tolerances:
  * `gs` is `amax / 2688` by IEEE division (the order of small-model/model_ref.py:42), written by the
    quantizer kernel itself, instead of `amax * (1/2688)` (llm-1b/nvq.py:43-44); at most one ulp apart.
  * `mm` applies alpha = gsA*gsB in FP32 inside the GEMM epilogue before the output cast, instead of
    rounding alpha to bf16 and multiplying a bf16 product (llm-1b/nvq.py:96).
  * stochastic rounding defaults to the reference's mantissa-dither method and random stream;
    `SR_MODE` switches to the hardware `cvt.rs` path.
"""
import torch

from . import _lib as L

# rounding used when a quantizer is called with sr=True (a per-call `sr_mode` overrides it):
# ROUND_SR_DITHER = the reference's rounding and random stream, ROUND_SR_HW = hardware cvt.rs
SR_MODE = L.ROUND_SR_DITHER


class Q:
    """Packed NVFP4 matrix [R, C]: d [R, C/2] fp4x2, s swizzled e4m3 (flat), gs = per-tensor scale
    (device, fp32).  Same container as llm-1b/nvq.py:24-29."""
    __slots__ = ("d", "s", "gs")

    def __init__(self, d, s, gs):
        self.d, self.s, self.gs = d, s, gs


def _mode(sr, sr_mode):
    return (sr_mode or SR_MODE) if sr else L.ROUND_NEAREST


def amax(x, out=None, clear=True):
    """max|x| of a contiguous bf16 tensor as a device fp32 [1] (llm-1b/nvq.py:32-40).  `clear=False` (an addition):
    `out` is a word the caller has zeroed, e.g. one of a batch cleared with a single fill, and is only raised."""
    return (L._host or L.host()).amax(x, out, clear)


def quant_rows(x, sr=False, seed=0, am=None, sr_mode=None):
    """x [R, C] bf16 (row-contiguous) -> Q quantized along C (llm-1b/nvq.py:47-57)."""
    return Q(*(L._host or L.host()).quant_rows(x, _mode(sr, sr_mode), seed, am))


def quant_cols_rht(x, signs, sr=False, seed=0, am=None, sr_mode=None):
    """x [M, C] -> Q of x^T [C, M] quantized along M, after a 16-pt RHT along M (llm-1b/nvq.py:60-70)."""
    return Q(*(L._host or L.host()).quant_cols_rht(x, signs & 0xFFFF, _mode(sr, sr_mode), seed, am))


def quant_rows_cols_rht(x, signs, sr=False, seed=0, seed_cols=0, am=None, sr_mode=None, want=(True, True)):
    """x [M, C] bf16 -> (Q of x along C, Q of x^T along M after the 16-pt RHT): the results of
    `quant_rows(x, ...)` and `quant_cols_rht(x, signs, ...)` (llm-1b/nvq.py:47-70) from one pass
    over x.  `seed` rounds the row operand, `seed_cols` the transposed one; `want` skips an output."""
    r, c = (L._host or L.host()).quant_rows_cols_rht(x, signs & 0xFFFF, _mode(sr, sr_mode), seed, seed_cols, am, want[0], want[1])
    return (Q(*r) if r is not None else None, Q(*c) if c is not None else None)


def quant_tile_status(reset=True):
    """Status word of the tile quantizer on the current device (0 = no wait ever expired)."""
    import ctypes
    out = ctypes.c_int(0)
    L.check(L.load().nvfp4_quant_tile_status(ctypes.byref(out), 1 if reset else 0), "quant_tile_status")
    return out.value


def quant_w2d(w, am=None, want=(True, True), out=None):
    """w [N, K] bf16 -> (Q of w, Q of w^T), identical values (16x16 blocks) (llm-1b/nvq.py:73-87).
    `want` lets a caller skip one of the two outputs (its slot is then None); `out` = a pair
    returned by an earlier call, overwritten in place (a per-step weight cache keeps its buffers)."""
    h = L._host or L.host()
    if out is not None:
        oq, oqt = out
        d, s = (oq.d, oq.s) if oq is not None else (None, None)
        dt, st = (oqt.d, oqt.s) if oqt is not None else (None, None)
        h.quant_w2d_into(w, am, d, s, dt, st, (oq or oqt).gs)
        return out
    q, qt = h.quant_w2d(w, am, want[0], want[1])
    return (Q(*q) if q is not None else None, Q(*qt) if qt is not None else None)


def mm(a: Q, b: Q, out_dtype=torch.bfloat16, scale=True, out=None, accumulate=False, splitk=1, owners=None):
    """a [M,K], b [N,K] (both K-major) -> a @ b^T [M, N].  If scale=False returns (raw, alpha)
    (llm-1b/nvq.py:90-96).  `out` / `accumulate` (fp32 only) are additions for in-place wgrad; `splitk=0` (fp32 only)
    lets the library slice a long contraction over the SMs (sums then land in no fixed order).
    `owners` (fp32 `out` only): the addresses of `out` on every data-parallel rank (peer mappings; this rank's own
    `out.data_ptr()` at its index); the product is then added into the row slab each rank owns instead of into `out`
    (`nvfp4_gemm_scatter_rows`)."""
    assert out_dtype in (torch.bfloat16, torch.float32)
    fp32 = out_dtype == torch.float32
    if owners is not None:
        M, N, K = a.d.shape[0], b.d.shape[0], a.d.shape[1] * 2
        assert fp32 and b.d.shape[1] * 2 == K and out.shape == (M, N) and out.dtype == out_dtype and out.stride(1) == 1
        L.require_cuda(a.d, b.d)
        L.check(L.load().nvfp4_gemm_scatter_rows(L.ptr(a.d), L.ptr(a.s), a.d.stride(0), L.ptr(b.d), L.ptr(b.s), b.d.stride(0),
                                                 L.ptr_array(owners), len(owners), out.stride(0), M, N, K,
                                                 L.ALPHA_GS if scale else L.ALPHA_ONE, L.ptr(a.gs) if scale else None,
                                                 L.ptr(b.gs) if scale else None, 1.0, 1.0, splitk,
                                                 L.ptr(L.status_word(a.d.device)), L.stream()), "mm (scatter)")
        return out
    out = (L._host or L.host()).mm(a.d, a.s, a.gs, b.d, b.s, b.gs, fp32, scale, out, accumulate, splitk)
    return out if scale else (out, a.gs * b.gs)


# ---------- reference decode (tests), llm-1b/nvq.py:99-117
_E2M1 = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, -0., -.5, -1, -1.5, -2, -3, -4, -6])


def unswizzle(s, R, C16):
    ncb = C16 // 4
    t = s.view(torch.uint8).reshape(R // 128, ncb, 32, 4, 4)       # rb, cb, r%32, (r%128)/32, c%4
    return t.permute(0, 3, 2, 1, 4).reshape(R, C16)                 # rb,(r/32),(r%32), cb, c%4


def dequant(q: Q):
    d = q.d.view(torch.uint8)
    R, C = d.shape[0], d.shape[1] * 2
    lo, hi = (d & 15).long(), (d >> 4).long()
    tab = _E2M1.to(d.device)
    v = torch.stack([tab[lo], tab[hi]], -1).reshape(R, C)
    s = unswizzle(q.s, R, C // 16).view(torch.float8_e4m3fn).float().repeat_interleave(16, 1)
    return v * s * q.gs
