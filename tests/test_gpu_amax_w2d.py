"""amax kernels and the weight quantizer at the edges of their work split: tensors shorter than one block's loads, around
one and several rounds of the rolling loads, and weights of one tile, of several tiles per CTA and of no whole tile."""
import numpy as np
import pytest
import torch

from oracle import nvfp4_oracle as O
from tests.gpu_util import make_w, to_dev, u8

pytestmark = pytest.mark.gpu

BLOCK, GRID = 256 * 4, 148 * 4          # loads of a block per round, most blocks


@pytest.mark.parametrize("loads", [1, 3, BLOCK - 1, BLOCK, BLOCK + 1, GRID * BLOCK - 1, GRID * BLOCK + 5, 3 * GRID * BLOCK + 7])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_amax_finds_the_largest_wherever_it_is(loads, dtype):
    from nvfp4_training_b200 import fp4ops
    per = 16 // torch.empty(0, dtype=dtype).element_size()
    n = loads * per
    x = torch.rand(n, device="cuda").to(dtype)
    for pos in (0, n // 2, n - 1):
        x[pos] = -3.5
        for _ in range(2):               # the meeting point of the blocks is clean again
            assert fp4ops.amax_of(x).item() == 3.5
        x[pos] = 0.25
    assert fp4ops.amax_of(torch.zeros_like(x)).item() == 0


def test_amax_words_outlive_their_consumers_on_several_streams():
    """quant_rows without an amax takes the library's passing words: many calls in flight on two streams, and one from
    another thread, give what a given amax gives."""
    import threading
    from nvfp4_training_b200 import nvq
    xs = [torch.randn(128, 256, device="cuda").bfloat16() * (k + 1) for k in range(24)]
    want = [nvq.quant_rows(x, am=x.abs().amax().float().reshape(1)) for x in xs]
    got = {}

    def work(tag, stream):
        with torch.cuda.stream(stream):
            got[tag] = [nvq.quant_rows(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for s in streams:
        work(s, s)
    t = threading.Thread(target=work, args=("thread", streams[0]))
    t.start()
    t.join()
    torch.cuda.synchronize()
    for qs in got.values():
        for a, b in zip(qs, want):
            assert torch.equal(a.gs, b.gs) and np.array_equal(u8(a.d), u8(b.d)) and np.array_equal(u8(a.s), u8(b.s))


@pytest.mark.parametrize("N,K", [(128, 128), (384, 256), (16, 48), (144, 208), (5120, 4096)])
def test_w2d_fp32_writes_both_scale_layouts(N, K):
    from nvfp4_training_b200 import fp4ops
    rng = np.random.default_rng(N + K)
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    w[:16, :16] = 0                      # a block of zeros
    q, qt = fp4ops.quant_w2d(torch.from_numpy(w).cuda())
    if N * K < 1 << 20:
        codes, scales, codes_t, scales_t, _ = O.quant_w2d(w)
        assert np.array_equal(u8(q.d), codes) and np.array_equal(u8(q.s), scales)
        assert np.array_equal(u8(qt.d), codes_t) and np.array_equal(u8(qt.s), scales_t)
    assert torch.equal(fp4ops.dequant(qt), fp4ops.dequant(q).t())
    whole = N % 128 == 0 and K % 128 == 0
    for p in (q, qt):
        assert (p.sw is not None) == whole
        if whole:
            assert torch.equal(p.sw, fp4ops.swizzle_scales(p.s))


@pytest.mark.parametrize("M,C", [(128, 128), (256, 384)])
def test_fp4ops_quantizers_write_both_scale_layouts(M, C):
    from nvfp4_training_b200 import fp4ops
    x = torch.randn(M, C, device="cuda").bfloat16()
    for q in (fp4ops.quant_rows(x), fp4ops.quant_cols_rht(x, 0xA6B1), *fp4ops.quant_rows_cols_rht(x, 0xA6B1)):
        assert torch.equal(q.sw, fp4ops.swizzle_scales(q.s))
        q.s.add_(1)                      # changed in place: the swizzled copy is no longer used
        assert q.swizzled() is None


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("N,K", [(128, 256), (384, 128), (16, 16), (48, 64), (80, 48), (1008, 208)])
def test_w2d_kernels_agree_in_every_layout(N, K, dtype):
    """Codes off their 16-byte boundaries take the kernel for any shape: the bits the oracle has, whole tiles in all three
    scale layouts, other shapes row-major; each operand also by itself."""
    from nvfp4_training_b200 import _lib as L
    lib = L.load()
    w = make_w(N * K, N, K)
    wd = to_dev(w) if dtype == "bf16" else torch.from_numpy(w).cuda()
    am = wd.abs().amax().float().reshape(1)
    codes, scales, codes_t, scales_t, _ = O.quant_w2d(w)
    whole = N % 128 == 0 and K % 128 == 0
    for layout in (L.SCALES_SWIZZLED, L.SCALES_LINEAR, L.SCALES_BOTH) if whole else (L.SCALES_LINEAR,):
        for want in ((True, True), (True, False), (False, True)):
            for off in (0, 4):
                bufs = [torch.zeros(N * K // d * m + 16, dtype=torch.uint8, device="cuda") for d, m in ((2, 1), (16, 2), (2, 1), (16, 2))]
                ptrs = [b.data_ptr() + off if want[i // 2] else None for i, b in enumerate(bufs)]
                assert lib.nvfp4_quant_w2d(wd.data_ptr(), L.DTYPE_BF16 if dtype == "bf16" else L.DTYPE_FP32, N, K, *ptrs, layout,
                                           am.data_ptr(), None, L.stream()) == 0
                for i, (d, s, R, C) in enumerate(((codes, scales, N, K), (codes_t, scales_t, K, N))):
                    q, sc = u8(bufs[2 * i]), u8(bufs[2 * i + 1])
                    n, m = (R * C // 2, R * C // 16) if want[i] else (0, 0)
                    assert np.array_equal(q[off:off + n].reshape(-1), np.asarray(d).reshape(-1)[:n]) and not q[off + n:].any()
                    if layout != L.SCALES_SWIZZLED:
                        assert np.array_equal(sc[off:off + m], np.asarray(s).reshape(-1)[:m])
                    if layout != L.SCALES_LINEAR and m:
                        at = off + (m if layout == L.SCALES_BOTH else 0)
                        assert np.array_equal(O.unswizzle_scales(sc[at:at + m], R, C // 16), s)
                    assert not sc[off + m * (2 if layout == L.SCALES_BOTH else 1):].any()
