"""amax kernels and the weight quantizer at the edges of their work split: tensors shorter than one block's loads, around
one and several rounds of the rolling loads, and weights of one tile, of several tiles per CTA and of no whole tile."""
import numpy as np
import pytest
import torch

from oracle import nvfp4_oracle as O
from tests.gpu_util import u8

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
