"""The general row and column quantizers at the edges of their CTA tiles (64 columns x 256 tokens; 32 blocks per warp)."""
import numpy as np
import pytest
import torch

from oracle import nvfp4_oracle as O
from tests.gpu_util import make_x, to_dev, u8

pytestmark = pytest.mark.gpu
SIGNS = 0xA6B1


# one block; a column tile's last 8 columns; 15, 16, 17 and 33 token blocks; scale rows of 4n, 4n + 1 .. bytes
@pytest.mark.parametrize("M,C", [(16, 16), (16, 8), (256, 64), (256, 72), (272, 56), (240, 1552), (528, 136), (2048, 24), (5008, 208)])
@pytest.mark.parametrize("mode", ["rn", "sr"])
def test_cols_rht_any_size(M, C, mode):
    from nvfp4_training_b200 import fp4ops
    x = make_x(M + C, M, C, outliers=0)
    x[-1, -1] = 40.0
    sr = dict(sr_mode=O.SR_DITHER_FP4K, seed=5) if mode == "sr" else {}
    codes, scales, _ = O.quant_cols_rht(x, SIGNS, **sr)
    q = fp4ops.quant_cols_rht(to_dev(x), SIGNS, sr=mode == "sr", seed=5)
    assert np.array_equal(u8(q.d), codes) and np.array_equal(u8(q.s), scales)


@pytest.mark.parametrize("R,C", [(1, 16), (3, 16), (31, 48), (33, 496), (64, 512), (5008, 1552)])
@pytest.mark.parametrize("mode", ["rn", "sr"])
def test_rows_any_size(R, C, mode):
    from nvfp4_training_b200 import fp4ops
    x = make_x(R + C, R, C, outliers=0)
    x[-1, -1] = 40.0
    shifted = torch.cat([torch.zeros(8, device="cuda", dtype=torch.bfloat16), to_dev(x).reshape(-1)])[8:].view(R, C)   # 16-byte aligned only
    sr = dict(sr_mode=O.SR_DITHER_FP4K, seed=5) if mode == "sr" else {}
    codes, scales, _ = O.quant_rows(x, **sr)
    for t in (to_dev(x), shifted):
        q = fp4ops.quant_rows(t, sr=mode == "sr", seed=5)
        assert np.array_equal(u8(q.d), codes) and np.array_equal(u8(q.s), scales)


@pytest.mark.parametrize("M,C", [(64, 128), (192, 640), (320, 128)])
def test_cols_rht_swizzled(M, C):
    from nvfp4_training_b200 import nvq
    x = make_x(M * C, M, C, outliers=0)
    codes, scales, _ = O.quant_cols_rht(x, SIGNS)
    q = nvq.quant_cols_rht(to_dev(x), SIGNS)                       # no whole 128-token tiles: the general kernel
    assert np.array_equal(u8(q.d), codes) and np.array_equal(O.unswizzle_scales(u8(q.s), C, M // 16), scales)
