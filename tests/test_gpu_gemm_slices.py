"""Few output tiles: K sliced over the CTAs of a cluster, and the caller's slice count as an upper bound."""
import pytest
import torch

from tests.gpu_util import make_w, make_x, to_dev

pytestmark = pytest.mark.gpu


# slices taken on 148 SMs: none, 2, 4, 8; uneven ones; a last K tile of 64 and of 192; the widest call that is sliced
@pytest.mark.parametrize("M,N,K", [(128, 128, 1472), (128, 9472, 3072), (256, 2048, 5632), (384, 1152, 2304), (128, 128, 4160),
                                   (128, 256, 4032), (2048, 128, 2112), (128, 4096, 8192)])
def test_few_tile_gemms(M, N, K):
    from nvfp4_training_b200 import _lib as L, emit, nvq
    L.load().nvfp4_gemm_force_tile_n(0)
    qa, qb = nvq.quant_rows(to_dev(make_x(M + K, M, K))), nvq.quant_rows(to_dev(make_w(N + K, N, K)))
    y = nvq.dequant(qa).double() @ nvq.dequant(qb).double().t()
    scale = y.abs().max()

    def close(c, want, rel, step):
        err = (c.double() - want).abs()
        assert (c.double() - want).norm() <= rel * want.norm()
        assert bool((err <= step * want.abs() + 1e-6 * scale).all())
    close(nvq.mm(qa, qb), y, 4e-3, 2 ** -8)
    close(nvq.mm(qa, qb, out_dtype=torch.float32), y, 1e-5, 1e-4)
    close(nvq.mm(qa, qb, out_dtype=torch.float32, splitk=0), y, 1e-5, 1e-4)
    wide = torch.full((M, N + 8), 3.0, device="cuda")              # a strided C, added to; its padding stays
    nvq.mm(qa, qb, out_dtype=torch.float32, out=wide[:, :N], accumulate=True, splitk=0)
    assert (wide[:, :N].double() - 3.0 - y).norm() <= 1e-5 * (y + 3.0).norm()
    assert bool((wide[:, N:] == 3.0).all())
    nvq.mm(qa, qb, out_dtype=torch.float32, out=wide[:, 4:N + 4])  # rows on 16-byte, not 32-byte, boundaries
    close(wide[:, 4:N + 4], y, 1e-5, 1e-4)
    half = torch.full((M, N + 8), 3.0, dtype=torch.bfloat16, device="cuda")
    nvq.mm(qa, qb, out=half[:, :N])
    close(half[:, :N], y, 4e-3, 2 ** -8)
    assert bool((half[:, N:] == 3.0).all()) and bool((wide[:, N + 4:] == 3.0).all())
    rs = torch.rand(M, device="cuda") + 0.5                        # a scale per row
    out = emit._gemm(qa.d, qa.s, qb.d, qb.s, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), L.ALPHA_ROW, rs, qb.gs)
    want = y * (rs / qa.gs).double()[:, None]
    assert (out.double() - want).norm() <= 4e-3 * want.norm()
    L.check_status()


# by pairs and clusters; atomic slices of one-CTA tiles, more than K has tiles for; of CTA pairs; uneven ones
@pytest.mark.parametrize("M,N,K", [(128, 512, 4096), (3072, 1024, 2048), (1024, 1024, 16384), (128, 128, 16384), (128, 128, 4480), (512, 512, 16384),
                                   (640, 640, 16384), (384, 384, 32640)])
@pytest.mark.parametrize("splitk", [2, 8, 16, 64])
def test_requested_slices_add_into_c(M, N, K, splitk):
    """However many slices the library takes, the product is added once to what C holds."""
    from nvfp4_training_b200 import _lib as L, fp4ops
    L.load().nvfp4_gemm_force_tile_n(0)
    a, b = fp4ops.quant_rows(to_dev(make_x(3, M, K, outliers=0))), fp4ops.quant_rows(to_dev(make_x(4, N, K, outliers=0)))
    y = fp4ops.dequant(a).double() @ fp4ops.dequant(b).double().t()
    out = torch.full((M, N), 2.0, device="cuda")
    fp4ops.gemm(a, b, out=out, splitk=splitk)
    fresh = fp4ops.gemm(a, b, splitk=splitk)
    assert fresh.dtype == torch.float32
    for got, want in ((out, y + 2), (fresh, y)):
        assert float((got.double() - want).norm() / want.norm()) <= 1e-5
    L.check_status()


@pytest.mark.parametrize("K", [64, 256])
def test_slices_of_a_single_k_tile_store(K):
    """K of one tile has one slice whatever the caller asks for: without `accumulate` it is stored, not added."""
    from nvfp4_training_b200 import _lib as L, nvq
    a, b = nvq.quant_rows(to_dev(make_x(5, 256, K))), nvq.quant_rows(to_dev(make_w(6, 384, K)))
    want = nvq.mm(a, b, out_dtype=torch.float32)
    out = torch.full((256, 384), 7.0, device="cuda")
    assert torch.equal(nvq.mm(a, b, out_dtype=torch.float32, out=out, splitk=4), want)
    out.fill_(7.0)
    nvq.mm(a, b, out_dtype=torch.float32, out=out, splitk=4, accumulate=True)
    assert float((out - 7 - want).abs().max()) <= 2 ** -22 * float(want.abs().max() + 7)      # the sum and the difference round
    # an empty contraction leaves zeros
    out.fill_(7.0)
    p = out.data_ptr()
    assert L.load().nvfp4_gemm(p, p, 16, p, p, 16, p, L.DTYPE_FP32, 384, 256, 384, 0, L.ALPHA_ONE, None, None, 1.0, 1.0, 0, 4, None, L.stream()) == 0
    assert not out.any()


@pytest.mark.parametrize("M,N,K", [(128, 128, 256), (256, 384, 4096), (2048, 1024, 8192)])
def test_slices_of_a_fresh_result(M, N, K):
    """`nvq.mm` without `out` gives the product, whatever the memory of its result held before."""
    from nvfp4_training_b200 import nvq
    a, b = nvq.quant_rows(to_dev(make_x(7, M, K))), nvq.quant_rows(to_dev(make_w(8, N, K)))
    want = nvq.dequant(a).double() @ nvq.dequant(b).double().t()
    for splitk in (1, 4):
        junk = [torch.full((M, N), 1e6, device="cuda") for _ in range(4)]
        del junk
        got = nvq.mm(a, b, out_dtype=torch.float32, splitk=splitk)
        assert float((got.double() - want).norm() / want.norm()) <= 1e-5
