"""The quantizer that finds a small tensor's amax itself: same bits as the amax kernel followed by the quantizer, from one
tile to its largest size, and where it has to decline."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from tests.gpu_util import u8

pytestmark = pytest.mark.gpu

SIGNS = 0xA6B1


def same(a, b):
    return all(np.array_equal(u8(p), u8(q)) for x, y in zip(a, b) for p, q in ((x.d, y.d), (x.s, y.s), (x.gs, y.gs)))


def launched(x):
    """Whether the library takes this tensor in one launch; its amax is then the amax kernel's."""
    from nvfp4_training_b200 import _lib as L, nvq
    M, C = x.shape
    out = [torch.empty(M * C // n, dtype=torch.uint8, device="cuda") for n in (2, 16)]
    am, flag = torch.empty(1, device="cuda"), ctypes.c_int(-1)
    L.check(L.load().nvfp4_quant_tile_amax(x.data_ptr(), x.stride(0), M, C, out[0].data_ptr(), out[1].data_ptr(), None, None, 0, am.data_ptr(),
                                           ctypes.byref(flag), None, None, SIGNS, 0, 0, 0, None, None, L.stream()), "quant_tile_amax")
    if flag.value and not torch.cuda.is_current_stream_capturing():
        assert torch.equal(am, nvq.amax(x.contiguous()))
    return bool(flag.value)


# 128 x 128 tiles, one per CTA of a cluster: of one CTA, of five, of eight; too many
@pytest.mark.parametrize("M,C,takes", [(128, 128, True), (640, 128, True), (256, 512, True), (128, 1024, True), (128, 1152, False),
                                       (1024, 1024, False)])
@pytest.mark.parametrize("mode", [0, 1, 3])
def test_same_bits_as_amax_then_quantize(M, C, takes, mode):
    from nvfp4_training_b200 import _lib as L, nvq
    x = torch.randn(M, C, device="cuda").bfloat16()
    for pos in ((0, 0), (M - 1, C - 1), (M // 2, C // 3)):
        x[pos] = -9.0 - pos[0] / M
        assert launched(x) == takes
        kw = dict(sr=mode != 0, seed=5, seed_cols=9, sr_mode=mode or None)
        got = nvq.quant_rows_cols_rht(x, SIGNS, **kw)
        assert same(got, nvq.quant_rows_cols_rht(x, SIGNS, am=x.abs().amax().float().reshape(1), **kw))
    L.check_status()


def test_strided_special_values_and_single_outputs():
    from nvfp4_training_b200 import _lib as L, nvq
    big = torch.randn(256, 640, device="cuda").bfloat16()
    big[:, 512:] = 100.0                                           # beyond the view: must not count
    x = big[:, :512]
    am = x.abs().amax().float().reshape(1)
    assert launched(x) and same(nvq.quant_rows_cols_rht(x, SIGNS), nvq.quant_rows_cols_rht(x, SIGNS, am=am))
    assert same([nvq.quant_cols_rht(x, SIGNS)], [nvq.quant_cols_rht(x, SIGNS, am=am)])
    for value in (0.0, float("inf"), float("nan"), -0.0, 3.3e38):
        x.fill_(0.0)
        x[77, 300] = value
        am = nvq.amax(x.contiguous())
        assert launched(x) and same(nvq.quant_rows_cols_rht(x, SIGNS), nvq.quant_rows_cols_rht(x, SIGNS, am=am))
    L.check_status()


def test_many_in_flight_on_several_streams_and_threads():
    from nvfp4_training_b200 import _lib as L, nvq
    xs = [torch.randn(256, 256 * (1 + k % 3), device="cuda").bfloat16() * (k + 1) for k in range(24)]
    want = [nvq.quant_rows_cols_rht(x, SIGNS, am=x.abs().amax().float().reshape(1)) for x in xs]
    got = {}

    def work(tag, stream):
        with torch.cuda.stream(stream):
            # the wider ones and quant_rows take an amax kernel
            got[tag] = [(nvq.quant_rows_cols_rht(x, SIGNS), nvq.quant_rows(x))[0] for x in xs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k, streams[k % 2])) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert len(got) == 4
    for qs in got.values():
        for a, b in zip(qs, want):
            assert same(a, b)
    L.check_status()


def test_captured():
    from nvfp4_training_b200 import nvq
    x = torch.randn(256, 512, device="cuda").bfloat16()
    want = nvq.quant_rows_cols_rht(x, SIGNS)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert launched(x)
        got = nvq.quant_rows_cols_rht(x, SIGNS)
    for _ in range(2):
        graph.replay()
    assert same(got, want)
