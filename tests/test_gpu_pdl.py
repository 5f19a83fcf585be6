"""Programmatic dependent launch of short launches (the default): chains of dependent calls on reused memory give the bits
they give without it, eagerly and replayed as a graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# few tiles and slices of K; CTA pairs; the cluster that finds its amax; tensors on both sides of the 48 MB line
@pytest.mark.parametrize("T,K,N", [(128, 256, 384), (256, 5632, 2048), (3200, 1408, 2176), (8320, 2944, 384), (8832, 2944, 384)])
@pytest.mark.parametrize("mode", [1, 2])
def test_chains_give_the_same_bits(T, K, N, mode):
    from nvfp4_training_b200 import _lib as L, nvq
    lib = L.load()
    xs = [(torch.randn(T, K, device="cuda") * (k + 1)).bfloat16() for k in range(3)]
    ws = [(torch.randn(N, K, device="cuda") * 0.02 * (k + 1)).bfloat16() for k in range(3)]

    def chain():
        out = []
        for x, w in zip(xs, ws):
            q, qt = nvq.quant_w2d(w)
            r, c = nvq.quant_rows_cols_rht(x, 0xA6B1)
            y = nvq.mm(r, q)                                       # every call reads what the call before it wrote,
            g = nvq.quant_rows_cols_rht(y, 0xA6B1, sr=True, seed=3, seed_cols=4)
            out += [y, nvq.mm(g[0], qt), nvq.mm(g[1], c, out_dtype=torch.float32)]
            del q, qt, r, c, g                                     # and its buffers go to the next round
        return out
    try:
        lib.nvfp4_set_pdl(0)
        want = chain()
        lib.nvfp4_set_pdl(mode)
        for _ in range(8):
            assert all(torch.equal(a, b) for a, b in zip(chain(), want))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = chain()
        for _ in range(3):
            graph.replay()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        lib.nvfp4_set_pdl(2)
    L.check_status()
