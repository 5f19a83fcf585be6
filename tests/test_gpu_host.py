"""The native host path (csrc/host.cpp): the autograd linear gives the same bits whichever gradients are asked for, with
and without a weight cache, and keeps autograd's rules (versions, freed graphs, error types)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(T, K, N, cache):
    from nvfp4_training_b200.linear import Linear
    torch.manual_seed(T + K + N)
    with torch.device("cuda"):
        lin = Linear(K, N, std=0.02, cache_weights=cache)
    lin = lin.bfloat16()
    lin.lid = 3
    lin.refresh()
    x = torch.randn(T, K, device="cuda").bfloat16()
    gy = (torch.randn(T, N, device="cuda") * 1e-3).bfloat16()
    return lin, x, gy


@pytest.mark.parametrize("cache", [False, True])
@pytest.mark.parametrize("T,K,N", [(128, 128, 128), (384, 256, 640)])
def test_linear_gradients_are_the_same_whichever_are_wanted(T, K, N, cache):
    lin, x, gy = _layer(T, K, N, cache)
    xg = x.clone().requires_grad_(True)
    y = lin(xg)
    gx, gw = torch.autograd.grad(y, (xg, lin.weight), gy, retain_graph=True)
    again = torch.autograd.grad(y, (xg, lin.weight), gy)
    assert torch.equal(gx, again[0]) and torch.equal(gw, again[1])
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y, (xg, lin.weight), gy)              # the graph has been freed
    with torch.no_grad():
        assert torch.equal(lin(xg), y)
    assert torch.equal(torch.autograd.grad(lin(x), lin.weight, gy)[0], gw)           # x needs no gradient
    assert torch.equal(torch.autograd.grad(lin(xg), xg, gy)[0], gx)                  # only x's asked for
    lin.weight.requires_grad_(False)                                                 # frozen weight
    y2 = lin(xg)
    assert torch.equal(y2, y) and torch.equal(torch.autograd.grad(y2, xg, gy)[0], gx)
    y3 = lin(xg.view(2, T // 2, K))                                                  # leading dimensions are flattened
    assert y3.shape == (2, T // 2, N) and torch.equal(y3.view(T, N), y)


def test_linear_notices_an_in_place_weight_change():
    lin, x, gy = _layer(128, 128, 256, False)
    y = lin(x)
    with torch.no_grad():
        lin.weight.mul_(2)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y, lin.weight, gy)


def test_host_errors_keep_their_types():
    from nvfp4_training_b200 import _lib, nvq
    with pytest.raises(_lib.Nvfp4Error):
        nvq.amax(torch.zeros(8, dtype=torch.bfloat16))
    with pytest.raises(AssertionError):
        nvq.quant_rows(torch.zeros(100, 64, dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(AssertionError):
        nvq.quant_rows(torch.zeros(128, 64, device="cuda"))
    q = nvq.quant_rows(torch.ones(128, 64, dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(AssertionError):
        nvq.mm(q, nvq.quant_rows(torch.ones(128, 128, dtype=torch.bfloat16, device="cuda")))


def test_linear_fwd_wants_contiguous_rows():
    from nvfp4_training_b200 import linear, nvq
    base = torch.randn(128, 512, device="cuda").bfloat16()
    qw = nvq.quant_w2d(torch.randn(256, 256, device="cuda").bfloat16())[0]
    with pytest.raises(AssertionError):
        linear.linear_fwd(base[:, ::2], qw, keep_xt=True)              # every other column
    with pytest.raises(AssertionError):
        linear.linear_fwd(base[:, :256].reshape(256, 128).t(), qw, keep_xt=True)
    for x in (base[:, :256], base[:, 256:]):                           # rows with a stride
        y, am, qxt = linear.linear_fwd(x, qw, keep_xt=True)
        y2, am2, qxt2 = linear.linear_fwd(x.contiguous(), qw, keep_xt=True)
        assert torch.equal(y, y2) and torch.equal(am, am2) and torch.equal(qxt.d.view(torch.uint8), qxt2.d.view(torch.uint8))


@pytest.mark.parametrize("call", ["amax", "layer"])
def test_other_threads_run_while_launches_wait(call):
    """Half a second of work in front of more launches than a stream's queue holds: calls block, the interpreter does not."""
    import threading
    import time
    from nvfp4_training_b200 import nvq
    lin, x, _ = _layer(128, 128, 128, False)
    word = torch.zeros(1, device="cuda")

    def launch():
        if call == "amax":
            nvq.amax(x, out=word, clear=False)
        else:
            with torch.no_grad():
                lin(x)
    for _ in range(3):
        launch()
    torch.cuda.synchronize()
    done, gap = threading.Event(), [0.0]

    def beat():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gap[0], last = max(gap[0], now - last), now
    thread = threading.Thread(target=beat)
    thread.start()
    torch.cuda._sleep(int(1e9))                              # cycles
    t0 = time.perf_counter()
    for _ in range(4000):
        launch()
    waited = time.perf_counter() - t0
    done.set()
    thread.join()
    torch.cuda.synchronize()
    assert waited > 0.25 and gap[0] < waited / 2


def test_errors_in_the_backward_pass_keep_their_types(monkeypatch):
    from nvfp4_training_b200 import _lib
    from nvfp4_training_b200.linear import LinCtx
    lin, x, gy = _layer(128, 128, 256, False)
    xg = x.clone().requires_grad_(True)
    off = torch.zeros(128 * 256 + 8, dtype=torch.bfloat16, device="cuda")[4:-4].view(128, 256)     # off its 16-byte boundary
    for cuda_grad, name, value, error in ((off, "seed", 1, _lib.Nvfp4Error), (gy, "wgrad_dtype", torch.float16, AssertionError),
                                          (gy, "wgrad_dtype", None, AssertionError), (gy, "wgrad_dtype", "float32", AssertionError),
                                          (gy, "seed", "one", TypeError)):
        with monkeypatch.context() as m:
            m.setattr(LinCtx, name, value)
            with pytest.raises(error) as caught:
                torch.autograd.grad(lin(xg), (xg, lin.weight), cuda_grad)
            assert caught.type is error
    torch.autograd.grad(lin(xg), (xg, lin.weight), gy)


@pytest.mark.parametrize("dtype", [torch.float16, torch.int32, None, "float32"])
def test_linear_bwd_refuses_other_gradient_types(dtype):
    from nvfp4_training_b200 import linear, nvq
    x, gy = (torch.randn(128, 128, device="cuda").bfloat16() for _ in range(2))
    qw, qwt = nvq.quant_w2d(x)
    _, am, qxt = linear.linear_fwd(x, qw, keep_xt=True)
    with pytest.raises(AssertionError):
        linear.linear_bwd(None, am, gy, qwt, 1, 2, qxt=qxt, wgrad_dtype=dtype)
    gw = torch.zeros(128, 128, device="cuda")                          # `gw_out` decides the type where it is given
    assert linear.linear_bwd(None, am, gy, qwt, 1, 2, qxt=qxt, wgrad_dtype=dtype, gw_out=gw)[1] is gw
    for ok in (torch.float32, torch.bfloat16):
        assert linear.linear_bwd(None, am, gy, qwt, 1, 2, qxt=qxt, wgrad_dtype=ok)[1].dtype == ok


def test_packed_operands_may_have_a_row_stride():
    """Codes with padding between their rows: the same results from the pair and from a layer whose cache holds them."""
    from nvfp4_training_b200 import linear, nvq

    def padded(q):
        wide = torch.full((q.d.shape[0], q.d.shape[1] + 32), 0x77, dtype=torch.uint8, device="cuda")
        wide[:, :q.d.shape[1]] = q.d.view(torch.uint8)
        return nvq.Q(wide[:, :q.d.shape[1]].view(q.d.dtype), q.s, q.gs)
    lin, x, gy = _layer(384, 256, 640, True)
    qw, qwt = lin.cache.q, lin.cache.qt
    y, am, qxt = linear.linear_fwd(x, qw, keep_xt=True)
    gx, gw = linear.linear_bwd(None, am, gy, qwt, 1, 2, qxt=qxt)
    y2, am2, _ = linear.linear_fwd(x, padded(qw), keep_xt=True)
    gx2, gw2 = linear.linear_bwd(None, am2, gy, padded(qwt), 1, 2, qxt=padded(qxt))
    assert torch.equal(y, y2) and torch.equal(gx, gx2) and torch.equal(gw, gw2)
    xg = x.clone().requires_grad_(True)
    want = torch.autograd.grad(lin(xg), (xg, lin.weight), gy)
    lin.cache.q, lin.cache.qt = padded(qw), padded(qwt)
    got = torch.autograd.grad(lin(xg), (xg, lin.weight), gy)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("T,K,N", [(128, 128, 256), (1024, 2048, 640)])
def test_calls_that_need_an_amax_can_be_captured(T, K, N):
    from nvfp4_training_b200 import fp4ops, nvq
    lin, x, gy = _layer(T, K, N, False)
    w32 = lin.weight.detach().float()

    def run():
        xg = x.clone().requires_grad_(True)
        y = lin(xg)
        q, qt = nvq.quant_w2d(lin.weight)
        k, kt = fp4ops.quant_w2d(w32)
        r, c = nvq.quant_rows(x), nvq.quant_cols_rht(x, 0xA6B1)
        return [y.detach(), *torch.autograd.grad(y, (xg, lin.weight), gy), nvq.amax(x), fp4ops.amax_of(w32), q.gs, k.s, kt.d, fp4ops.quant_rows(x).s,
                q.d.view(torch.uint8), qt.s.view(torch.uint8), r.d.view(torch.uint8), c.d.view(torch.uint8)]
    want = run()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    for _ in range(2):
        for t in got:
            t.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_forward_mode_is_refused():
    import torch.autograd.forward_ad as fwd
    lin, x, _ = _layer(128, 128, 128, False)
    with fwd.dual_level():
        with pytest.raises(NotImplementedError):
            lin(fwd.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("cache", [False, True])
def test_the_function_is_an_autograd_function(cache):
    """Derived functions run their own forward and backward; positional arguments only, as autograd's apply takes them."""
    from nvfp4_training_b200.linear import FP4LinearFn
    assert issubclass(FP4LinearFn, torch.autograd.Function)
    lin, x, gy = _layer(256, 128, 384, cache)
    xg = x.clone().requires_grad_(True)
    seen = []

    class Doubled(FP4LinearFn):
        @staticmethod
        def forward(ctx, *args):
            seen.append("forward")
            return FP4LinearFn.forward(ctx, *args) * 2

        @staticmethod
        def backward(ctx, g):
            seen.append("backward")
            return FP4LinearFn.backward(ctx, g)
    y = FP4LinearFn.apply(xg, lin.weight, lin.lid, lin.cache)
    want = torch.autograd.grad(y, (xg, lin.weight), gy)
    y2 = Doubled.apply(xg, lin.weight, lin.lid, lin.cache)
    got = torch.autograd.grad(y2, (xg, lin.weight), gy)
    assert seen == ["forward", "backward"] and torch.equal(y2, y * 2)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    for bad in ({"lid": 3}, {"lid": 3, "cache": None}):
        with pytest.raises(TypeError):
            FP4LinearFn.apply(x, lin.weight, **bad)
    for args in ((x,), (x, lin.weight, 3, None, None)):
        with pytest.raises(TypeError):
            FP4LinearFn.apply(*args)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda a: FP4LinearFn.apply(a, lin.weight.detach(), 3, lin.cache).float().sum())(x)
    with pytest.raises(RuntimeError):
        torch.vmap(lambda a: FP4LinearFn.apply(a, lin.weight.detach(), 3, lin.cache))(torch.stack([x, x]))


def test_a_compiled_model_runs_the_layer():
    """torch.compile breaks its graph at the layer and runs it as it is."""
    lin, x, gy = _layer(128, 128, 256, False)
    xg = x.clone().requires_grad_(True)
    y = lin(xg.relu())
    want = torch.autograd.grad(y, (xg, lin.weight), gy)
    f = torch.compile(lambda a: lin(a.relu()), backend="eager")
    y2 = f(xg)
    assert torch.equal(y, y2)
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y2, (xg, lin.weight), gy), want))


def test_backward_passes_of_several_threads_over_one_graph():
    """Each gets the gradients, or the error for a graph another thread has freed."""
    from concurrent.futures import ThreadPoolExecutor
    lin, x, gy = _layer(128, 128, 256, False)
    xg = x.clone().requires_grad_(True)

    def grads(y, keep):
        try:
            got = torch.autograd.grad(y, (xg, lin.weight), gy, retain_graph=keep)
            torch.cuda.synchronize()
            return got
        except RuntimeError as e:
            assert "second time" in str(e)
            return None
    want = grads(lin(xg), False)
    with ThreadPoolExecutor(8) as pool:
        for keep in (True, False):
            for _ in range(20):
                y = lin(xg)
                results = list(pool.map(lambda _: grads(y, keep), range(8)))
                assert any(r is not None for r in results) and (not keep or None not in results)
                for r in results:
                    assert r is None or all(torch.equal(a, b) for a, b in zip(r, want))
