"""The work a training or inference program hands to this library, as timed cases.

Every case is one pass through the public entry points, called the way a model calls them: the autograd linear
(`linear.Linear`), the gradient-accumulating pair (`linear.linear_fwd` / `linear_bwd`), the row-major-scale contract of
the compiled model (`fp4torch`, `fp4ops`), the operand emitters (`emit`), the per-step weight re-quantization
(`nvq.quant_w2d`, `FP4Weight.refresh`), the quantizers and the GEMM by themselves (`nvq`), and the graph-replayed
training step (`stack.LinearStack`).  Distributions are those of a transformer's linears: activations N(0, 1), weights
truncated N(0, 0.02), output gradients Student-t with 3 degrees of freedom x 1e-3.
"""
import math

import torch

from nvfp4_training_b200 import _lib, emit, fp4ops, fp4torch, linear, nvq, stack

_SIGNS = 0b1010011010110001
_PACKED = 0.5625          # bytes of one packed value: half a byte of code and a sixteenth of a scale byte


def listed():
    return [
        # the smallest layer the library takes, drop-in autograd form (weights quantized in the call): launches and host
        # work are all there is
        dict(name="linear_small", kind="linear", T=128, K=256, N=384, cache=False),
        # one attention projection of a 2 x 2048-token microbatch in the same drop-in form
        dict(name="linear_qkv", kind="linear", T=4096, K=2048, N=3072, cache=False),
        # odd multiples of 128 everywhere: no dimension is a multiple of the wide tiles; weights cached per step
        dict(name="linear_odd", kind="linear", T=3200, K=1408, N=2176, cache=True),
        # inference: a short prompt (or a batch of decoding sequences) through the down projection, weights quantized
        # once, no gradient recorded
        dict(name="infer_down", kind="infer", T=256, K=5632, N=2048),
        # gate/up projection of a large microbatch, FP32 gradients accumulated over microbatches, hardware SR
        dict(name="accum_gate_up", kind="accum", T=16384, K=2048, N=11264, first=False),
        # the LM head of one microbatch, first microbatch of a step (gradient overwritten)
        dict(name="accum_lm_head", kind="accum", T=4096, K=2048, N=49152, first=True),
        # the compiled model's layer: row-major scales, FP32 master weight refreshed every step, split-K gradient
        dict(name="compiled_step", kind="compiled", T=2048, K=1024, N=3072),
        # a batch whose size fits no tile, quantized row-wise and column-wise with row-major scales
        dict(name="quant_ragged", kind="ragged", M=5008, C=1552),
        # one optimizer step's re-quantization of a block's four bf16 weights into kept buffers
        dict(name="refresh_block", kind="refresh", d=2048, ff=5632, heads=16, kv_heads=4),
        # feed-forward block through the operand emitters: RMSNorm, gate/up, SwiGLU, down, and their gradients, ending
        # in the momentum accumulation
        dict(name="emit_ffn", kind="emit", T=4096, D=2048, F=5632),
        # weight gradient over a long token dimension: both operands quantized, FP32 result
        dict(name="wgrad_16384", kind="wgrad", T=16384, K=2048, N=5632),
        # training step of two transformer blocks, graphs replayed, two microbatches of 8192 rows
        dict(name="stack_step", kind="stack", T=8192, layers=2, n_micro=2),
    ]


def _multiple(rng, lo, hi, of):
    """A multiple of `of` in [lo, hi], spread over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + of)))
    return min(hi, max(lo, int(v) // of * of))


def draw(rng):
    kind = rng.choice(["linear", "linear", "infer", "accum", "accum", "compiled", "ragged", "refresh", "emit", "wgrad", "stack"])
    if kind == "ragged":
        return dict(kind=kind, M=_multiple(rng, 16, 20000, 16), C=_multiple(rng, 16, 6000, 16))
    if kind == "refresh":
        heads = rng.randint(2, 20)
        return dict(kind=kind, d=heads * 128, ff=_multiple(rng, 256, 8192, 128), heads=heads, kv_heads=rng.randint(1, heads))
    if kind == "emit":
        return dict(kind=kind, T=_multiple(rng, 256, 16384, 256), D=rng.choice([1024, 2048]), F=_multiple(rng, 512, 6144, 256))
    if kind == "stack":
        return dict(kind=kind, T=_multiple(rng, 256, 8192, 128), layers=rng.randint(1, 2), n_micro=rng.randint(1, 2))
    T = _multiple(rng, 128, 16384, 128)
    K = _multiple(rng, 128, 5632, 128)
    N = _multiple(rng, 128, 11264, 128)
    while T * K * N > 16384 * 2048 * 11264:
        T = max(128, T // 256 * 128)
    case = dict(kind=kind, T=T, K=K, N=N)
    if kind == "linear":
        case["cache"] = rng.random() < 0.5
    if kind == "accum":
        case["first"] = rng.random() < 0.5
    return case


# ---------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _x(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda").bfloat16()


def _w(g, N, K):
    return torch.nn.init.trunc_normal_(torch.empty(N, K, device="cuda"), std=0.02, a=-0.06, b=0.06, generator=g)


def _gy(g, *shape):
    """Student-t, 3 degrees of freedom, x 1e-3: heavy-tailed like the gradients of a language model."""
    chi = torch.zeros(*shape, device="cuda")
    for _ in range(3):
        chi += torch.randn(*shape, generator=g, device="cuda").square_()
    return (torch.randn(*shape, generator=g, device="cuda") / torch.sqrt(chi / 3) * 1e-3).bfloat16()


def _seed_words(g):
    return torch.randint(-2 ** 31, 2 ** 31 - 1, (2,), generator=g, device="cuda", dtype=torch.int32)


def _weights_of(case):
    """(N, K) of a block's four projections."""
    d, hd = case["d"], case["d"] // case["heads"]
    return [((case["heads"] + 2 * case["kv_heads"]) * hd, d), (d, d), (2 * case["ff"], d), (d, case["ff"])]


def _prepare_linear(case, g):
    T, K, N = case["T"], case["K"], case["N"]
    with torch.device("cuda"):
        lin = linear.Linear(K, N, std=0.02, cache_weights=case["kind"] == "infer" or case["cache"])
    lin = lin.bfloat16()
    lin.lid = 5                                    # the layer's number seeds its stochastic rounding
    with torch.no_grad():
        lin.weight.copy_(_w(g, N, K))
    lin.refresh()
    if case["kind"] == "infer":
        return dict(lin=lin, x=_x(g, T, K))
    return dict(lin=lin, x=_x(g, T, K).requires_grad_(True), gy=_gy(g, T, N))


def _run_linear(s):
    y = s["lin"](s["x"])
    gx, gw = torch.autograd.grad(y, (s["x"], s["lin"].weight), s["gy"])
    return y, gx, gw


def _run_infer(s):
    with torch.no_grad():
        return s["lin"](s["x"])


def _prepare_accum(case, g):
    T, K, N = case["T"], case["K"], case["N"]
    qw, qwt = nvq.quant_w2d(_w(g, N, K).bfloat16())
    return dict(qw=qw, qwt=qwt, x=_x(g, T, K), gy=_gy(g, T, N), gw=torch.zeros(N, K, device="cuda"),
                seeds=_seed_words(g), first=case["first"])


def _run_accum(s):
    y, am, qxt = linear.linear_fwd(s["x"], s["qw"], keep_xt=True)
    gx, gw = linear.linear_bwd(None, am, s["gy"], s["qwt"], s["seeds"][0:1], s["seeds"][1:2], gw_out=s["gw"],
                               sr_mode=_lib.ROUND_SR_HW, overwrite=s["first"], qxt=qxt)
    return y, gx, gw


def _prepare_compiled(case, g):
    T, K, N = case["T"], case["K"], case["N"]
    return dict(fw=fp4torch.FP4Weight(_w(g, N, K)), x=_x(g, T, K), gy=_gy(g, T, N), seed=int(_seed_words(g)[0]) & 0xFFFFFFFF)


def _run_compiled(s):
    fw, g = s["fw"].refresh(), s["gy"]
    y = fp4torch.fp4_fwd(s["x"], fw.wd, fw.ws, fw.amax)
    # the backward of the custom op, with the caller's seeds instead of a process-wide count
    qg, qgt = fp4ops.quant_rows_cols_rht(g, _SIGNS, sr=True, seed=s["seed"], seed_cols=s["seed"] ^ 0x5BD1E995)
    gx = fp4ops.gemm(qg, fp4ops.Q(fw.wtd, fw.wts, fw.amax))
    gw = fp4ops.gemm(qgt, fp4ops.quant_cols_rht(s["x"], _SIGNS), splitk=16)
    return y, gx, gw


def _prepare_ragged(case, g):
    return dict(x=_x(g, case["M"], case["C"]), seed=int(_seed_words(g)[0]) & 0xFFFFFFFF)


def _run_ragged(s):
    a = fp4ops.amax_of(s["x"])
    qr = fp4ops.quant_rows(s["x"], amax=a)
    qc = fp4ops.quant_cols_rht(s["x"], _SIGNS, sr=True, seed=s["seed"], amax=a)
    return qr.d, qr.s, qc.d, qc.s, a


def _prepare_refresh(case, g):
    ws = [_w(g, N, K).bfloat16() for N, K in _weights_of(case)]
    return dict(ws=ws, pairs=[nvq.quant_w2d(w) for w in ws])


def _run_refresh(s):
    out = []
    for w, pair in zip(s["ws"], s["pairs"]):
        for q in nvq.quant_w2d(w, out=pair):
            out += [q.d.view(torch.uint8), q.s.view(torch.uint8), q.gs]
    return out


def _prepare_wgrad(case, g):
    return dict(x=_x(g, case["T"], case["K"]), gy=_gy(g, case["T"], case["N"]), seed=_seed_words(g)[0:1])


def _run_wgrad(s):
    qgt = nvq.quant_cols_rht(s["gy"], _SIGNS, sr=True, seed=s["seed"], sr_mode=_lib.ROUND_SR_HW)
    qxt = nvq.quant_cols_rht(s["x"], _SIGNS)
    return nvq.mm(qgt, qxt, out_dtype=torch.float32, splitk=0)


def _prepare_emit(case, g):
    T, D, F = case["T"], case["D"], case["F"]
    s = dict(x=_x(g, T, D), branch=_x(g, T, D), branch_rs=torch.rand(T, generator=g, device="cuda") + 0.5,
             branch_gs=torch.full((1,), 0.1, device="cuda"), norm=(1 + 0.1 * torch.randn(D, generator=g, device="cuda")).bfloat16(),
             gy=_gy(g, T, D), dgu=_gy(g, T, 2 * F), xout=torch.empty(T, D, dtype=torch.bfloat16, device="cuda"),
             h=torch.empty(T, D, dtype=torch.bfloat16, device="cuda"), rstd=torch.empty(T, device="cuda"),
             a=torch.empty(T, F, dtype=torch.bfloat16, device="cuda"),
             w_gu=emit.WQ(2 * F, D).refresh(_w(g, 2 * F, D)), w_down=emit.WQ(D, F).refresh(_w(g, D, F)),
             rq={k: emit.RowQ(T, c) for k, c in (("h", D), ("a", F), ("gy", D), ("dgu", 2 * F))},
             cq={k: emit.ColQ(T, c) for k, c in (("h", D), ("a", F), ("gy", D), ("dgu", 2 * F))},
             use={k: torch.full((1,), 1e3, device="cuda") for k in ("h", "a", "gy", "dgu")},
             cur={k: torch.zeros(1, dtype=torch.int32, device="cuda") for k in ("h", "a", "gy", "dgu")},
             rng=_seed_words(g), alpha=torch.ones(1, device="cuda"),
             m_gu=torch.zeros(2 * F, D, dtype=torch.bfloat16, device="cuda"), m_down=torch.zeros(D, F, dtype=torch.bfloat16, device="cuda"))
    # the delayed scales come from the previous microbatch's observed maxima, times a margin of 2
    _run_emit(s)
    for k, word in s["cur"].items():
        s["use"][k].copy_(word.view(torch.float32) * 2)
    s["m_gu"].zero_()
    s["m_down"].zero_()
    return s


def _run_emit(s):
    rq, cq, use, cur, rng = s["rq"], s["cq"], s["use"], s["cur"], s["rng"]
    for word in cur.values():
        word.zero_()

    def col(k, x, sr, salt):
        return emit.col_emit(x, cq[k], use[k], cur[k], rng, sr=sr, salt=salt)

    # forward: residual add, norm, gate | up, SwiGLU, down
    emit.rms_emit(s["x"], s["norm"], q=rq["h"], h=s["h"], rstd=s["rstd"], y=s["branch"], ys=s["branch_rs"], ygw=s["branch_gs"],
                  xout=s["xout"])
    col("h", s["h"], False, 0)
    gu = emit.mm_row_w(rq["h"], s["w_gu"])
    emit.swiglu_emit(gu, rq["h"].rs, s["w_gu"].gs, q=rq["a"], a=s["a"])
    col("a", s["a"], False, 0)
    y = emit.mm_row_w(rq["a"], s["w_down"], scale=True)
    # backward: the gradient of the SwiGLU itself belongs to the model, its result is an input here
    emit.row_emit(s["gy"], rq["gy"], rng, sr="hw", salt=1)
    col("gy", s["gy"], "hw", 2)
    da = emit.mm_row_wt(rq["gy"], s["w_down"], scale=True)
    emit.mom_acc(s["m_down"], emit.mm_col(cq["gy"], cq["a"], out_dtype=torch.bfloat16), s["alpha"], 1e-6, rng, salt=3)
    emit.row_emit(s["dgu"], rq["dgu"], rng, sr="hw", salt=4)
    col("dgu", s["dgu"], "hw", 5)
    dh = emit.mm_row_wt(rq["dgu"], s["w_gu"], scale=True)
    emit.mom_acc(s["m_gu"], emit.mm_col(cq["dgu"], cq["h"], out_dtype=torch.bfloat16), s["alpha"], 1e-6, rng, salt=6)
    return [s["xout"], s["rstd"], y, da, dh, s["m_down"], s["m_gu"], cur["h"].view(torch.float32), cur["a"].view(torch.float32),
            cur["gy"].view(torch.float32), cur["dgu"].view(torch.float32)]


def _prepare_stack(case, seed):
    st = stack.LinearStack(stack.StackConfig(layers=case["layers"], lm_head=False), case["T"], "cuda", seed=seed)
    st.capture()
    return dict(st=st, n_micro=case["n_micro"])


def _run_stack(s):
    s["st"].step(s["n_micro"], do_allreduce=False)
    return [p.gw for projs in s["st"].blocks for p in projs]


_RUN = dict(linear=_run_linear, infer=_run_infer, accum=_run_accum, compiled=_run_compiled, ragged=_run_ragged,
            refresh=_run_refresh, emit=_run_emit, wgrad=_run_wgrad, stack=_run_stack)
_PREPARE = dict(linear=_prepare_linear, infer=_prepare_linear, accum=_prepare_accum, compiled=_prepare_compiled,
                ragged=_prepare_ragged, refresh=_prepare_refresh, emit=_prepare_emit, wgrad=_prepare_wgrad)


def prepare(case, seed):
    kind = case["kind"]
    s = _prepare_stack(case, seed) if kind == "stack" else _PREPARE[kind](case, _gen(seed))
    s["kind"] = kind
    return s


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------------------------------- accounting
def work(case):
    kind = case["kind"]
    if kind == "ragged":
        n = case["M"] * case["C"]
        return dict(bytes=n * (2 + 2 * _PACKED), flops=0)
    if kind == "refresh":
        return dict(bytes=sum(N * K for N, K in _weights_of(case)) * (2 + 2 * _PACKED), flops=0)
    if kind == "emit":
        T, D, F = case["T"], case["D"], case["F"]
        w = 3 * D * F
        # x, branch, xout, y, gy, dh; dgu; da; packed weights in both orientations; momenta read and written
        return dict(bytes=T * (12 * D + 4 * F + 2 * F + 8) + w * (2 * _PACKED + 4), flops=6 * T * w)
    if kind == "stack":
        d, ff = 2048, 5632
        T, micro = case["T"], case["n_micro"]
        total = dict(bytes=0, flops=0)
        for N, K in _weights_of(dict(d=d, ff=ff, heads=16, kv_heads=4)):
            # activations per microbatch; the weight once in bf16, its packed forms written once and read by each
            # microbatch; the FP32 gradient written by the first microbatch, read and written by the others
            total["bytes"] += case["layers"] * (micro * 4 * T * (N + K) + N * K * (2 + 2 * _PACKED * (1 + micro) + 4 + 8 * (micro - 1)))
            total["flops"] += case["layers"] * micro * 6 * T * N * K
        return total
    T, K, N = case["T"], case["K"], case["N"]
    if kind == "infer":
        return dict(bytes=2 * T * (K + N) + _PACKED * N * K, flops=2 * T * N * K)
    if kind == "wgrad":
        return dict(bytes=2 * T * (K + N) + 4 * N * K, flops=2 * T * N * K)
    per_weight = {"linear": (2 * _PACKED if case.get("cache") else 2) + 2,             # bf16 gradient
                  "accum": 2 * _PACKED + (4 if case.get("first") else 8),             # FP32 gradient, added to or overwritten
                  "compiled": 4 + 2 * _PACKED + 4}[kind]                              # FP32 weight and gradient, packed copies written
    return dict(bytes=4 * T * (K + N) + per_weight * N * K, flops=6 * T * N * K)


def tolerance(case):
    kind = case["kind"]
    if kind in ("ragged", "refresh"):
        return "exact"                                   # codes, scale bytes and scales are the same everywhere
    if kind in ("wgrad", "stack"):
        return {"rel": 1e-5, "max": 1e-4}                # FP32 sums of exact products, in another order
    # products rounded to bf16 from FP32 sums of another order: a result next to a rounding boundary moves by one step
    return {"rel": 4e-3, "max": 1e-2}
