"""The swizzled scales a `fp4ops.Q` carries beside its row-major ones serve only while the two are known to agree: once
somebody has got hold of the row-major tensor, whatever that tensor holds is what `gemm` multiplies with."""
import copy
import pickle

import pytest
import torch

from nvfp4_training_b200 import fp4ops


def _replace(q):
    q.s = torch.zeros_like(q.s)


def _in_place(q):
    q.s.bitwise_and_(0x77)


def _data(q):
    q.s.data.zero_()


def _storage(q):
    q.s.untyped_storage().fill_(0)


def _copy(q):
    copy.copy(q).s.data.zero_()


WRITES = [_replace, _in_place, _data, _storage, _copy]


def _made():
    s = torch.arange(128 * 8, dtype=torch.uint8).reshape(128, 8)
    return fp4ops.Q._made(torch.zeros(128, 64, dtype=torch.uint8), s, torch.ones(1), 1.0, s.flatten().clone())


@pytest.mark.parametrize("write", WRITES)
def test_scales_in_other_hands_are_not_replaced_by_a_copy(write):
    q = _made()
    assert q.swizzled() is q.sw
    write(q)
    assert q.swizzled() is None


def test_an_sw_of_the_callers_serves_until_s_changes():
    s = torch.zeros(128, 8, dtype=torch.uint8)
    for change in (_replace, _in_place):
        q = fp4ops.Q(None, s.clone(), None, 1.0, s.flatten())
        assert q.s is not None and q.swizzled() is q.sw
        change(q)
        assert q.swizzled() is None
    q = fp4ops.Q(None, s, None)
    assert q.sw is None and q.swizzled() is None
    q.sw = s.flatten()
    assert q.swizzled() is q.sw


def test_copies_and_pickles_keep_the_slots():
    q = _made()
    for r in (copy.copy(q), copy.deepcopy(q), pickle.loads(pickle.dumps(q))):
        assert torch.equal(r.swizzled(), q.sw) and torch.equal(r.d, q.d) and r.k == q.k
        assert torch.equal(r.s, q._scales.s)
    # the slots of a Q without the shared state, in the order they had
    r = fp4ops.Q.__new__(fp4ops.Q)
    for name in ("d", "s", "amax", "k", "sw"):
        setattr(r, name, getattr(q, name))
    assert r.s is q.s and r.sw is q.sw


@pytest.mark.gpu
@pytest.mark.parametrize("write", WRITES)
def test_gemm_multiplies_with_the_scales_as_they_stand(write):
    x, w = (torch.randn(128, 256, device="cuda").bfloat16() for _ in range(2))
    for make in (fp4ops.quant_rows, lambda t: fp4ops.quant_cols_rht(t.t().contiguous(), 0xA6B1),
                 lambda t: fp4ops.quant_rows_cols_rht(t, 0xA6B1)[0], lambda t: fp4ops.quant_w2d(t.float())[0]):
        q, b = make(x), fp4ops.quant_rows(w)
        assert torch.equal(fp4ops.gemm(q, b), fp4ops.gemm(fp4ops.Q(q.d, q.s.clone(), q.amax, q.k), b))
        q = make(x)
        write(q)
        want = fp4ops.gemm(fp4ops.Q(q.d, q.s.clone(), q.amax, q.k), b)
        assert torch.equal(fp4ops.gemm(q, b), want)
        if write is not _in_place:
            assert not want.any()


def test_an_sw_can_be_given_in_inference_mode():
    with torch.inference_mode():
        s = torch.zeros(128, 8, dtype=torch.uint8)
        q = fp4ops.Q(None, s, None, 1.0, s.flatten())
        assert q.swizzled() is q.sw
        _replace(q)
        assert q.swizzled() is None


@pytest.mark.gpu
def test_inference_mode():
    from nvfp4_training_b200 import fp4torch
    x, w = torch.randn(128, 256, device="cuda").bfloat16(), torch.randn(256, 256, device="cuda") * 0.02

    def run():
        fw = fp4torch.FP4Weight(w)
        fw.refresh()
        a, c = fp4ops.quant_rows_cols_rht(x, 0xA6B1)
        return [fp4torch.fp4_fwd(x, fw.wd, fw.ws, fw.amax), fp4torch.fp4_linear(x, w, fw.wd, fw.ws, fw.wtd, fw.wts, fw.amax),
                fp4ops.gemm(a, fp4ops.quant_w2d(w)[0]), fp4ops.gemm(c, c, splitk=2),
                fp4ops.gemm(fp4ops.quant_rows(x), fp4ops.quant_rows(w.bfloat16())), fp4ops.quant_cols_rht(x, 0xA6B1).s]
    want = run()
    with torch.inference_mode():
        got = run()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
