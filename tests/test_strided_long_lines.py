"""Strided axes whose lines are long: columns past the two-buffer limit take
two passes, few long columns a CTA each (as strided rows), against numpy in
64 bits (2-norm bounds of every route: 2e-6 in f32, 1e-14 in f64)."""
import numpy as np
import pytest

import wgpufft_b200 as w

PREC = {"f32": w.FftPrecision.F32, "f64": w.FftPrecision.F64}


def config(shape, prec, batch=1, inverse=False):
    return (w.FftConfig.new_nd(shape).with_axes([1]).with_batch(batch).with_precision(PREC[prec])
            .with_direction(w.FftDirection.Inverse if inverse else w.FftDirection.Forward))


def stages(shape, prec, batch=1):
    plan = w.FftPlan.plan_only(config(shape, prec, batch), w.FftTransformKind.C2c)
    return plan.diagnostics()["stages"]


@pytest.mark.parametrize("n,prec", [(14014, "f32"), (20000, "f32"), (28800, "f32"), (7000, "f64"),
                                    (13500, "f64")])
@pytest.mark.parametrize("s", [2, 8, 15])
def test_long_columns_take_two_passes(n, prec, s):
    """One column a CTA uses a quarter of each sector; a row still takes one
    pass."""
    assert len(stages([s, n], prec)) == 2
    plan = w.FftPlan.plan_only(w.FftConfig.new(n).with_precision(PREC[prec]), w.FftTransformKind.C2c)
    assert len(plan.diagnostics()["stages"]) == 1


@pytest.mark.parametrize("n,prec", [(4099, "f32"), (4999, "f32"), (9240, "f32"), (2039, "f64"),
                                    (3011, "f64")])
@pytest.mark.parametrize("s,batch", [(2, 1), (8, 1), (16, 1), (8, 9)])
def test_few_long_columns_have_a_cta_each(n, prec, s, batch):
    if n == 9240 and s >= 16:
        pytest.skip("sixteen columns or more take two passes")
    (stage,) = stages([s, n], prec, batch)
    assert stage["lines_per_block"] == 1 and stage["grid"] == s * batch


CASES = [([2, 20000], 3, "f32"), ([15, 28800], 1, "f32"), ([3, 13500], 1, "f64"),
         ([16, 4099], 2, "f32"), ([2, 9240], 2, "f32"), ([200, 3011], 1, "f32"),
         ([5, 12601], 1, "f32"), ([6, 8009], 1, "f32"), ([3, 12011], 30, "f32"),
         ([3, 14051], 1, "f32"), ([7, 2039], 2, "f64"), ([2, 4051], 2, "f64")]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,batch,prec", CASES)
@pytest.mark.parametrize("inverse", [False, True])
def test_against_numpy(shape, batch, prec, inverse):
    import torch
    g = torch.Generator().manual_seed(5)
    x = torch.randn([batch] + shape[::-1], generator=g,
                    dtype=torch.complex64 if prec == "f32" else torch.complex128).cuda()
    out = torch.empty_like(x)
    plan = w.FftPlan.c2c(config(shape, prec, batch, inverse))
    plan.execute_checked(x, out)
    z = x.cpu().numpy().astype(np.complex128)
    # the library scales an inverse transform by its whole shape
    ref = np.fft.ifft(z, axis=1) / shape[0] if inverse else np.fft.fft(z, axis=1)
    tol = 2e-6 if prec == "f32" else 1e-14
    assert np.linalg.norm(out.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
    plan.execute_in_place(x)
    assert torch.equal(x, out)
