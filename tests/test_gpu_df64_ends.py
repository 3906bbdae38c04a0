"""df64 plans compute in f64 between words in and words out: every kind of
first and last pass converts (or does not) on the right side.  The output's
hi + lo pair holds at least 48 bits, so one rounding of the result is below
2^-48 and the f64 transform's own error about 1e-15: 1e-14 in the 2-norm."""
import numpy as np
import pytest
import torch

import wgpufft_b200 as w

pytestmark = pytest.mark.gpu


def words(z):
    v = np.stack([z.real, z.imag], -1)
    hi = v.astype(np.float32)
    lo = (v - hi).astype(np.float32)
    return np.stack([hi, lo], -1).reshape(z.shape + (4,))


def value(x):
    x = x.astype(np.float64)
    return (x[..., 0] + x[..., 1]) + 1j * (x[..., 2] + x[..., 3])


# one pass, two and three passes, strided axes, Rader, Bluestein (one CTA and
# elementwise ends), multipass Rader
@pytest.mark.parametrize("shape,batch,axes", [
    ([16], 3, None), ([4096], 2, None), ([8192], 2, None), ([1 << 17], 1, None),
    ([360], 5, None), ([6000], 2, None), ([15015], 1, None), ([1009], 2, None), ([34], 7, None),
    ([2003], 1, None), ([40961], 1, None), ([20011], 1, None), ([48, 9], 2, None),
    ([30, 64, 17], 1, None), ([30, 64, 17], 1, [1]), ([12, 5, 9], 2, [1])])
@pytest.mark.parametrize("inverse", [False, True])
def test_words_in_words_out(shape, batch, axes, inverse):
    rng = np.random.default_rng(11)
    dims = [batch] + shape[::-1]
    z = value(words(rng.standard_normal(dims) + 1j * rng.standard_normal(dims)))
    ax = list(range(len(shape))) if axes is None else axes
    cfg = (w.FftConfig.new_nd(shape).with_batch(batch).with_axes(ax)
           .with_precision(w.FftPrecision.Df64).with_normalization(w.Normalization.NONE)
           .with_direction(w.FftDirection.Inverse if inverse else w.FftDirection.Forward))
    d = torch.from_numpy(words(z)).cuda()
    out = torch.empty_like(d)
    plan = w.FftPlan.c2c(cfg)
    plan.execute_checked(d, out)
    nax = [len(shape) - a for a in ax]
    n = np.prod([shape[a] for a in ax])
    ref = np.fft.ifftn(z, axes=nax) * n if inverse else np.fft.fftn(z, axes=nax)
    got = out.cpu().numpy()
    assert np.linalg.norm(value(got) - ref) <= 1e-14 * np.linalg.norm(ref)
    # a normalised pair: the low word below half an ulp of the high one
    assert (np.abs(got[..., 1]) <= np.abs(got[..., 0]) * 2.0 ** -23).all()
    if plan.supports_in_place():
        plan.execute_in_place(d)
        assert torch.equal(d, out)


def test_values_past_the_f32_range():
    z = np.zeros(64, dtype=np.complex128)
    z[0] = 3e38
    z[1] = 3e38
    d = torch.from_numpy(words(z)).cuda()
    out = torch.empty_like(d)
    w.FftPlan.c2c(w.FftConfig.new(64).with_precision(w.FftPrecision.Df64)).execute_checked(d, out)
    got = out.cpu().numpy()
    assert np.isposinf(got[0, 0]) and got[0, 1] == 0.0  # 6e38: an infinite high word, no NaN
    assert np.isfinite(got[32]).all()
    z[0] = np.nan
    d = torch.from_numpy(words(z)).cuda()
    w.FftPlan.c2c(w.FftConfig.new(64).with_precision(w.FftPrecision.Df64)).execute_checked(d, out)
    assert np.isnan(out.cpu().numpy()[..., 0]).all()
