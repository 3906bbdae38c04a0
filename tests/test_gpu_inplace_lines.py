"""The in-place mixed-radix kernels at the edges of their ranges: the
shortest and longest lines of one CTA, ragged last tiles, fewer lines than a
tile, rows, columns and transposed stores, Rader, Bluestein and packed real
transforms, f32 and f64, against numpy in 64 bits and against the ping-pong
engine (which a plan with an explicit lines_per_block runs).

Bounds: an N-point transform of s stages has a 2-norm error of a few units
of the last place per stage; 2e-6 (f32) and 1e-14 (f64) are the bounds every
route of the library is held to."""
import numpy as np
import pytest
import torch

import wgpufft_b200 as w

pytestmark = pytest.mark.gpu
TOL = {"f32": 2e-6, "f64": 1e-14}
PREC = {"f32": w.FftPrecision.F32, "f64": w.FftPrecision.F64}
CT = {"f32": torch.complex64, "f64": torch.complex128}


def run(shape, batch, axes, prec, inverse, tuning=None):
    cfg = (w.FftConfig.new_nd(shape).with_batch(batch).with_precision(PREC[prec])
           .with_direction(w.FftDirection.Inverse if inverse else w.FftDirection.Forward))
    if axes is not None:
        cfg = cfg.with_axes(axes)
    if tuning is not None:
        cfg = cfg.with_tuning(tuning)
    plan = w.FftPlan.c2c(cfg)
    g = torch.Generator().manual_seed(5)
    x = torch.randn([batch] + shape[::-1], dtype=CT[prec], generator=g).cuda()
    out = torch.empty_like(x)
    plan.execute_checked(x, out)
    return plan, x, out


def check(shape, batch, axes, prec, inverse):
    plan, x, out = run(shape, batch, axes, prec, inverse)
    ax = range(len(shape)) if axes is None else axes
    dims = [len(shape) - a for a in ax]
    z = x.cpu().numpy().astype(np.complex128)
    ref = np.fft.ifftn(z, axes=dims) if inverse else np.fft.fftn(z, axes=dims)
    got = out.cpu().numpy()
    if inverse and axes is not None:  # the library scales by its whole shape
        ref = ref * np.prod([shape[a] for a in ax]) / np.prod(shape)
    assert np.linalg.norm(got - ref) <= TOL[prec] * np.linalg.norm(ref)
    plan.execute_in_place(x)
    assert torch.equal(x, out)
    return plan


# 18..30030: two to five stages, every radix, one CTA up to about 28,900
# (f32) and 14,400 (f64) points
@pytest.mark.parametrize("n,batch,prec", [
    (18, 1, "f32"), (18, 1001, "f32"), (22, 7, "f32"), (26, 513, "f32"), (35, 100, "f32"),
    (96, 85, "f32"), (143, 33, "f32"), (169, 50, "f32"), (182, 91, "f32"), (1001, 9, "f32"),
    (2187, 5, "f32"), (3125, 3, "f32"), (13860, 2, "f32"), (15625, 2, "f32"), (16807, 2, "f32"),
    (28800, 2, "f32"), (28812, 1, "f32"), (28875, 3, "f32"), (30030, 2, "f32"),
    (18, 300, "f64"), (330, 7, "f64"), (7000, 3, "f64"), (14336, 2, "f64"), (14406, 2, "f64"),
    (15015, 1, "f64")])
@pytest.mark.parametrize("inverse", [False, True])
def test_rows(n, batch, prec, inverse):
    check([n], batch, None, prec, inverse)


# strided axes: fewer adjacent lines than a tile, one more than a tile, long
# columns of narrow tiles
@pytest.mark.parametrize("shape,axes,batch,prec", [
    ([2, 18], [1], 3, "f32"), ([3, 100], [1], 2, "f32"), ([17, 60], [1], 1, "f32"),
    ([33, 1080], [1], 1, "f32"), ([5, 1848], [1], 2, "f32"), ([15, 2002], [1], 1, "f32"),
    ([16, 2002], [1], 1, "f32"), ([3, 14000], [1], 1, "f32"), ([7, 30, 11], [1], 2, "f32"),
    ([40, 30, 21], None, 2, "f32"), ([3, 100], [1], 2, "f64"), ([9, 1000], [1], 1, "f64"),
    ([40, 30, 21], [2, 0], 1, "f64"), ([60, 36], [1, 0], 3, "f32")])
@pytest.mark.parametrize("inverse", [False, True])
def test_columns(shape, axes, batch, prec, inverse):
    check(shape, batch, axes, prec, inverse)


# four-step lines: columns with the twiddle on store, rows stored lines first
@pytest.mark.parametrize("n,batch,prec", [(30030, 2, "f32"), (90000, 1, "f32"), (450450, 1, "f32"),
                                          (6250000, 1, "f32"), (100100, 1, "f64")])
def test_four_step(n, batch, prec):
    check([n], batch, None, prec, False)


@pytest.mark.parametrize("shape,axes,batch,prec", [
    ([17], None, 1, "f32"), ([17], None, 777, "f32"), ([19], None, 100, "f32"),
    ([8191], None, 3, "f32"), ([2003 - 2], None, 4, "f32"), ([337], None, 5, "f64"),
    ([8191], None, 2, "f64"), ([3, 17], [1], 2, "f32"), ([20, 1009], [1], 1, "f32"),
    ([5, 6301], [1], 1, "f32"), ([9, 337], [1], 2, "f64")])
@pytest.mark.parametrize("inverse", [False, True])
def test_rader(shape, axes, batch, prec, inverse):
    check(shape, batch, axes, prec, inverse)


@pytest.mark.parametrize("shape,axes,batch,prec", [
    ([34], None, 1, "f32"), ([47], None, 500, "f32"), ([2003], None, 5, "f32"),
    ([4099], None, 3, "f32"), ([13997], None, 2, "f32"), ([14398], None, 2, "f32"),
    ([14561], None, 1, "f32"), ([94], None, 11, "f64"), ([6997], None, 2, "f64"),
    ([3, 34], [1], 2, "f32"), ([18, 457], [1], 2, "f32"), ([2, 7001], [1], 1, "f32"),
    ([5, 457], [1], 2, "f64")])
@pytest.mark.parametrize("inverse", [False, True])
def test_bluestein(shape, axes, batch, prec, inverse):
    check(shape, batch, axes, prec, inverse)


# the ping-pong engine on the same lines
@pytest.mark.parametrize("shape,axes,batch,prec", [
    ([360], None, 9, "f32"), ([1009], None, 5, "f32"), ([94], None, 9, "f32"),
    ([12, 90], [1], 3, "f32"), ([12, 29], [1], 3, "f64"), ([9, 94, 5], [1], 1, "f32"),
    ([30030], None, 1, "f32")])
def test_against_the_ping_pong_engine(shape, axes, batch, prec):
    _, _, a = run(shape, batch, axes, prec, False)
    _, _, b = run(shape, batch, axes, prec, False, w.FftTuning().with_lines_per_block(1))
    d = torch.linalg.vector_norm((a - b).flatten()) / torch.linalg.vector_norm(b.flatten())
    assert float(d) <= 2 * TOL[prec]


# even lengths with a half that is not a power of two: packed pairs in one
# CTA (R2C holds two buffers, C2R one)
@pytest.mark.parametrize("shape,batch,prec", [
    ([36], 1, "f32"), ([36], 999, "f32"), ([90], 77, "f32"), ([1920], 5, "f32"),
    ([28800], 2, "f32"), ([28812], 2, "f32"), ([30030], 1, "f32"), ([57600], 1, "f32"),
    ([60, 7], 2, "f32"), ([1000], 3, "f64"), ([14400], 1, "f64"), ([42, 20, 9], 1, "f64")])
def test_real(shape, batch, prec):
    cfg = w.FftConfig.new_nd(shape).with_batch(batch).with_precision(PREC[prec])
    rt = torch.float32 if prec == "f32" else torch.float64
    x = torch.randn([batch] + shape[::-1], dtype=rt, generator=torch.Generator().manual_seed(7)).cuda()
    spec = torch.empty([batch] + shape[:0:-1] + [shape[0] // 2 + 1], dtype=CT[prec], device="cuda")
    back = torch.empty_like(x)
    w.FftPlan.r2c(cfg).execute_checked(x, spec)
    w.FftPlan.c2r(cfg.with_direction(w.FftDirection.Inverse)).execute_checked(spec, back)
    ref = np.fft.rfftn(x.cpu().numpy().astype(np.float64), axes=range(1, len(shape) + 1))
    assert np.linalg.norm(spec.cpu().numpy() - ref) <= TOL[prec] * np.linalg.norm(ref)
    err = torch.linalg.vector_norm((back - x).flatten()) / torch.linalg.vector_norm(x.flatten())
    assert float(err) <= 2 * TOL[prec]
