"""The workspace of a C2R plan holds the packed spectrum whatever route its
strided axes take (a Rader or one-CTA Bluestein axis once left it unsized,
and the plan wrote through a null workspace)."""
import numpy as np
import pytest

import wgpufft_b200 as w

SHAPES = [[64, 17], [64, 457], [64, 1009], [30, 34], [96, 60], [48, 17, 34]]


def config(shape, kind):
    cfg = w.FftConfig.new_nd(shape)
    return cfg.with_direction(w.FftDirection.Inverse) if kind == w.FftTransformKind.C2r else cfg


@pytest.mark.parametrize("shape", SHAPES)
def test_workspace_holds_the_spectrum(shape):
    kind = w.FftTransformKind.C2r
    plan = w.FftPlan.plan_only(config(shape, kind), kind)
    packed = (shape[0] // 2 + 1) * int(np.prod(shape[1:])) * 8
    bufs = {s["dst"] for s in plan.diagnostics()["stages"]} - {1}
    assert plan.workspace_size_bytes() >= packed * len(bufs)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_real_round_trip(shape):
    import torch
    x = np.random.default_rng(3).standard_normal(shape[::-1]).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    spec = torch.empty(shape[:0:-1] + [shape[0] // 2 + 1], dtype=torch.complex64, device="cuda")
    back = torch.empty_like(d)
    w.FftPlan.r2c(config(shape, w.FftTransformKind.R2c)).execute_checked(d, spec)
    w.FftPlan.c2r(config(shape, w.FftTransformKind.C2r)).execute_checked(spec, back)
    ref = np.fft.rfftn(x.astype(np.float64))
    assert np.linalg.norm(spec.cpu().numpy() - ref) <= 2e-6 * np.linalg.norm(ref)
    assert np.linalg.norm(back.cpu().numpy() - x) <= 4e-6 * np.linalg.norm(x)
