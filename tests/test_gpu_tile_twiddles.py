"""The four-step twiddle of the fixed-length column tiles: tiles inside one
row, tiles of adjacent rows (their shared table) and tiles that straddle
rows, ragged last tiles, against numpy in 64 bits (the f32 bound, 2e-6)."""
import numpy as np
import pytest
import torch

import wgpufft_b200 as w

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,batch,axes", [
    ([1 << 15], 3, None), ([1 << 17], 2, None), ([1 << 19], 1, None), ([1 << 23], 1, None),
    ([3 << 16], 2, None),                       # a power-of-two column pass over a smooth line
    ([64, 4096], 2, [1]), ([96, 4096], 1, [1]), ([17, 2048], 2, [1]), ([24, 2048], 2, [1]),
    ([1000, 2048], 1, [1]), ([16, 8192], 1, [1]), ([128, 4096], 1, None)])
@pytest.mark.parametrize("inverse", [False, True])
def test_tiles(shape, batch, axes, inverse):
    cfg = (w.FftConfig.new_nd(shape).with_batch(batch)
           .with_direction(w.FftDirection.Inverse if inverse else w.FftDirection.Forward))
    if axes is not None:
        cfg = cfg.with_axes(axes)
    plan = w.FftPlan.c2c(cfg)
    g = torch.Generator().manual_seed(9)
    x = torch.randn([batch] + shape[::-1], dtype=torch.complex64, generator=g).cuda()
    out = torch.empty_like(x)
    plan.execute_checked(x, out)
    ax = list(range(len(shape))) if axes is None else axes
    dims = [len(shape) - a for a in ax]
    z = x.cpu().numpy().astype(np.complex128)
    ref = np.fft.ifftn(z, axes=dims) if inverse else np.fft.fftn(z, axes=dims)
    if inverse:
        ref = ref * np.prod([shape[a] for a in ax]) / np.prod(shape)
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 2e-6 * np.linalg.norm(ref)
    plan.execute_in_place(x)
    assert torch.equal(x, out)
