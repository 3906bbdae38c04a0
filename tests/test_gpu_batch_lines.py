"""The batch kernels at the edges of their ranges: lines of one CTA (tiny,
smooth, Rader, Bluestein) up to the longest that fits, the shortest
and longest lines of the two- and three-pass routes, one ragged column or
row, passes of two to four stages, prime powers, and Bluestein lines whose
convolution is odd, against numpy in 64 bits (bound of every f32 route:
2e-6 in the 2-norm)."""
import numpy as np
import pytest
import torch

import wgpufft_b200 as w
from wgpufft_b200 import workloads

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 13, 16, 17, 18, 19, 23, 34, 94, 97, 337, 1000, 1409, 2521, 2731, 2777, 2801, 5600, 5616, 2816, 3024, 4394, 6561, 6655, 14641, 15625, 16807, 28561, 65536, 131072, 262144, 250000,
           200200, 1409, 1418, 2837, 2999, 8200, 34607, 65521, 65537, 99990, 116033]


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("repeat", [1, 3])
def test_long_lines(inverse, repeat):
    lengths = np.array(LENGTHS * repeat)
    off = workloads.packed_offsets(lengths)
    x = workloads.normal_complex(int(lengths.sum()), 17)
    d = torch.from_numpy(x).cuda()
    out = torch.empty_like(d)
    b = w.FftBatch(lengths, off, direction=w.FftDirection.Inverse if inverse else w.FftDirection.Forward)
    b.execute(d, out)
    y = out.cpu().numpy()
    for n, o in zip(lengths, off):
        z = x[o:o + n].astype(np.complex128)
        ref = np.fft.ifft(z) if inverse else np.fft.fft(z)
        assert np.linalg.norm(y[o:o + n] - ref) <= 2e-6 * np.linalg.norm(ref), n
    b.execute(d, d)  # in place
    assert torch.equal(d, out)


def test_a_line_alone_equals_the_same_line_among_others():
    n = 30011
    x = torch.from_numpy(workloads.normal_complex(n, 3)).cuda()
    alone = torch.empty_like(x)
    w.FftBatch([n], [0]).execute(x, alone)
    lengths = np.array([20000, n, 65521, 4096])
    off = workloads.packed_offsets(lengths)
    d = torch.zeros(int(lengths.sum()), dtype=torch.complex64, device="cuda")
    d[off[1]:off[1] + n] = x
    out = torch.empty_like(d)
    w.FftBatch(lengths, off).execute(d, out)
    assert torch.equal(out[off[1]:off[1] + n], alone)


@pytest.mark.parametrize("n", [5003, 6000, 15015, 65521])
@pytest.mark.parametrize("count", [1, 7, 40])
def test_few_long_lines_take_one_task_a_cta(n, count):
    """As long as a phase has fewer tasks than CTAs fit (two an SM at least),
    every task has a CTA of its own."""
    lengths = np.full(count, n)
    off = workloads.packed_offsets(lengths)
    x = workloads.normal_complex(int(lengths.sum()), n)
    d = torch.from_numpy(x).cuda()
    out = torch.empty_like(d)
    b = w.FftBatch(lengths, off)
    b.execute(d, out)
    ref = np.fft.fft(x.reshape(count, n).astype(np.complex128))
    y = out.cpu().numpy().reshape(count, n)
    assert np.all(np.linalg.norm(y - ref, axis=1) <= 2e-6 * np.linalg.norm(ref, axis=1))
    info = b.diagnostics()
    most = max(info["long_tasks"])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert info["long_grid"] >= min(most, 2 * sms)


def test_tasks_dealt_out_and_from_the_queue_agree():
    """Either side of the count from which tasks come from the work queue:
    the same lines, bit for bit (a line's arithmetic depends on neither)."""
    n = 6000
    few, many = 9000, 10000
    g = torch.Generator(device="cuda").manual_seed(5)
    d = torch.randn(many * n, dtype=torch.complex64, device="cuda", generator=g)
    grids, outs = [], []
    for count in (few, many):
        b = w.FftBatch(np.full(count, n), np.arange(count) * n)
        info = b.diagnostics()
        grids.append(info["long_tasks"][0] / info["long_grid"])
        out = torch.empty_like(d[:count * n])
        b.execute(d[:count * n], out)
        outs.append(out)
    assert grids[0] <= 32 < grids[1], grids
    assert torch.equal(outs[0], outs[1][:few * n])


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("count", [1, 3, 150, 1000, 40000])
@pytest.mark.parametrize("n", [13, 16, 17, 32, 122, 1009, 2600])
def test_tasks_of_short_lines(n, count, inverse):
    """One task, a task for every CTA, and more than that (the queue); few
    lines are spread over the chip, not packed into full tasks."""
    if n * count > 1 << 24:
        pytest.skip("more points than this needs")
    b = w.FftBatch(np.full(count, n), np.arange(count) * n,
                   direction=w.FftDirection.Inverse if inverse else w.FftDirection.Forward)
    x = workloads.normal_complex(count * n, n)
    d = torch.from_numpy(x).cuda()
    out = torch.empty_like(d)
    for _ in range(2):  # a second call finds the queue as it must be
        out.zero_()
        b.execute(d, out)
    z = x.reshape(count, n).astype(np.complex128)
    ref = np.fft.ifft(z) if inverse else np.fft.fft(z)
    y = out.cpu().numpy().reshape(count, n)
    assert np.all(np.linalg.norm(y - ref, axis=1) <= 2e-6 * np.linalg.norm(ref, axis=1))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert b.diagnostics()["cta_tasks"] >= min(count, 2 * sms, count * n // 1500)


@pytest.mark.parametrize("n", [2, 16, 17, 18, 19, 47, 2731, 2777, 5600])
def test_tasks_keep_their_share_of_shared_memory(n):
    """A full task of any length fits a quarter of an SM (44 KiB of lines)."""
    b = w.FftBatch(np.full(40000, n), np.arange(40000) * n)
    assert 0 < b.diagnostics()["cta_smem"] <= 44 * 1024
