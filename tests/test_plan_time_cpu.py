"""Building a plan costs what its tables cost."""
import time

import wgpufft_b200 as w


def best_ms(precision):
    cfg = w.FftConfig.new(1 << 24).with_precision(precision)
    times = []
    for _ in range(20):
        t = time.perf_counter()
        w.FftPlan.plan_only(cfg, w.FftTransformKind.C2c)
        times.append(time.perf_counter() - t)
    return min(times) * 1e3


def test_tile_twiddles_take_no_roots_of_their_own():
    """The f32 tables beside the f64 plan's come from roots that both have
    (1.25 times the f64 plan's time; 2.3 with roots of their own)."""
    assert best_ms(w.FftPrecision.F32) <= 1.7 * best_ms(w.FftPrecision.F64)
