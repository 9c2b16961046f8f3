"""Which settings the autotuner leaves applied, from made-up times (CPU)."""
import pytest


@pytest.fixture
def tuned(monkeypatch):
    from pptk_b200 import autotune
    knobs = {"lane_span": 1024, "warm_bound": 1, "topk_min": 0, "warm_mult": 2}
    monkeypatch.setattr(autotune.N, "tune_get", lambda name: knobs[name])
    monkeypatch.setattr(autotune.N, "tune_set", lambda name, v: knobs.__setitem__(name, v))
    bucket = [None]

    def run(seconds):
        monkeypatch.setattr(autotune, "_time", lambda *a: seconds(bucket[0], **knobs))
        out = autotune.tune(lambda: None, lambda b: bucket.__setitem__(0, b), sync=lambda: None)
        assert out["bucket"] == bucket[0]
        return out, knobs

    return run


def test_noise_does_not_move_a_setting(tuned):
    # every setting runs the same kernels: times differ by a percent
    noise = {-1: 0.99, 64: 1.0, 256: 0.995, 1024: 1.01}
    out, knobs = tuned(lambda bucket, lane_span, warm_mult, **_: noise[lane_span] * (0.99 if warm_mult == 3 else 1.0))
    assert knobs == {"lane_span": 1024, "warm_bound": 1, "topk_min": 0, "warm_mult": 2}
    assert out["lane_span"] == 1024 and out["warm_mult"] == 2


def test_a_clearly_faster_setting_is_taken(tuned):
    out, knobs = tuned(lambda bucket, lane_span, warm_mult, warm_bound, **_:
                       1.0 - 0.1 * (bucket == 32) - 0.1 * (lane_span == 256) - 0.1 * (warm_mult == 3)
                       - 0.1 * (warm_bound == 0))
    assert out["bucket"] == 32 and knobs["lane_span"] == 256
    assert knobs["warm_mult"] == 3 and knobs["warm_bound"] == 0 and knobs["topk_min"] == 0
