"""What bench.py reports where steps have no cost of their own: a system without
a consumer pays per rebuild and per call, whatever number of steps lies between,
so its probe gives that cost and none per step; and a phase that was not timed
has no roofline.  CPU only, on the model clock of test_bench_probe."""
import warnings

import pytest

import bench
from test_bench_probe import ModelClock, ModelSystem, model_events  # noqa: F401


class StretchSystem(ModelSystem):
    """Each rebuild costs `extra` with the stretch before it, each call
    `per_call`, a step nothing."""

    def step(self, n):
        ms = self.per_call
        for _ in range(n):
            self.k += 1
            if self.k % self.period == 0:
                self.rebuilds += 1
                ms += self.extra
        ModelClock.now += ms


@pytest.mark.parametrize("period", [7, 11, 25])
def test_stretches_have_a_cost_per_rebuild(model_events, period):  # noqa: F811
    s = StretchSystem(light=0.0, extra=0.085, per_call=0.03, period=period)
    out = bench.rebuild_probe(s, stream=None, min_rebuilds=20, stretches=True)
    assert out["rebuilds"] >= 20
    assert out["ms_per_light_step"] is None and out["ms_per_rebuild_step"] is None
    assert out["ms_per_rebuild_cycle"] == pytest.approx(0.085, rel=1e-9)
    total = ModelClock.now
    assert out["ms_per_step_at_rebuild_rate"] == pytest.approx(total / out["steps"], rel=1e-9)
    assert out["neighbor_builds_per_s"] == pytest.approx(out["rebuilds"] / total * 1e3, rel=1e-9)


def test_no_roofline_without_a_timed_launch():
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert bench.phase_roofline("k", "force", 1e6, 0.0, 0, 6537.3, "measured", None) is None
    r = bench.phase_roofline("k", "force", 6.5373e9, 4.0, 2, 6537.3, "measured", None)
    assert r["mean_launch_ms"] == 2.0 and r["launches"] == 2
    assert r["frac"] == pytest.approx(0.5, rel=1e-12)
