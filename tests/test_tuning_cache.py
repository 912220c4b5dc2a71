"""The tuners' choices and their cache, on stand-ins for the plans (no GPU): the present launch shape is one of
the candidates, and what other kernels were tuned to, by an earlier cache or another generation
kernel, is not applied."""
import json

import pytest

from qmctoolscl_gb300 import batch, halton


@pytest.fixture(autouse=True)
def cache(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("QMCGB_TUNE_CACHE", str(path))
    monkeypatch.setattr(batch, "time_plan", lambda plan, stream, reps: plan.ms())
    return path


class NetPlan:
    default = (4, 1, 1 << 15)

    def __init__(self):
        self.shape = self.default

    def shape_class(self):
        return "net|coords2^20|d2^4|req2^2|gpu"

    def get_tuning(self):
        return self.shape

    def set_tuning(self, *shape):
        self.shape = shape

    def ms(self):
        return 1.0 if self.shape == self.default else 2.0


def test_default_shape_is_a_candidate(cache):
    plan = NetPlan()
    assert batch.autotune(plan, stream=object())[:3] == NetPlan.default
    assert plan.shape == NetPlan.default
    other = NetPlan()
    other.shape = (8, 16, 1 << 18)
    assert tuple(batch.autotune(other, stream=object())[:3]) == NetPlan.default == other.shape  # cached


def test_earlier_shapes_are_not_applied(cache):
    cache.write_text(json.dumps({NetPlan().shape_class(): [2, 16, 1 << 18, 0.5]}))
    plan = NetPlan()
    batch.autotune(plan, stream=object())
    assert plan.shape == NetPlan.default


class HaltonPlan(halton.HaltonBatch):
    """Fastest at share 1 with tables, at 0.5 without."""

    def __init__(self, tables):
        self.tables, self.coords, self.nreq, self.share = tables, 1 << 22, 1, 1.0

    def info(self):
        return {"has_tables": self.tables, "uses_tables": self.tables and self.share == 1.0}

    def prepare(self, stream=None):
        pass

    def set_fp64_share(self, share):
        self.share = share

    def ms(self):
        return abs(self.share - (1.0 if self.tables else 0.5))


def test_share_of_one_kernel_is_not_applied_to_the_other(cache):
    for tables, share in ((False, 0.5), (True, 1.0), (False, 0.5), (True, 1.0)):
        plan = HaltonPlan(tables)
        assert plan.tune(stream=object())[0] == share == plan.share


def test_earlier_shares_are_not_applied(cache):
    cache.write_text(json.dumps({"halton|coords2^22|req2^0|%s" % batch._device_name(): [0.5, 1.0]}))
    plan = HaltonPlan(True)
    assert plan.tune(stream=object())[0] == 1.0 == plan.share
