"""The launch-shape sweeps of the autotuner on the CPU, with timings of a fake
force field: the pair kernel's own rules take part and stay unless beaten by
more than the noise, no residency beyond the register budget is tried, and
cached results of another kernel are not taken over."""

import json
from types import SimpleNamespace

import pytest

from heddle_b200 import _native as N
from heddle_b200 import autotune as T

SPEC = SimpleNamespace(n=3000, grid=(36, 36, 36), r_cut_coul=17.0, alpha=0.2, order=4)


@pytest.fixture
def tuned(monkeypatch, tmp_path):
    """tune(times) with times(param values) -> ms; returns (result, values tried)."""

    def tune(times, cache=None):
        tried = []

        class Fake:
            def __init__(self):
                self.h, self.shape = None, {}
                self.lib = SimpleNamespace(hb_forcefield_set_launch=self.set)

            def set(self, h, param, value):
                self.shape[param] = value
                tried.append((param, value))
                return 0

            def close(self):
                pass

        monkeypatch.setattr(T, "ForceField", SimpleNamespace(from_spec=lambda *a, **k: Fake()))
        monkeypatch.setattr(T, "_time_steps", lambda ctx, s, ff, *a: times(ff.shape))
        return T.tune_skin(None, None, SPEC, None, {}, cache=cache), tried

    return tune


def by(param, table):
    return lambda shape: table.get(shape.get(param, 0), 1.0)


def test_rules_stay_when_nothing_is_faster(tuned):
    r, tried = tuned(lambda shape: 1.0)
    assert r["pair_blocks_per_sm"] == 0 and r["pair_chunk"] == 0
    blocks = {v for p, v in tried if p == N.HB_LAUNCH_PAIR_BLOCKS_PER_SM}
    assert blocks == {0, 3, 4, 5, 6}  # the register budget is cut for 5 and 6
    assert {0, 1} <= {v for p, v in tried if p == N.HB_LAUNCH_PAIR_CHUNK}


def test_noise_does_not_replace_a_rule(tuned):
    r, _ = tuned(by(N.HB_LAUNCH_PAIR_BLOCKS_PER_SM, {0: 1.0, 6: 0.99}))
    assert r["pair_blocks_per_sm"] == 0


def test_a_faster_shape_is_taken(tuned):
    r, tried = tuned(by(N.HB_LAUNCH_PAIR_CHUNK, {0: 1.0, 1: 0.9}))
    assert r["pair_chunk"] == 1
    assert [v for p, v in tried if p == N.HB_LAUNCH_PAIR_CHUNK][-1] == 1


def test_forms_take_zero_as_a_value(tuned):
    r, _ = tuned(by(N.HB_LAUNCH_GATHER_FORM, {1: 1.0, 0: 0.995}))
    assert r["gather_form"] == 0


def test_cached_results_of_another_kernel_are_not_used(tuned, tmp_path):
    cache = tmp_path / "tuned.json"
    cache.write_text(json.dumps({"n3000-grid36x36x36-rc17.000": {"best_A": 1.0, "pair_blocks_per_sm": 8}}))
    r, tried = tuned(lambda shape: 1.0, cache)
    assert tried and r["pair_blocks_per_sm"] == 0
    again, tried = tuned(lambda shape: 1.0, cache)
    assert not tried and again == r
