"""The batch autotuner without a GPU: launches that are the same under several
tunings are timed once, and a cached choice holds for the kernels it was
measured with only."""
import json

import pytest

from mplb_b200 import batch as bmod
from mplb_b200.batch import CavitySpec, autotune, default_candidates


class FakeBatch:
    """Counts launches and device time as the native batch does; `resident`:
    persistent = 0 takes launches of many steps."""
    specs = [CavitySpec(64, 100.0, 0.05), CavitySpec(96, 100.0, 0.05)]
    precision = "fp32"
    total_nodes = sum(s.n * s.n for s in specs)

    def __init__(self, resident, ms):
        self.resident, self.ms = resident, ms
        self.tuned, self.timed = None, []
        self.count = dict(device_ms=0.0, node_updates=0, launches=0)

    def set_tuning(self, **t):
        self.tuned = t

    def init(self):
        self.timed.append(dict(self.tuned))

    def step(self, n):
        t = self.tuned
        one = self.resident and not t["persistent"]
        self.count["launches"] += 1 if one else -(-n // t["chunk"]) if \
            t["persistent"] else n
        self.count["device_ms"] += n * self.ms(t)

    def stats(self):
        return dict(self.count)


def test_resident_launches_are_timed_once(tmp_path):
    cache = str(tmp_path / "t.json")
    # a noise that would make the last of the equal candidates win
    noise = iter(range(100, 0, -1))
    b = FakeBatch(True, lambda t: 2.0 if t["persistent"] else
                  1.0 + 1e-3 * next(noise))
    best = autotune(b, steps=20, cache=cache)
    assert sum(not t["persistent"] for t in b.timed) == 1
    assert best["route"] == "resident"
    assert best["tuning"] == default_candidates()[0] == b.tuned
    assert len(best["all"]) == len(default_candidates())
    assert {r["route"] for r in best["all"]} == {"resident", "persistent"}


@pytest.mark.parametrize("fast", [0, 1])
def test_step_launches_are_timed_each(tmp_path, fast):
    b = FakeBatch(False, lambda t: (1.0 if t["persistent"] == fast else 2.0) +
                  1.0 / t["tile_nodes"])
    best = autotune(b, steps=20, cache=str(tmp_path / "t.json"))
    assert len(b.timed) == len(default_candidates())
    assert best["route"] == ("persistent" if fast else "steps")
    assert best["tuning"]["tile_nodes"] == 256


def test_a_choice_of_other_kernels_is_not_taken(tmp_path, monkeypatch):
    cache = str(tmp_path / "t.json")
    slow = FakeBatch(False, lambda t: 1.0 if t["persistent"] else 2.0)
    assert autotune(slow, steps=20, cache=cache)["route"] == "persistent"
    again = FakeBatch(True, lambda t: 1.0)
    assert autotune(again, steps=20, cache=cache)["route"] == "persistent"
    assert not again.timed
    # the same batch, built from other sources
    monkeypatch.setattr(bmod, "_kernel_build", lambda: "other")
    b = FakeBatch(True, lambda t: 2.0 if t["persistent"] else 1.0)
    assert autotune(b, steps=20, cache=cache)["route"] == "resident"
    assert len(json.load(open(cache))) == 2


def test_the_build_is_of_the_kernels():
    assert bmod._cache_key(FakeBatch(True, None)).endswith(
        bmod._kernel_build())
    assert len(bmod._kernel_build()) == 12
