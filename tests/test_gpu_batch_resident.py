"""Batched cavities held in shared memory (several steps per launch) against
the persistent one-step sweep of the same batch, bit for bit: sides at the
edges of what one CTA, one cluster and overlapping strips hold, step counts
that end on either kind of step and in either array, lone cavities (large
clusters) and crowded batches (small ones)."""
import numpy as np
import pytest

from mplb_b200.batch import Batch, CavitySpec

pytestmark = pytest.mark.gpu

# sides: 3, the slots of a quarter, half and whole SM (28 / 40 / 56 / 80 in
# one of the two forms), clusters, strips (250 on), the largest
SIDES = {"fp64": [3, 28, 29, 40, 41, 56, 57, 97, 128, 199, 250, 400],
         "fp32": [3, 40, 41, 56, 57, 80, 81, 133, 200, 256, 317, 800]}


def fields(specs, seed):
    rng = np.random.default_rng(seed)
    out = [[], [], []]
    for s in specs:
        out[0].append(1.0 + 0.01 * rng.uniform(-1, 1, (s.n, s.n)))
        for c in (1, 2):
            out[c].append(0.02 * rng.uniform(-1, 1, (s.n, s.n)))
    return out


def moments(specs, precision, persistent, steps, start):
    b = Batch(specs, precision)
    b.set_tuning(tile_nodes=128, persistent=persistent, chunk=2, ctas_per_sm=4)
    b.init(*start)
    for n in steps:
        b.step(n)
    got = b.macro()
    b.close()
    return got


def check(specs, precision, steps, seed):
    start = fields(specs, seed)
    got = moments(specs, precision, 0, steps, start)
    want = moments(specs, precision, 1, steps, start)
    for s, g, w in zip(specs, got, want):
        for x, y in zip(g, w):
            assert np.array_equal(x, y), (s.n, precision, steps)


@pytest.mark.parametrize("steps", [(4,), (5,), (33, 3, 6), (131, 130)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sides_bitwise(gpu_lib, precision, steps):
    specs = [CavitySpec(n, 50.0 + n, 0.02 + 0.0001 * n)
             for n in SIDES[precision]]
    check(specs, precision, steps, 1)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [24, 64, 100, 211])
def test_alone_and_crowded_bitwise(gpu_lib, precision, n):
    check([CavitySpec(n, 100.0, 0.05)], precision, (9,), n)
    check([CavitySpec(n, 60.0 + k, 0.05) for k in range(400 if n < 200 else 90)],
          precision, (9, 4), n)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_run_drops_and_replans(gpu_lib, precision):
    """Cavities that converge leave; the rest, planned again, end with the
    steps, residuals and fields of the one-step sweep."""
    specs = [CavitySpec(16, 5.0, 0.02)] * 40 + [CavitySpec(60, 300.0, 0.08)] * 3
    got = {}
    for persistent in (0, 1):
        b = Batch(specs, precision)
        b.set_tuning(tile_nodes=64, persistent=persistent, chunk=4,
                     ctas_per_sm=4)
        b.init()
        got[persistent] = b.run(max_steps=1200, check_period=100,
                                criterion=1e-4) + (b.macro(),)
        b.close()
    for k in range(3):
        assert np.array_equal(got[0][k], got[1][k])
    assert got[0][2][0] and got[0][0][0] < got[0][0][-1]
    for g, w in zip(got[0][3], got[1][3]):
        for x, y in zip(g, w):
            assert np.array_equal(x, y)
