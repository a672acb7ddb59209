"""Which launches a batch's steps take, by their number, and the route that
batches with a side beyond the resident strips keep: one launch a step, chunks
of steps replayed from a CUDA graph, bit for bit the persistent sweep."""
import numpy as np
import pytest

from mplb_b200.batch import Batch, CavitySpec

pytestmark = pytest.mark.gpu


def run(specs, precision, steps, **tuning):
    rng = np.random.default_rng(5)
    start = [[f + s * rng.uniform(-1, 1, (c.n, c.n)) for c in specs]
             for f, s in ((1.0, 0.01), (0.0, 0.02), (0.0, 0.02))]
    b = Batch(specs, precision)
    b.set_tuning(**tuning)
    b.init(*start)
    launches = []
    for n in steps:
        before = b.stats()["launches"]
        b.step(n)
        launches.append(b.stats()["launches"] - before)
    macro = b.macro()
    b.close()
    return macro, launches


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_steps_of_a_call_share_a_launch(gpu_lib, precision):
    specs = [CavitySpec(24, 100.0, 0.05)] * 8
    assert run(specs, precision, (3, 4, 128, 129))[1] == [3, 1, 1, 2]
    large = 401 if precision == "fp64" else 801
    specs = [CavitySpec(large, 100.0, 0.05), CavitySpec(24, 100.0, 0.05)]
    assert run(specs, precision, (4, 20), chunk=4)[1] == [4, 20]


@pytest.mark.parametrize("chunk", [2, 10])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_replayed_chunks_bitwise(gpu_lib, precision, chunk):
    large = 401 if precision == "fp64" else 801
    specs = [CavitySpec(n, 50.0 + n, 0.05) for n in (large, 3, 24, 97)]
    steps = (37, 20, 1, 10, 23)     # chunks, remainders, either array
    got, _ = run(specs, precision, steps, tile_nodes=64, persistent=0,
                 chunk=chunk, ctas_per_sm=4)
    want, _ = run(specs, precision, steps, tile_nodes=128, persistent=1,
                  chunk=2, ctas_per_sm=4)
    for g, w in zip(got, want):
        for x, y in zip(g, w):
            assert np.array_equal(x, y)
