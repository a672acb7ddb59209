"""The step's launch orders and staged segments: a block on either side of the
size from which the walls no longer run first steps as the two-part step does
(shell rows in a launch of their own), bit for bit; the staged FP16 interior
with one to eight segments a warp, ragged rows among them, follows FP64; the
device time of chained single-step calls is one step's."""
import numpy as np
import pytest

from mplb_b200 import Solver, config

pytestmark = pytest.mark.gpu


def box(size, precision):
    dim = len(size)
    case = config.cavity(dim, 64, 0.05, re=100.0, precision=precision)
    case.block_sizes = [tuple(size)]
    return case


def start(solver, case, seed=3):
    rng = np.random.default_rng(seed)
    shape = tuple(reversed(case.size3(0)))
    u = [0.02 * rng.uniform(-1, 1, shape) for _ in range(case.space_dim)]
    solver.init_macro(0, 1.0 + 0.01 * rng.uniform(-1, 1, shape), *u)


# FP64 arrays of 96 and 108 MB (3D), 94 and 110 MB (2D): the line is 100 MB
@pytest.mark.parametrize("size", [(66, 67, 68), (70, 69, 70), (801, 811),
                                  (870, 873)])
def test_orders_bitwise(gpu_lib, size):
    case = box(size, "fp64")
    got = []
    for parts in (False, True):
        s = Solver(case)
        start(s, case)
        for _ in range(5):
            if parts:
                s._check(s.lib.mplbgpu_step_begin(s.h))
                s._check(s.lib.mplbgpu_step_finish(s.h))
            else:
                s.stream_collision()
        s.update_macro_vars()
        got.append(s.macro(0))
        s.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


# 1, 2, 4 and 8 segments a warp (up to 2,960 / 5,920 / 11,840 segments and
# more), rows of one to three segments
@pytest.mark.parametrize("size", [(40, 40, 40), (65, 50, 50), (129, 60, 60),
                                  (64, 112, 112), (190, 70, 70), (64, 4000),
                                  (130, 9000)])
def test_staged_segments_follow_fp64(gpu_lib, size):
    got = {}
    for precision in ("fp64", "fp16"):
        case = box(size, precision)
        s = Solver(case)
        start(s, case)
        s.stream_collision(6)
        s.update_macro_vars()
        got[precision] = s.macro(0)
        s.close()
    # stochastic rounding of half precision: 2^-11 of a population a step, as
    # much as 20 % of the smallest velocities here; a misplaced segment is off
    # by the velocities themselves
    for a, b in zip(got["fp16"][1:], got["fp64"][1:]):
        assert np.linalg.norm(a - b) < 0.05 * np.linalg.norm(b)
    assert np.abs(got["fp16"][0] - got["fp64"][0]).max() < 0.01


def test_chained_calls_time_one_step(gpu_lib):
    case = box((48, 48, 48), "fp64")
    s = Solver(case)
    start(s, case)
    s.stream_collision(400)
    per_step = s.last_step_ms() / 400
    for _ in range(200):
        s.stream_collision()
    last = s.last_step_ms()
    assert 0.2 * per_step < last < 20 * per_step
    s.update_macro_vars()
    s.stream_collision(400)
    assert s.last_step_ms() > 40 * per_step
    s.close()
