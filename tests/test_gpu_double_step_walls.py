"""Two steps to a launch where test_gpu_double_step.py has no case: a block
periodic in y, boundaries whose nodes take f = 0 (FDPeriodic), and boundary
nodes with populations that keep their initial values (a side without a
boundary), against one call a step, bit for bit."""
import dataclasses

import numpy as np
import pytest

import special_cases
from mplb_b200 import Solver, config

pytestmark = pytest.mark.gpu

# around the tile (64 or 32 wide, 26 high) and below it
SIZES = [(3, 3), (25, 4), (31, 26), (33, 28), (64, 53), (65, 54), (97, 79)]


@pytest.fixture(autouse=True)
def any_size(monkeypatch):
    monkeypatch.setenv("MPLB_B200_TWO_STEPS", "1")


def upright_channel(nx, ny, wall):
    """config.poiseuille turned by 90 degrees: walls left and right, periodic
    in y, force along y."""
    c = config.poiseuille(2, ny, nx, g_lattice=1e-5, wall=wall)
    turn = {"Left": "Bottom", "Right": "Top", "Top": "Right",
            "Bottom": "Left"}
    return dataclasses.replace(
        c, block_sizes=[(nx, ny)], accel=(0.0, c.accel[0], 0.0),
        boundaries=[dataclasses.replace(b, surface=turn[b.surface])
                    for b in c.boundaries],
        connections=[dataclasses.replace(x, from_surface=turn[x.from_surface],
                                         to_surface=turn[x.to_surface])
                     for x in c.connections])


def open_cavity(nx, ny, wall, missing):
    c = config.cavity(2, 64, 0.05, re=100.0, wall=wall)
    return dataclasses.replace(
        c, block_sizes=[(nx, ny)],
        boundaries=[b for b in c.boundaries if b.surface not in missing])


def cases(nx, ny):
    for wall in ("EQMDiffuseRefl", "HalfwayBounceBack"):
        yield upright_channel(nx, ny, wall)
        yield open_cavity(nx, ny, wall, ("Left",))
        yield open_cavity(nx, ny, wall, ("Top", "Right"))
    yield dataclasses.replace(special_cases.fdperiodic_box(2),
                              block_sizes=[(nx, ny)])


def run(case, calls):
    rng = np.random.default_rng(11)
    nx, ny, _ = case.size3(0)
    s = Solver(case)
    s.init_macro(0, 1.0 + 0.01 * rng.uniform(-1, 1, (1, ny, nx)),
                 0.02 * rng.uniform(-1, 1, (1, ny, nx)),
                 0.02 * rng.uniform(-1, 1, (1, ny, nx)))
    before = s.launch_count()
    for n in calls:
        s.stream_collision(n)
    launches = s.launch_count() - before
    s.update_macro_vars()
    out = [s.f(0)] + list(s.macro(0))
    s.stream_collision(1)
    out.append(s.f(0))
    s.close()
    return out, launches


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("size", SIZES)
def test_two_steps_a_launch_bitwise(gpu_lib, size, precision):
    for case in cases(*size):
        case = dataclasses.replace(case, precision=precision)
        want, single = run(case, (1,) * 9)
        for calls in ((9,), (4, 5)):
            got, launches = run(case, calls)
            for a, b in zip(got, want):
                assert np.array_equal(a, b, equal_nan=True), (case.case_name,
                                                              calls)
            # nine steps: four launches and a step, or one and two steps twice
            halos = 1 if case.connections else 0
            assert single == 9 * (1 + halos) + halos
            pairs = {(9,): 4, (4, 5): 3}[calls]
            steps = 9 - 2 * pairs
            assert launches == (pairs + len(calls) * halos +
                                steps * (1 + halos) + halos), calls
