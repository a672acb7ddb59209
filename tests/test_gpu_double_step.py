"""Two steps to a launch (2D blocks, several steps in a call) against one call a
step, bit for bit: sizes around the tile (64 or 32 wide, 26 high) and below it,
odd and even step counts, diffuse and halfway walls, a moving lid, a wall
velocity per node, one periodic axis with a body force, both forms."""
import dataclasses

import numpy as np
import pytest

from mplb_b200 import Solver, config

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def any_size(request, monkeypatch):
    """Small blocks take the path too (by themselves only those beyond the L2
    cache do)."""
    if "default" not in request.node.name:
        monkeypatch.setenv("MPLB_B200_TWO_STEPS", "1")

SIZES = [(3, 3), (4, 25), (31, 26), (32, 27), (33, 28), (63, 52), (64, 53),
         (65, 54), (66, 3), (97, 79), (130, 26), (200, 131)]


def cases(nx, ny):
    for wall in ("EQMDiffuseRefl", "HalfwayBounceBack"):
        yield dataclasses.replace(
            config.cavity(2, 64, 0.05, re=100.0, wall=wall,
                          order=("Top", "Left", "Bottom", "Right")),
            block_sizes=[(nx, ny)])
        yield config.poiseuille(2, nx, ny, g_lattice=1e-5, wall=wall)


def run(case, calls, velocity=None):
    rng = np.random.default_rng(7)
    nx, ny, _ = case.size3(0)
    s = Solver(case)
    s.init_macro(0, 1.0 + 0.01 * rng.uniform(-1, 1, (1, ny, nx)),
                 0.02 * rng.uniform(-1, 1, (1, ny, nx)),
                 0.02 * rng.uniform(-1, 1, (1, ny, nx)))
    if velocity is not None:
        ex = s.boundary_extent(velocity)
        s.set_boundary_velocity(velocity, *(
            0.02 * rng.uniform(-1, 1, (ex[2], ex[1], ex[0]))
            for _ in range(2)))
    for n in calls:
        s.stream_collision(n)
    s.update_macro_vars()
    out = [s.f(0)] + list(s.macro(0))
    s.stream_collision(1)       # from the arrays and halos the calls left
    out.append(s.f(0))
    s.close()
    return out


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("size", SIZES)
def test_two_steps_a_launch_bitwise(gpu_lib, size, precision):
    for case in cases(*size):
        case = dataclasses.replace(case, precision=precision)
        for calls in ((3,), (8,), (5, 4, 1, 7)):
            got = run(case, calls)
            want = run(case, (1,) * sum(calls))
            for a, b in zip(got, want):
                assert np.array_equal(a, b), (case.case_name, calls)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_per_node_walls_bitwise(gpu_lib, precision):
    for wall in ("EQMDiffuseRefl", "HalfwayBounceBack"):
        case = dataclasses.replace(
            config.cavity(2, 64, 0.05, re=100.0, wall=wall,
                          precision=precision), block_sizes=[(70, 40)])
        for a, b in zip(run(case, (9,), 2), run(case, (1,) * 9, 2)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision, size", [("fp64", (900, 901)),
                                             ("fp32", (1301, 1100))])
def test_default_above_l2(gpu_lib, precision, size):
    """Blocks on the default's side of the line: 117 and 103 MB of
    populations."""
    case = dataclasses.replace(
        config.poiseuille(2, *size, g_lattice=1e-5, wall="EQMDiffuseRefl"),
        precision=precision)
    s = Solver(case)
    s.init_uniform()
    launches = s.launch_count()
    s.stream_collision(9)
    # first halos, four launches of two steps, halos, one step and its halos
    assert s.launch_count() - launches == 8
    s.close()
    for a, b in zip(run(case, (9,)), run(case, (1,) * 9)):
        assert np.array_equal(a, b)
