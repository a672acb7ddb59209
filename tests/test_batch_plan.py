"""How batched cavities are cut for shared memory (batch_plan.h), compiled here
and asked for every side the strips take: the CTAs of a form fit on an SM
together, a strip fits its cluster's slots, and a cavity's strips store each of
its rows once, from rows whose edges are far enough away."""
import os
import subprocess

import pytest

from mplb_b200 import build

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "batch_plan.h"
using namespace mplb;
int main() {
    char what[16];
    int f64, n, count;
    while (scanf("%15s %d %d %d", what, &f64, &n, &count) == 4) {
        if (!strcmp(what, "form")) {
            printf("%d %d\n", ResidentSlots(f64, n), ResidentSmem(f64, n));
            continue;
        }
        ResidentHeld held;
        for (int h = 0; h < 3; h++)
            for (int r = 0; r < kNumResidentRanks; r++)
                held.at[h][r] = !strcmp(what, "plan") ||
                                (!strcmp(what, "portable") &&
                                 kResidentRanks[r] <= 8) ||
                                (!strcmp(what, "single") && h > 0 &&
                                 kResidentRanks[r] == 1);
        std::vector<int> active, sides(count, n), base(count, 0);
        for (int c = 0; c < count; c++) active.push_back(c);
        printf("%d", ResidentMaxSide(f64));
        for (const ResidentClass& k : PlanStrips(active, sides, base, f64, 148,
                                               held))
            for (const ResidentItem& i : k.items)
                if (i.cav == 0)
                    printf(" %d %d %d %d %d %d %d %d", k.halves, k.ranks,
                           k.warps, k.max_steps, i.row0, i.rows, i.vrow0,
                           i.vrows);
        printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "ask.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", build.CSRC, "-o",
                    d / "ask", d / "ask.cpp"], check=True)

    def run(lines):
        out = subprocess.run([d / "ask"], input="\n".join(lines), text=True,
                             capture_output=True, check=True).stdout
        return [list(map(int, line.split())) for line in out.splitlines()]
    return run


@pytest.mark.parametrize("f64", [0, 1])
def test_the_ctas_of_a_form_share_an_sm(ask, f64):
    for halves, (slots, smem) in enumerate(
            ask([f"form {f64} {h} 0" for h in range(3)])):
        assert smem == slots * 9 * (8 if f64 else 4)
        # 228 KB an SM, 1 KB of each CTA's is the driver's, 227 KB a CTA
        assert (smem + 1024) * 2**halves <= 228 * 1024
        assert smem <= 227 * 1024


@pytest.mark.parametrize("f64", [0, 1])
@pytest.mark.parametrize("what, most_ranks, least_halves", [
    ("plan", 9, 0), ("portable", 8, 0), ("single", 1, 1)])
@pytest.mark.parametrize("count", [1, 30, 3000])
def test_strips_cover_every_side(ask, f64, count, what, most_ranks,
                                 least_halves):
    """On a whole GPU, and on one that cannot hold clusters beyond the portable
    size, or none and no CTA of a whole SM's slots."""
    largest = 400 if f64 else 800
    slots = [s for s, _ in ask([f"form {f64} {h} 0" for h in range(3)])]
    sides = list(range(3, largest + 1, 1 if what == "plan" else 7))
    got = ask([f"{what} {f64} {n} {count}" for n in sides])
    for n, (most, *flat) in zip(sides, got):
        assert most == largest
        strips = sorted((flat[i:i + 8] for i in range(0, len(flat), 8)),
                        key=lambda s: s[4])
        if not strips:      # too few rows of slots for any overlap
            assert what == "single" and slots[1] // n < 2 * 3 + 1
            continue
        row = 0
        for halves, ranks, warps, steps, row0, rows, vrow0, vrows in strips:
            assert -(-rows // ranks) * n <= slots[halves]
            assert 2 <= warps <= 24 >> halves
            assert ranks <= most_ranks and halves >= least_halves
            assert row0 + vrow0 == row and vrows > 0
            row += vrows
            # a cut edge's wrong values travel a row a step after the first
            if row0 > 0:
                assert vrow0 >= steps - 1
            if row0 + rows < n:
                assert rows - vrow0 - vrows >= steps - 1
            assert 0 <= row0 and row0 + rows <= n
        assert row == n, n


def test_a_side_beyond_the_slots_has_no_strips(ask):
    assert ask(["plan 0 801 2", "plan 1 401 2"]) == [[800], [400]]


def test_a_device_that_holds_none_has_no_strips(ask):
    assert ask(["none 0 64 2", "none 1 64 2"]) == [[800], [400]]
