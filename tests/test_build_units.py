"""Every kernel is compiled by one unit of the library.  A template kernel that
two units instantiate is in the library twice, compiled with the floating-point
flags of either, and which of the two a process runs differs from process to
process."""
import os
import subprocess
from collections import defaultdict

from mplb_b200 import build


def test_each_kernel_is_defined_once():
    build.build()
    objects = [obj for obj, _ in build.compile_commands()]
    if not all(os.path.exists(o) for o in objects):
        build.build(force=True)
    units = defaultdict(set)
    for obj in objects:
        names = subprocess.run(["nm", "-C", "--defined-only", obj],
                               capture_output=True, text=True,
                               check=True).stdout
        for line in names.splitlines():
            name = line.split(None, 2)[-1]
            if "Kernel" in name.split("(")[0]:
                units[name].add(os.path.basename(obj))
    assert any("BatchInitKernel<float>" in n for n in units)
    twice = {n: sorted(u) for n, u in units.items() if len(u) > 1}
    assert not twice, twice
