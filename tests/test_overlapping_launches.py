"""What kernels that are placed while the launch before them still writes (dsmd_launch.cuh) may not do: read by the read-only path."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepscalemd_b200", "csrc")
SOURCES = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read()) for p in sorted(glob.glob(os.path.join(CSRC, "dsmd_*.cu*")))}


def kernels():
    for name, text in SOURCES.items():
        for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?(\w+)\(([^;{}]*)\)\s*\{", text):
            yield name, m.group(1), m.group(2), text[m.end():text.index("\n}\n", m.end())]


def test_no_read_only_loads():
    found = list(kernels())
    waiting = {kernel: parameters for _, kernel, parameters, body in found if "after_previous" in body}
    assert {"k_pair", "k_step", "k_pack", "k_constrained", "k_bonded_terms", "k_build_rows", "k_reorder", "k_edge_search", "k_cell_starts"} <= set(waiting)
    assert not {k for k, parameters in waiting.items() if re.search(r"const [\w ]+\*\s*__restrict__", parameters)}
    assert not [name for name, text in SOURCES.items() if "__ldg(" in text]


@pytest.mark.parametrize("name", sorted(SOURCES))
def test_whoever_is_launched_to_overlap_waits(name):
    waiting = {kernel for _, kernel, _, body in kernels() if "after_previous" in body}
    launched = set(re.findall(r"launch_next\((k_\w+)", SOURCES[name]))
    assert launched <= waiting
