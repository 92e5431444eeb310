"""What the 2D and Born tile kernels read before they wait for the launch before them (CPU).

The kernels are programmatic dependents: until griddepcontrol.wait a thread may read only
what was written two launches ago or earlier, which is a thread's own cells, the model and the
profiles.  The step index is written by the launch just before the first step of a pass, the
history and the strain adjoint by the kernel just before; such reads, and what depends on the
index, belong behind `tile2_go(false)`.  Read from the sources, since a read that is too early
gives a wrong value only when the launches happen to overlap that way."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "2d_and_3d_elastic_reverse_time_migration_b200", "csrc")
LATE = r"\b(step_index|it_ptr|wavelet|wsrc|traces|shot_traces|ha0[xz]|hv0[xz]|ex_v|ex_tp|img)\b"


def _early_parts():
    parts = []
    for name in ("step_kernels_2d.cuh", "born.cu"):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\((?:[^{])*\{", text):
            end = text.find("__global__", m.end())
            body = text[m.end():end if end > 0 else None]
            if "tile2_begin(" not in body:
                continue
            assert body.count("tile2_go(false)") == 1, m.group(1)
            parts.append((m.group(1), body[:body.index("tile2_go(false)")]))
    return parts


def test_every_tile_kernel_is_looked_at():
    assert sorted(n for n, _ in _early_parts()) == ["k_adj_str", "k_adj_vm", "k_born_stress", "k_born_velocity",
                                                    "k_stress2d", "k_velocity2d"]


@pytest.mark.parametrize("name,early", _early_parts(), ids=lambda v: v if v.startswith("k_") and len(v) < 40 else "")
def test_nothing_of_the_previous_launch_is_read_ahead_of_the_wait(name, early):
    found = sorted(set(re.findall(LATE, early)))
    # Born velocity only asks whether there are traces (a kernel argument)
    if name == "k_born_velocity":
        early = early.replace("BORN && a.traces ?", "")
        found = sorted(set(re.findall(LATE, early)))
    assert not found, f"{name} reads {found} before it waits"
