"""Kernels that start before their predecessor in the stream has ended (programmatic dependent launch) read what
it writes as ordinary memory.

A `const T* __restrict__` parameter or __ldg() reads through the read-only path, which is only defined for data
that no one writes while the kernel lives, and such a kernel lives while its predecessor still writes: a race
that no output has to show.  So the sources are checked: of the kernels that wait for a predecessor
(grid_dependency_wait), only the inputs named here, which no kernel of their chain writes, are read that way.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pct_reconstruction_b200" / "csrc"
# hull: set before the chain.  WEPL, offsets: of the loaded histories.  paths, path_n, chord (and p, into
# paths): written by the path kernel, on which a chain's first kernel depends in full.
UNWRITTEN = {"hull", "WEPL", "offsets", "paths", "path_n", "chord", "p", "g.s_curve"}


def kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\b", text):
        i = text.index("(", m.end())
        if text[m.end():i].strip().startswith("__launch_bounds__"):
            i = text.index("(", matching(text, i))
        name = re.search(r"(\w+)\s*$", text[:i]).group(1)
        end = matching(text, i)
        if text[end + 1:].lstrip().startswith("{"):
            j = text.index("{", end)
            yield name, text[i + 1:end], text[j:matching(text, j)]


def matching(text, i):
    close = {"(": ")", "{": "}"}[text[i]]
    depth = 0
    for k in range(i, len(text)):
        depth += (text[k] == text[i]) - (text[k] == close)
        if depth == 0:
            return k
    raise AssertionError("unbalanced source")


def overlapped():
    for f in sorted(CSRC.glob("*.cu")):
        for name, params, body in kernels(f.read_text()):
            if "grid_dependency_wait()" in body:
                yield pytest.param(params, body, id=f"{f.stem}-{name}")


def test_the_overlapped_kernels_are_found():
    names = {p.id for p in overlapped()}
    assert {"pct_drop_exact-drop_phase2_kernel", "pct_image-image_update_kernel", "pct_tvs-tvs_gradient_kernel",
            "pct_tvs-tvs_trials_kernel", "pct_tvs-tvs_apply_kernel", "pct_unet-conv3_slab_kernel",
            "pct_unet-avgpool_kernel"} <= names


@pytest.mark.parametrize("params,body", list(overlapped()))
def test_read_only_loads_are_of_unwritten_data(params, body):
    promised = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
    loaded = set(re.findall(r"__ldg\(\s*([\w.]+)", body))
    assert promised | loaded <= UNWRITTEN
