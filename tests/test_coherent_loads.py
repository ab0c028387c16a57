"""The step's kernels are links of a chain of dependent launches: a grid is
resident while its predecessor still writes.  A non-coherent load (__ldg,
ld.global.nc) may only read what nothing writes during the grid's lifetime, so
none of them reads a vector that a kernel of the step writes (no GPU: the
sources are searched)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "soft-body-simulation-cuda_gb300" / "csrc"
# iterate, right-hand side, solve vectors, state: members of the kernels' arguments
WRITTEN = "sn|prev|out|b|bsave|r|y|y_next|x|x0|dx|z|v|xt|done|st"
NC = re.compile(r"(?:__ldg|ld_hint)\s*\(\s*(?:reinterpret_cast<[^>]*>\()?\s*&?\s*\w+(?:\.|->)(?:" + WRITTEN + r")\b")


@pytest.mark.parametrize("name", ["kernels.cu", "solve.cu", "scene.cuh", "scene.cu"])
def test_no_non_coherent_load_of_what_a_step_writes(name):
    found = [f"{name}:{i}: {line.strip()}" for i, line in enumerate((CSRC / name).read_text().splitlines(), 1)
             if NC.search(line)]
    assert not found, "\n".join(found)


def test_the_search_finds_one():
    assert NC.search("const float4 p = __ldg(&a.sn[v]);") and NC.search("__ldg(a.x + i)")
    assert not NC.search("__ldg(&a.tile_verts[k])") and not NC.search("__ldg(&q.base[i])")
