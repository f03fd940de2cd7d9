"""The benchmark's count of a solve's kernels against the launch lists."""
import os
import re
import sys
from types import SimpleNamespace

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


@pytest.mark.parametrize("name,entry", [("launches_config1_fp64.md", "pcg_grid"),
                                        ("launches_config1_mixed.md", "pcg_cluster")])
def test_count_equals_the_list(name, entry):
    import bench

    text = open(os.path.join(ROOT, "profiles", name)).read()
    rows = re.findall(r"^\| `([^`]+)` \| (\d+) \|", text, re.M)
    pcg = sum(int(n) for k, n in rows if "k_pcg" in k)
    s = SimpleNamespace(num_iterations=50, num_linear_solver_iterations=100 * pcg)
    assert bench.launches_per_solve(s, {"schur_form": 50, entry: pcg}) == sum(int(n) for _, n in rows)
