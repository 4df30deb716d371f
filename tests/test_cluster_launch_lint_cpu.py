"""Kernels launched by launch_cluster (csrc/sevc_topology.cu) carry the
programmatic-serialisation attribute like those of launch_dep: their first
statement must be griddep_wait(), or they race with the kernel before them."""
import re

from test_launch_dep_lint_cpu import _sources


def test_kernels_launched_as_a_cluster_wait_first():
    src = _sources()
    launched = set()
    for text in src.values():
        launched |= set(re.findall(r"launch_cluster\(\s*(k_\w+)", text))
    assert {"k_tail", "k_deferred"} <= launched
    for name in sorted(launched):
        bodies = [text[mo.end():] for text in src.values()
                  for mo in re.finditer(r"__global__ void (?:__launch_bounds__\([^)]*\)\s*)?" + name + r"\([^)]*\)\s*\{", text)]
        assert len(bodies) == 1, name
        assert bodies[0].lstrip().split(";", 1)[0].strip() == "griddep_wait()", name
