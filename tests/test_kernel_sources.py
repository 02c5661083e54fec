"""Rules of the device code that a wrong result shows only by chance, checked on the source text."""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "spin_colour_kernel_b200" / "csrc"


def kernel_body(file: str, name: str) -> str:
    """The braces of __global__ function `name`."""
    text = (CSRC / file).read_text()
    at = re.search(r"__global__[^;{]*\b" + name + r"\([^{;]*\{", text)
    assert at, name
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at.start():i]


def test_in_place_word_loads_stay_off_the_read_only_path():
    """ising_march_kernel loads 4-byte words that hold spins of the class it is updating in the same launch:
    ld.global.nc (__ldg) is for memory that no thread of the launch writes."""
    body = kernel_body("fast_sweep.cu", "ising_march_kernel")
    assert "dst[" in body and "src" in body
    assert not re.search(r"__ldg|\.nc\b|__restrict__", body)


def test_task_launches_refuse_ising_plans():
    """No class task kernel takes Ising spins: a task launch of an Ising plan is an error, not a launch of nothing."""
    text = (CSRC / "fast_sweep.cu").read_text()
    body = text[text.index("static int launch_tasks("):]
    body = body[:body.index("\n}\n")]
    assert re.search(r"if \(plan->geom\.n == 1\) return cuda_status\(cudaErrorInvalidValue", body)
    one = text[text.index("static void launch_one("):]
    assert "N > 1" not in one[:one.index("\n}\n")]
