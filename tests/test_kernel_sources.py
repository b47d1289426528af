"""What the kernels' sources promise about memory order between blocks, read from the text: no run could show it reliably."""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "bare_cuda_4gib_b200" / "csrc"


@pytest.mark.parametrize("name", ["attention_f32.cu", "matmul_f32.cu"])
def test_a_block_whose_shared_memory_others_read_waits_for_the_reads(name):
    """A kernel that loads from other blocks' shared memory ends each such stretch at the cluster's barrier, behind which the owner
    writes again or leaves.  A relaxed arrival orders nothing that came before it, so every arrival releases and every
    wait acquires."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    assert "ld.shared::cluster" in text
    arrivals = re.findall(r"barrier\.cluster\.arrive([.a-z]*)", text)
    waits = re.findall(r"barrier\.cluster\.wait([.a-z]*)", text)
    assert arrivals and all(".release" in a for a in arrivals), arrivals
    assert waits and all(".acquire" in w for w in waits), waits
