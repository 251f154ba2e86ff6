"""Places in shared memory that the other blocks of a cluster read."""

import re

from models_b200.kernels import build


def test_a_block_writes_what_the_others_read_once():
    """A second number in the same place could meet a block that still reads the first: between the two there is a barrier before the read, and
    none behind it."""
    text = re.sub(r"//[^\n]*", "", (build.CSRC / "sampling.cu").read_text())
    read = sorted(set(re.findall(r"map_shared_rank\(&(slot_\w+)", text)))
    assert read == ["slot_mass", "slot_sum", "slot_ties"]
    for name in read:
        assert len(re.findall(rf"\b{name}\s*=[^=]", text)) == 1, name
