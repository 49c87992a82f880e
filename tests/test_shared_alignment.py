"""Dynamic shared memory starts where the static part ends: an array that is
read in 16-byte words has to say so, or its start is only as aligned as its
element type.  A misaligned access would fault, so the declarations are read."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ursa_b200", "csrc")


def test_dynamic_shared_memory_is_declared_aligned():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        for line in re.findall(r"extern __shared__[^;]*;", open(os.path.join(CSRC, name)).read()):
            seen += 1
            assert re.search(r"__align__\((16|128|1024)\)", line), f"{name}: {line}"
    assert seen
