"""What the compiler has to be told about inline assembly, checked in the sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mask_b200", "csrc")


def test_assembly_that_touches_shared_memory_is_ordered_with_the_rest():
    """Loads, stores and copies of shared memory name "memory": a barrier between two lanes' accesses is no assembly, and orders
    them only if the compiler may not move them across it."""
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        for text in re.findall(r"\basm\b[^;]*?\((?:\s*\"(?:[^\"\\]|\\.)*\")+[^;]*;", open(path).read()):
            if re.search(r"\b(?:ld|st|red|atom)\.shared|\bcp\.async", text):
                found += 1
                assert text.rstrip("; \n)").endswith('"memory"'), (os.path.basename(path), text)
    assert found >= 10
