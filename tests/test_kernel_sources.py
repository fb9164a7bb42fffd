"""What the kernel sources may not contain, read as text (no GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "blazr_b200", "csrc")


def test_no_copy_into_shared_memory_is_sent_to_several_blocks():
    """A copy that one block starts and several blocks of a cluster receive is closed to code that multi-GPU calls run: both libraries serve tensor
    parallelism.  (A tensor-core commit that arrives on barriers of both blocks of a pair is no copy.)"""
    copy, many = "cp.async." + "bulk", "multi" + "cast"
    seen = 0
    for folder, _, files in os.walk(CSRC):
        for name in files:
            if not name.endswith((".cu", ".cuh", ".h")):
                continue
            seen += 1
            with open(os.path.join(folder, name)) as f:
                for statement in re.split(r";\s*\n", f.read()):
                    assert not (copy in statement and many in statement), f"{name}: {statement.strip()[:160]}"
    assert seen > 20
