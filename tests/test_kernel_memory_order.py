"""What the kernels' sources promise about memory order, where no run can show it (a weaker form gave the same bits in every test)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blazr_b200", "csrc")


def sources():
    files = sorted(f for ext in ("cu", "cuh", "h") for f in glob.glob(os.path.join(CSRC, "**", "*." + ext), recursive=True))
    assert len(files) > 20
    return {os.path.relpath(f, CSRC): open(f).read() for f in files}


def test_arrivals_at_another_cta_release_at_cluster_scope():
    """an arrival without a scope is one of the CTA: it hands nothing over to a thread of another CTA"""
    seen = 0
    for name, text in sources().items():
        for m in re.finditer(r"mbarrier\.arrive[\w.:]*", text):
            if "shared::cluster" in m.group(0):
                seen += 1
                # (or relaxed, at once behind a release fence of that scope for what lies in shared memory)
                fenced = ".relaxed.cluster." in m.group(0) and "fence.release.sync_restrict::shared::cta.cluster;" in text[max(0, m.start() - 200):m.start()]
                assert ".release.cluster." in m.group(0) or fenced, f"{name}: {m.group(0)}"
    assert seen
