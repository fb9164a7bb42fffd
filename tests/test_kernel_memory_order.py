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


def bodies(text):
    """{function name: [(parameter list, body)]} of a source's functions"""
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(r"\b(\w+)\s*(?:<[\w, ]*>)?\(", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, b = text[m.end():i - 1], re.compile(r"\s*\{").match(text, i)
        if not b or m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__"):
            continue
        depth, j = 1, b.end()
        while depth and j < len(text):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        out.setdefault(m.group(1), []).append((params, text[b.end():j]))
    return out


def test_programmatic_successors_make_no_read_only_loads():
    """a kernel of launch_chained starts while the one ahead writes its operands: nothing it reads is constant for the whole kernel"""
    seen = 0
    for name, text in sources().items():
        if not name.startswith("seq" + os.sep):
            continue
        fns = bodies(text)
        for kernel in [k for k, v in fns.items() for _, b in v if re.match(r"\s*chain_enter\(", b)]:
            seen += 1
            todo, reached = [kernel], set()
            while todo:
                f = todo.pop()
                if f in reached:
                    continue
                reached.add(f)
                for params, body in fns[f]:
                    assert "__ldg" not in body and "ld.global.nc" not in body, f"{name}: {f}, called by {kernel}"
                    todo += [w for w in re.findall(r"\b\w+\b", body) if w in fns]
            for params, body in fns[kernel]:
                const = {p.split()[-1] for p in params.split(",") if "const" in p and "__restrict__" in p}
                entered = set(re.findall(r"\w+", re.search(r"chain_enter\(([^)]*)\)", body).group(1)))
                assert const == entered, f"{name}: {kernel} enters {entered}, its read-only pointers are {const}"
    assert seen >= 16
