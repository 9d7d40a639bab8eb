"""Rules of the device code that no run can show to hold (a break of one may
give right results for years), read off the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openmp-blas_gb300", "csrc")


def sources():
    """{file name: its text without comments}"""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            out[f] = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
    return out


def block(text, start):
    """The {...} that opens at or after `start`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise ValueError("unbalanced braces")


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    """barrier.cluster.*.aligned is undefined for a diverged warp: each function
    that issues one brings the warp together first."""
    found = 0
    for name, text in sources().items():
        for m in re.finditer(r"barrier\.cluster\.arrive[a-z.]*\.aligned", text):
            body = text[text.rindex("__device__", 0, m.start()):m.start()]
            assert "__syncwarp();" in body, f"{name}: {body}"
            found += 1
    assert found == 2
