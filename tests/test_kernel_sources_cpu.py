"""What the kernels' sources promise, read from them: the cluster kernel leaves
out its transforms where a CTA has no rows."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "channel_rl_gb300", "csrc")


def _body(text, start):
    depth, at = 1, start
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return text[start:at]


def _sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _kernels(src):
    for f, text in src.items():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^;{]*?\)\s*\{", text):
            yield f, m.group(1), _body(text, m.end())


def test_cluster_kernel_skips_transforms_without_rows():
    body = next(b for _, n, b in _kernels(_sources()) if n == "k_zsolve")
    calls = [m.start() for m in re.finditer(r"\bfx_fft<", body)]
    assert len(calls) == 2
    for at in calls:
        assert re.search(r"if \(nr > 0\)\s*$", body[:at]), "a CTA without rows reaches a division by their number"
