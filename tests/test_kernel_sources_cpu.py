"""What the kernels' sources promise, read from them: every kernel that forms a
field index from x, y and z goes through the checks of the bounds-checked build,
and the cluster kernel leaves out its transforms where a CTA has no rows."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "channel_rl_gb300", "csrc")

# kernels without an (x, y, z) index, and what they run over
FLAT = {
    "k_fix": "whole fields, a flat index below their length",
    "k_fftz": "spectrum columns", "k_tri": "spectrum columns", "k_tri_staged": "spectrum columns",
    "k_tri_scan": "spectrum columns", "k_zsolve": "spectrum columns",
    "k_pack": "whole fields, caller's extents", "k_unpack3": "whole fields, caller's extents",
    "k_pack3": "whole fields, caller's extents", "k_pack_unique": "whole fields, rows given by the host",
    "k_minabs_init": "minima", "k_tadvance": "scalars", "k_divmax_final": "plane partials",
    "k_qflow_final": "plane partials", "k_stats_final": "row partials", "k_sqrt_selftest": "test values",
    "k_tc_selftest": "test operands", "k_div_planes": "caller's arrays and extents", "k_div_final": "plane partials",
}
CHECK = re.compile(r"\b(cidx|vidx|chl_clamp)\(")


def _body(text, start):
    depth, at = 1, start
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return text[start:at]


def _functions(text):
    """name -> body of every function that is defined in text."""
    found = {}
    for m in re.finditer(r"\b(?:void|double|Rhs|bool|int4?|unsigned)\s+(\w+)\s*\([^;{]*?\)\s*\{", text):
        found[m.group(1)] = _body(text, m.end())
    for m in re.finditer(r"\bstruct\s+(\w+)\s*(?::[^{;]*)?\{", text):
        found[m.group(1)] = _body(text, m.end())
    return found


def _sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _kernels(src):
    for f, text in src.items():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^;{]*?\)\s*\{", text):
            yield f, m.group(1), _body(text, m.end())


def test_every_kernel_with_a_field_index_is_checked():
    src = _sources()
    funcs = {}
    for text in src.values():
        funcs.update(_functions(text))

    def checked(body, depth=3):
        if CHECK.search(body):
            return True
        called = set(re.findall(r"\w+", body)) & set(funcs)
        return depth > 0 and any(checked(funcs[c], depth - 1) for c in called)

    names = []
    for f, name, body in _kernels(src):
        names.append(name)
        assert checked(body) != (name in FLAT), (f, name)
    assert set(FLAT) <= set(names)


def test_cluster_kernel_skips_transforms_without_rows():
    body = next(b for _, n, b in _kernels(_sources()) if n == "k_zsolve")
    calls = [m.start() for m in re.finditer(r"\bfx_fft<", body)]
    assert len(calls) == 2
    for at in calls:
        assert re.search(r"if \(nr > 0\)\s*$", body[:at]), "a CTA without rows reaches a division by their number"
