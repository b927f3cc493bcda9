"""Kernels launched as programmatic dependents run while the kernel before them still writes: what they read
of its output must not go through the read-only path, whose loads the compiler may move above the wait
(the source, since with one compiler the results show nothing)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lum_gb300", "csrc")
WORLD = {"grid"}   # written by plain launches and copies only, which end before any dependent starts


def _source():
    text = "\n".join(open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))
    return re.sub(r"//[^\n]*", "", text)


def _body(text, at):
    start = text.index("{", at)
    depth, i = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def _kernels(text):
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(([^)]*)\)\s*\{", text):
        yield m.group(1), m.group(2), _body(text, m.end() - 1)


def test_parameters_of_waiting_kernels():
    waiting = {name: params for name, params, body in _kernels(_source()) if "grid_dependency_wait()" in body}
    assert {"list_flags_kernel", "list_write_kernel", "shift_kernel", "gather_kernel", "pack_rgb_kernel"} <= set(waiting)
    for name, params in waiting.items():
        read_only = set(re.findall(r"const\s[^,]*\*\s*__restrict__\s+(\w+)", params))
        assert read_only <= WORLD, (name, read_only)


def test_volumes_and_lists_by_ordinary_loads():
    text = _source()
    loads = [_body(text, m.end()) for m in re.finditer(r"float3 load\(const T\* p, int i\)", text)]
    assert len(loads) == 4 and not any("__ldg" in b for b in loads)
    for field in ("req", "prev", "next", "dev_count", "copy_src", "count_src", "rays", "stats"):
        assert not re.search(r"__ldg\([^;]*\b%s\b" % field, text), field
    m = re.search(r"float3 gather_point\(([^)]*)\)", text)
    assert "__restrict__" not in m.group(1)
