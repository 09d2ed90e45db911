"""CPU: the order of griddepcontrol.wait and .launch_dependents in every kernel, read from the sources.

A kernel that lets its successor begin before it has itself waited passes on no guarantee about the kernels before it: in
a chain writer -> such a kernel -> W4A16, the W4A16 kernel reads weights, scales and zero-points ahead of its own wait
while nothing has waited for the writer's stores. Waiting first, a successor begins behind all of them."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kernel_set_b200", "csrc")
# These two begin to read their weights under any kernel before them and let their own successor do the same.
EARLY = {"w4a16_umma_kernel", "w4a16_decode_kernel"}
CALL = re.compile(r"\b(grid_dependency_wait|grid_launch_dependents|grid_start)\s*\(\s*\)")


def _body(text, at):
    start = depth = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]
    raise AssertionError("unbalanced braces")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _kernels():
    texts = list(_sources())
    start = next(_body(t, m.end()) for t in texts for m in [re.search(r"void grid_start\(\)", t)] if m)
    expanded = [m[1] for m in CALL.finditer(start)]
    out = {}
    for t in texts:
        for m in re.finditer(r"__global__ void(?: __launch_bounds__\([^\n]*\))?\s*\n?(\w+)\(", t):
            steps = []
            for c in CALL.finditer(_body(t, m.end())):
                steps += expanded if c[1] == "grid_start" else [c[1]]
            out[m[1]] = steps
    return out, "\n".join(texts)


def test_a_kernel_waits_before_it_lets_its_successor_begin():
    kernels, _ = _kernels()
    assert EARLY <= set(kernels) and "quant_group128_kernel" in kernels
    for name, steps in kernels.items():
        if "grid_launch_dependents" in steps and name not in EARLY:
            assert steps.index("grid_dependency_wait") < steps.index("grid_launch_dependents"), name


def test_a_kernel_launched_programmatically_waits():
    kernels, text = _kernels()
    launched = set(re.findall(r"launch_programmatic(?:_cluster)?\(\s*(\w+)", text)) & set(kernels)
    assert len(launched) >= 15
    for name in launched:
        assert "grid_dependency_wait" in kernels[name], name
