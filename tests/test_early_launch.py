"""Kernels that are brought in while the kernel before them still runs: what their sources have to keep to.

Such a kernel is resident while its predecessor writes the populations, so it may read them only after its wait, and
not through the read-only path, which is for data that nobody writes while the kernel is resident.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "erlbm_gb300", "csrc")
WAIT = "after_previous();"


def sources():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            yield name, re.sub(r"//[^\n]*", "", f.read())


def matching(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced " + pair)


def kernels():
    """(file, name, parameters, body) of every kernel."""
    for name, text in sources():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\()?", text):
            at = m.end()
            if m.group().endswith("("):
                at = matching(text, at - 1, "()") + 1
            k = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            end = matching(text, k.end() - 1, "()")
            brace = re.compile(r"\s*\{").match(text, end + 1)
            if brace:
                yield name, k.group(1), text[k.end():end], text[brace.end():matching(text, brace.end() - 1, "{}")]


EARLY = [k for k in kernels() if WAIT in k[3]]


def test_early_kernels_are_found():
    assert {"k_step", "k_step_quad", "k_step_pair", "k_periodic_d2q9", "k_periodic_d2q9_x2s", "k_periodic_d2q9_x3s",
            "k_periodic_d2q9_x3a", "k_periodic_d3q19", "k_d2q9_hybrid", "k_listed_step"} <= {k[1] for k in EARLY}


def test_early_kernels_wait_before_anything_else():
    for _, name, _, body in EARLY:
        assert body.split(";")[0].strip() + ";" == WAIT, name


def test_early_kernels_read_populations_by_ordinary_loads():
    for _, name, params, body in EARLY:
        for p in params.split(","):
            if re.search(r"\bconst\s+(float2?|double2?|typename\s+P::T)\s*\*", p):
                assert "__restrict__" not in p, (name, p)
        assert "__ldg" not in body, name
    # nor do the functions that read populations for them
    for name, text in sources():
        if name not in {k[0] for k in EARLY}:
            continue
        assert "__ldg" not in text and ".nc." not in text, name
        for m in re.finditer(r"\b(pull4|gather|state_after_x_planes|state_after_planes|step_node)\(([^)]*)\)\s*\{", text):
            assert not re.search(r"const[^,]*\*\s*__restrict__\s*(src|row)\b", m.group(2)), (name, m.group(1))


def test_every_early_launch_is_of_a_kernel_that_waits():
    early = {k[1] for k in EARLY}
    for name, text in sources():
        if name == "launch.cuh":
            continue
        for m in re.finditer(r"\blaunch_step_kernel<(k_\w+)|\blaunch_after\([^,]*,\s*(k_\w+)|\bKERN\s*=\s*(k_\w+)", text):
            assert next(g for g in m.groups() if g) in early, (name, m.group())
