"""Kernels that start while the kernel before them still runs: nothing that
other kernels write may reach them through the read-only load path, which asks
for data that is constant while a kernel is resident.  Read from the sources,
since the hardware seldom shows the difference."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mld-ainv_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def functions(text, head):
    """(name, parameters, body) of every function that `head` introduces."""
    for m in re.finditer(head + r"[^;{}]*?\b(\w+)\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
        at, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), m.group(2), text[m.end():at]


def test_dependent_kernels_take_plain_pointers():
    seen = set()
    for name in ("kernels.cu", "krylov.cu"):
        for kernel, params, body in functions(source(name), r"__launch_bounds__\("):
            if "dep_wait(" in body or "for_each_info<" in body:
                seen.add(kernel)
                assert "__restrict__" not in params, kernel
                for arg in re.findall(r"(?:__ldg|ldd)\(([^;]*)", body):
                    assert re.match(r"m[12]?\.", arg), (kernel, arg)
    launched = set()
    for name in ("kernels.cu", "krylov.cu"):
        text = source(name)
        launched |= set(re.findall(r"launch_dep\((k_\w+)", text))
        launched |= set(re.findall(r"auto kern = (k_\w+)<", text)) - {"k_persist"}
    assert launched == seen and len(seen) > 10


def test_shared_walks_read_vectors_with_plain_loads():
    found = set()
    for name, params, body in functions(source("sell_device.cuh"), r"__device__ __forceinline__"):
        if name in ("info_dot", "for_each_info", "fold_range"):
            found.add(name)
            assert "__restrict__" not in params, name
            for arg in re.findall(r"(?:__ldg|ldd)\(([^;]*)", body):
                assert re.match(r"m\.", arg), (name, arg)
    assert found == {"info_dot", "for_each_info", "fold_range"}
