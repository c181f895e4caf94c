"""Kernels that may begin beside the end of the ones ahead of them: what the source has to keep to."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sten_b200", "csrc")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def _kernels(text):
    """(name, signature and body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\([^;{]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.start():i]


WAIT = re.compile(r"dependents_wait\(\)|griddepcontrol\.wait")


def test_early_kernels_wait_and_read_with_ordinary_loads():
    """A read-only load asserts that nothing writes there during the kernel's life, which began beside the kernels ahead."""
    seen = 0
    for name, text in _sources():
        early = set(re.findall(r"launch_early\((\w+)", text))
        for kernel, code in _kernels(text):
            if kernel in early:
                assert WAIT.search(code), f"{name}: {kernel} is launched early and never waits"
            if not WAIT.search(code):
                continue
            seen += 1
            assert "__ldg" not in code and "__restrict__" not in code, f"{name}: {kernel}"
        if name in ("nmg_expand.cuh", "nmg_tc_common.cuh"):  # device functions that they call
            assert "__ldg" not in text and "__restrict__" not in text, name
    assert seen >= 9


def test_bounded_waits_begin_behind_the_kernels_ahead():
    """A wait that gives up after a time must not count the time that earlier kernels of the stream take."""
    seen = 0
    for name, text in _sources():
        for kernel, code in _kernels(text):
            if kernel not in ("gemm_tc_kernel", "gemm_sp_kernel", "spmm_tc_kernel"):
                continue
            parts = re.split(r"// -{20,}", code)  # what comes before the roles of the warps, then a part for each
            ahead = parts[0].count("dependents_wait();") == 3  # spmm_tc_kernel: all three branches of its set-up
            for part in parts[1:]:
                first = re.search(r"[^_]wait\(&|mbar_wait\w*\(", part)
                if first:
                    seen += 1
                    assert ahead or "dependents_wait();" in part[:first.start()], f"{name}: {kernel}: {part.strip().splitlines()[0]}"
    assert seen >= 9
