"""Kernels that may start before the one in front of them has finished (launch_dependent): each waits before anything else, and neither it
nor a device function that it calls reads global memory through the read-only path, whose loads may be moved above the wait."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "boundflow_b200", "csrc")
READ_ONLY = re.compile(r"__ldg\b|\bld\.global\.nc\b|\bconst\b[^,;(){}]*__restrict__")


def _functions():
    """({kernel: (parameters, body)}, {device function: text}, all sources without comments)"""
    kernels, device, sources = {}, {}, ""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as fh:
                text = re.sub(r"//[^\n]*|/\*.*?\*/", "", fh.read(), flags=re.S)
            sources += text
            for m in re.finditer(r"(__global__|__device__)\b[^;{}()]*?(?:__launch_bounds__\([^{;]*?\)\s*)?(\w+)\s*\(([^;{}]*)\)\s*\{", text):
                depth, end = 1, m.end()
                while depth:
                    depth += {"{": 1, "}": -1}.get(text[end], 0)
                    end += 1
                if m.group(1) == "__global__":
                    assert m.group(2) not in kernels, m.group(2)
                    kernels[m.group(2)] = (m.group(3), text[m.end():end])
                else:
                    device[m.group(2)] = device.get(m.group(2), "") + m.group(3) + text[m.end():end]
    return kernels, device, sources


def test_dependent_kernels_wait_first_and_read_with_plain_loads():
    kernels, device, sources = _functions()
    launched = set(re.findall(r"launch_dependent\(\s*(?:bf::)?(\w+_kernel)", sources))
    # the clusters of conv_tile_kernel are launched with the attribute among others
    launched |= set(re.findall(r"cudaLaunchKernelEx\(&cfg, (\w+_kernel)", sources)) & {"conv_tile_kernel"}
    assert len(launched) >= 13 and launched <= set(kernels), launched - set(kernels)
    waiting = {k for k, (_, body) in kernels.items() if "grid_wait()" in body}
    assert waiting == launched, waiting ^ launched
    for k in sorted(launched):
        params, body = kernels[k]
        assert re.match(r"\s*grid_wait\(\);", body), f"{k}: the wait is not the first statement"
        assert "__restrict__" not in params, f"{k}: a __restrict__ parameter's loads may pass the wait"
        seen, todo = set(), [body]
        while todo:
            text = todo.pop()
            assert not READ_ONLY.search(text), f"{k}: {READ_ONLY.search(text).group(0)}"
            for f in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", text)) & set(device) - seen:
                seen.add(f)
                todo.append(device[f])


def test_kernels_that_wait_after_their_setup_touch_no_global_memory_before():
    """launch_after_setup: in front of grid_wait_after_setup() a kernel sets up barriers, tensor memory and indices only."""
    kernels, device, sources = _functions()
    launched = set(re.findall(r"launch_after_setup\(\s*(?:\w+::)*(\w+_kernel)", sources))
    waiting = {k for k, (_, body) in kernels.items() if "grid_wait_after_setup()" in body}
    assert launched and launched == waiting, launched ^ waiting
    for k in sorted(launched):
        params, body = kernels[k]
        front, behind = body.split("grid_wait_after_setup();")
        assert "__restrict__" not in params and "grid_release()" not in front and "grid_release()" in behind
        # no loads, stores, copies or atomics; the only subscripts are those of barriers in shared memory
        assert not re.search(r"\bload\w*\(|\bld_\w*\(|\bbulk_copy|\*\s*reinterpret_cast|\.global\b|atomic|\bg\.\w+\[", front), k
        assert set(re.findall(r"(\w+(?:\.\w+)?)\[[^\]]*\]\s*[;,)=+]", front)) <= {"ctl.full", "ctl.summed", "ctl.drained", "row_part", "con_part", "st_smem"}, k
        seen, todo = set(), [body]
        while todo:
            text = todo.pop()
            assert not READ_ONLY.search(text), f"{k}: {READ_ONLY.search(text).group(0)}"
            for f in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", text)) & set(device) - seen:
                seen.add(f)
                todo.append(device[f])
