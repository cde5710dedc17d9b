"""CPU: kernels that are launched before their predecessor is complete read memory coherently.  Such a kernel's life overlaps
its predecessor's writes, and a load through the non-coherent path (__ldg, or a const __restrict__ pointer that the compiler
may read that way) is only defined for data that nobody writes meanwhile."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "updes_gb300", "csrc")
SOURCES = {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _early_kernels():
    names = set()
    for text in SOURCES.values():
        names |= {m.group(1) for m in re.finditer(r"launch_next\([^,]+, (\w+_kernel)", text)}
    return sorted(names | {"panel_cluster_kernel"})


def _function(text, name):
    """The text of the function `name`: its parameters and its body."""
    start = re.search(r"\b%s\(" % name, text[text.index("void"):]).start() + text.index("void")
    depth, i = 0, text.index("{", start)
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[start:j + 1]
    raise ValueError(name)


def _definition(name):
    for text in SOURCES.values():
        m = re.search(r"__global__[^;{]*?\b%s\(" % name, text)
        if m:
            return text, _function(text[m.start():], name)
    raise ValueError(name)


def test_the_early_kernels_are_found():
    assert {"digits_kernel", "digits64_kernel", "ozaki3_kernel", "ozaki64_kernel", "trsm_df64_kernel", "trsm64_kernel",
            "block_row_df_kernel"} <= set(_early_kernels())


@pytest.mark.parametrize("name", _early_kernels())
def test_early_kernels_load_coherently(name):
    text, code = _definition(name)
    # the kernel and the device functions of its file that it calls
    pending, seen = [code], {name}
    while pending:
        body = pending.pop()
        assert "__ldg(" not in body
        assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", body)
        for callee in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", body)) - seen:
            if re.search(r"__device__[^;{]*?\b%s\(" % callee, text):
                seen.add(callee)
                m = re.search(r"__device__[^;{]*?\b%s\(" % callee, text)
                pending.append(_function("void " + text[m.start():], callee))
    assert "wait_previous" in seen or "wait_previous()" in code
