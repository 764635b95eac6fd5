"""A kernel that starts while the one before it still writes (after_previous) reads nothing through
ld.global.nc, which is defined only for data that is read-only for the kernel's whole lifetime: neither
the kernel nor a device function that it calls uses __ldg or an .nc load, and none of the kernel's
parameters is __restrict__ (from const __restrict__ the compiler makes the same load)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "watercube_gb300" / "csrc"


def functions(text):
    """name -> (signature, body) of the functions that a brace at the end of a line opens."""
    found = {}
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"^[^\n;{}#/]*(?:__global__|__device__)[^;{}]*?(\w+)\s*\(([^;{}]*)\)\s*\{", text, re.M):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        found.setdefault(m[1], []).append((m[0], text[m.end():i]))
    return found


@pytest.mark.parametrize("name", ["wc_nn_gemm.cu", "wc_nn_ops.cu"])
def test_overlapping_kernels_load_coherently(name):
    text = "\n".join(line.split("//")[0] for line in (CSRC / name).read_text().splitlines())
    funcs = functions(text)
    kernels = [k for k, v in funcs.items() for _, body in v if "after_previous()" in body and k != "after_previous"]
    assert len(kernels) >= 3, kernels
    todo, seen = list(kernels), set()
    while todo:
        k = todo.pop()
        if k in seen:
            continue
        seen.add(k)
        for signature, body in funcs[k]:
            assert "__ldg" not in body and ".nc." not in body, k
            if k in kernels:
                assert "__restrict__" not in signature, k
            todo += [w for w in set(re.findall(r"\b(\w+)\s*(?:<[^;<>]*>)?\s*\(", body)) if w in funcs]
    assert len(text.split("launch_after(")) - 1 >= len(kernels)
