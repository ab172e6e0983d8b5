"""Kernels that start while the one before them is still running read what it writes: rules their sources keep (no GPU)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "apt_serve_b200" / "csrc"


def kernels():
    """name -> parameter list and body of every __global__ function."""
    found = {}
    for f in sorted(CSRC.glob("*.cu")):
        text = f.read_text()
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__[^\n]*\n)?\s*(\w+)\(", text):
            end = text.index(") {", m.end())
            depth, i = 1, end + 3
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            found.setdefault(f"{f.name}:{m.group(1)}", (text[m.end():end], text[end:i]))
    return found


def chained():
    names = set()
    for f in sorted(CSRC.glob("*.cu")):
        text = f.read_text()
        for m in re.finditer(r"launch_chained\(([^;]*);", text):
            names |= {f"{f.name}:{k}" for k in re.findall(r"\b(\w+_kernel)\b", re.sub(r'"[^"]*"', "", m.group(1)))}
        for m in re.finditer(r"auto k(?:ernel)? = &?(\w+_kernel)<", text):   # launched through a local name
            if re.search(r"launch_chained\([^;]*\bk(?:ernel)?,", text[m.end():m.end() + 1200]):
                names.add(f"{f.name}:{m.group(1)}")
    return names


def test_all_chained_kernels_are_found():
    names, all_kernels = chained(), kernels()
    assert names <= set(all_kernels)
    assert {"paged_attention.cu:combine_kernel", "paged_attention.cu:plan_kernel", "paged_attention.cu:kv_attention_tma_kernel",
            "hidden_attention.cu:scores_kernel", "hidden_attention.cu:sum_kernel", "cache_ops.cu:bulk_copy_kernel",
            "hidden_fp32.cu:attend32_kernel", "hidden_attention.cu:step_plan_kernel"} <= names


def test_their_parameters_are_not_restrict():
    """A read-only no-alias parameter lets the compiler load through it before the wait for the kernel that writes it."""
    all_kernels = kernels()
    for name in chained():
        params, body = all_kernels[name]
        assert "__restrict__" not in params, name
        assert "chain_wait()" in body, name
