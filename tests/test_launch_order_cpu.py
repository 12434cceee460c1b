"""Kernels that become resident while the launch ahead of them still runs (``launch_overlapped`` in ``csrc/kernels/common.h``), read as text: every
thread waits for that launch before it can leave, so that the end of such a kernel implies the end of all before it."""
import re
from pathlib import Path

KERNELS = Path(__file__).resolve().parent.parent / "neuralfn_b200" / "csrc" / "kernels"


def _bodies():
    """(name, body) of every kernel in the sources; comments taken out."""
    for path in sorted(KERNELS.iterdir()):
        if path.suffix not in (".cu", ".cuh"):
            continue
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\([^{}]*?\)\s*)*(\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, end = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield m.group(1), text[start:end]


def test_no_overlapped_kernel_leaves_before_it_has_waited():
    seen = set()
    for name, body in _bodies():
        if "grid_wait()" in body:
            seen.add(name)
            before = body[:body.index("grid_wait()")]
            assert not re.search(r"\breturn\s*;", before), f"{name} can return ahead of grid_wait()"
    assert {"attn_fwd2_kernel", "gemm_bf16_kernel", "gemv_bf16_kernel", "decode_attention_mma_kernel", "norm_fwd_kernel"} <= seen


def test_every_overlapped_launch_is_of_a_kernel_that_waits():
    waits = {name for name, body in _bodies() if "grid_wait()" in body}
    launched = set()
    for path in KERNELS.glob("*.cu"):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        if "launch_overlapped(" in text:
            launched |= set(re.findall(r"launch_overlapped\(\s*(\w+_kernel)\b", text)) | set(re.findall(r"\brun\((\w+_kernel)\b", text))
    assert len(launched) > 10 and launched <= waits, launched - waits
