"""Kernels launched behind the one before them (launch_behind in csrc/common.cuh) may touch what that one reads or writes only past
grid_wait(): each of them calls it before its first access to global memory."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "pratchya_b200" / "csrc"


def test_every_kernel_launched_behind_another_waits_for_it():
    launched, seen = set(), 0
    sources = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu"))}
    for text in sources.values():
        launched |= set(re.findall(r"launch_behind\(\(?(\w+)", text)) - {"kernel", "KERNEL"}
        launched |= set(re.findall(r"PB_ROW128_LAUNCH\(\((\w+)", text)) | set(re.findall(r"go\((\w+)<", text)) | set(re.findall(r"cudaLaunchKernelEx\(&config, (\w+)", text)) - {"kernel"}
    launched.discard("void")
    assert len(launched) >= 30, launched
    for name, text in sources.items():
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\((?:[^{};]|\{[^}]*\})*?\)\s*\{\n", text):
            if m.group(1) not in launched:
                continue
            seen += 1
            end = text.index("\n}\n", m.end())
            body = text[m.end():end]
            at = body.find("grid_wait();")
            assert at >= 0, f"{name}: {m.group(1)} is launched behind another kernel and does not wait for it"
            before = body[:at]
            assert not re.search(r"__ldg|\bp\.\w+\[|tma_load|load_box|cp_async16|return;", before), f"{name}: {m.group(1)} reads global memory, or leaves, before it waits"
    assert seen == len(launched), (seen, launched)
