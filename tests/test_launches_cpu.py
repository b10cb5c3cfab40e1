"""Kernels launched behind the one before them (launch_behind in csrc/common.cuh) may touch what that one reads or writes only past
grid_wait(): each of them calls it before its first access to global memory."""
import re
import subprocess
from pathlib import Path

from pratchya_b200.csrc import build

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


def test_launch_arguments_convert_as_in_a_call(tmp_path):
    """What a launch with <<<>>> refuses to compile, launch_behind refuses too; what it takes, it takes."""
    src = tmp_path / "launch.cu"
    src.write_text("""
#include "common.cuh"
#include <type_traits>
namespace pb {
__global__ void kernel(const float* in, float* out, int64_t n) { grid_wait(); if (n) *out = *in; }
template <typename... A>
auto takes(int, A... a) -> decltype(launch_behind(kernel, 1u, 1, 0, cudaStream_t(), a...), std::true_type());
template <typename... A>
std::false_type takes(long, A...);
#define TAKES(...) decltype(takes(0, __VA_ARGS__))::value
static_assert(TAKES((const float*)0, (float*)0, (int64_t)0) && TAKES((float*)0, (float*)0, 3) && TAKES(nullptr, (float*)0, 3u), "as declared");
static_assert(!TAKES((const uint8_t*)0, (float*)0, 3) && !TAKES((const float*)0, (uint8_t*)0, 3), "a pointer to another type");
static_assert(!TAKES((const float*)0, (const float*)0, 3), "a dropped const");
static_assert(!TAKES((const float*)0, (uintptr_t)0, 3) && !TAKES((const float*)0, (float*)0, (float*)0), "an integer for a pointer, a pointer for an integer");
static_assert(!TAKES((const float*)0, (float*)0), "too few");
int launch(const float* in, float* out) { return (int)launch_behind(kernel, 1u, 1, 0, nullptr, in, out, 1); }
}
""")
    r = subprocess.run([build._nvcc(), *build.NVCC_FLAGS, f"-I{build.INCLUDE}", f"-I{CSRC}", "-c", str(src), "-o", str(tmp_path / "launch.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
