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


# what may be called before the wait: addresses in shared memory, barriers, fences
BEFORE = {"smem_u32", "dot_smem_u32", "bar_init", "mbar_init", "full", "empty", "acc_full", "acc_empty", "bar_full", "bar_empty", "bar_acc_full", "bar_acc_empty", "tc_before", "tc_after",
          "tc_fence_before", "tc_fence_after", "__syncthreads", "cluster_sync_all", "cluster_ctarank", "__align__", "volatile", "for", "if", "sizeof"}


def _touches(params, before):
    """What the text in front of a kernel's wait, whose parameters are `params`, has that may reach global memory."""
    found = []
    before = re.sub(r"//[^\n]*", "", before)
    for text, operands in re.findall(r'asm volatile\("((?:[^"\\]|\\.)*)"([^;]*);', before):
        if not re.match(r"fence\.mbarrier_init|tcgen05\.(alloc|relinquish_alloc_permit)\.", text) or "[" in operands.replace("[%0]", "").replace("[]", ""):
            found.append(text)
    before = re.sub(r'asm volatile\([^;]*;', "", before)
    names = {re.findall(r"\w+", part)[-1] for part in params.split(",")}
    found += [m for m in re.findall(r"\b\w+(?:\.\w+)?", before) if m.split(".")[0] in names and m != "p.splitk"]
    found += [m for m in re.findall(r"\b(\w+)\s*\(", before) if m not in BEFORE and not m.startswith("k") and m not in ("uintptr_t",)]
    found += [m for m in re.findall(r"\b(\w+)\[", before) if m not in ("bars", "dot_smem", "split_smem", "smem_raw")]
    found += [m for m in re.findall(r"(?:^|[=(,;{])\s*\*\s*(\(?\w+)", before, re.M) if m not in ("tmem_slot", "abort_flag", "(volatile")]
    return found


def test_nothing_outside_the_cta_is_touched_before_the_wait():
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(((?:[^{};]|\{[^}]*\})*?)\)\s*\{\n", text):
            body = text[m.end():text.index("\n}\n", m.end())]
            if "grid_wait();" in body:
                seen += 1
                assert not _touches(m.group(2), body[:body.index("grid_wait();")]), (path.name, m.group(1))
    assert seen >= 40
    for line in ("float a = in[0];", "float a = *in;", "const float a = __ldg(other);", "load(s);", "x = p.scale;", "float a = *(in + 3);", "const auto q = in;", "prefetch(&map);",
                 'asm volatile("ld.global.f32 %0, [%1];" : "=f"(a) : "l"(q));', "if (q[3]) return;"):
        assert _touches("const float* __restrict__ in, const __grid_constant__ Params p, CUtensorMap map", line + "\n"), line


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
