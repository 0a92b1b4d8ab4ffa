"""A refused request for scratch leaves an error message (csrc/internal.h, compiled for the host against a CUDA
runtime that has no memory left), and the windowed product takes every such refusal as "not done"."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "gb_kun_b200" / "csrc"

HARNESS = r"""
#include "internal.h"
#include <cstdarg>
#include <cstdio>
#include <cstring>
static char text[256] = "an older error";
static int freed = 0, given = 1;
extern "C" cudaError_t cudaMallocAsync(void** p, size_t, cudaStream_t) {
    static char block;
    if (given-- > 0) return *p = &block, cudaSuccess;
    return cudaErrorMemoryAllocation;
}
extern "C" cudaError_t cudaFreeAsync(void*, cudaStream_t) { return ++freed, cudaSuccess; }
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }
namespace gbk {
void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(text, sizeof(text), fmt, ap);
    va_end(ap);
}
}
int main() {
    {
        gbk::StreamScratch dev(nullptr);
        int *a = nullptr, *b = nullptr;
        if (dev.get(&a, 4) != GBK_SUCCESS || !a || strcmp(text, "an older error")) return 1;
        if (dev.get(&b, 123456) != GBK_OUT_OF_MEMORY || b) return 2;
    }
    if (!strstr(text, "out of device memory") || !strstr(text, "123456")) return 3;
    return freed == 1 ? 0 : 4;
}
"""


def test_refused_scratch_leaves_a_message(tmp_path):
    cxx, cuda = shutil.which("g++"), Path("/usr/local/cuda/include")
    if not cxx or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    (tmp_path / "s.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), "-I", str(ROOT / "include"), "-I", str(cuda),
                    str(tmp_path / "s.cpp"), "-o", str(tmp_path / "s")], check=True)
    assert subprocess.run([str(tmp_path / "s")]).returncode == 0


def test_windows_fall_back_before_the_first_block():
    src = (CSRC / "spgemm_window.cu").read_text()
    body = src[src.index("int window_t("):src.index("k_win_numeric<SR, T><<<")]
    returns = re.findall(r"dev\.get\([^;{]*?\)\)\s*return (GBK_\w+);", body)
    assert len(returns) >= 6 and set(returns) == {"GBK_SUCCESS"}
