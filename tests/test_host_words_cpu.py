"""The words by which kernels report to the host, compiled and run on the CPU."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "dist-gpu-sampling_b200", "csrc")

# what the host could see, in the order in which the device makes it visible
ORDER = r"""
#include <cstdint>
#include <cstdio>
#define __device__
#define __forceinline__ inline
static int64_t words[2] = {-1, -1};
static int32_t status = 0;
static void show(const char* at) { std::printf("%s %d %lld %lld\n", at, status, (long long)words[0], (long long)words[1]); }
static void __threadfence_system() { show("fence"); }
namespace dgs {
static void raise_status(int32_t* s, int32_t code) { *s = code; }
}
#include "kernels/host_report.cuh"
int main() {
  const int64_t a = 5, b = 6;
  const int64_t* src[2] = {&a, &b};
  dgs::report_sizes(words, src, 2, CODE, &status);
  show("end");
}
"""


TEXTS = r"""
#include <cstdio>
#include "binding/host_words.h"
int main() {
  for (int code : {DGS_ERR_INVALID, DGS_ERR_RANGE, DGS_ERR_TABLE_FULL, DGS_ERR_ID_SPACE}) std::puts(dgs::status_text(code));
}
"""


def compiled(tmp_path, text, *flags):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(text)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe), *flags], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()


@pytest.mark.parametrize("code", [0, 9])
def test_an_error_that_decides_is_at_the_host_before_the_sizes_are(tmp_path, code):
    seen = compiled(tmp_path, ORDER.replace("CODE", str(code)))
    assert seen[-1] == f"end {code} 5 6"
    assert seen[0] == ("fence 9 -1 -1" if code else "fence 0 5 6")


def test_every_status_that_kernels_raise_has_words(tmp_path):
    from torch.utils import cpp_extension
    flags = [f for p in cpp_extension.include_paths() + ["/usr/local/cuda/include"] for f in ("-isystem", p)]
    assert compiled(tmp_path, TEXTS, *flags) == ["an error", "an out-of-range id", "a full hash table", "an id beyond the id space"]
