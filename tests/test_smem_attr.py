"""allow_smem (csrc/common.cuh), the attribute that lets a kernel have more than 48 KB of dynamic shared memory: compiled for the CPU against a fake of the
two calls, since it is about several devices in one process and about a call that fails."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pegainfer_b200", "csrc")

FAKE = r"""
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstdio>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
static int device = 0, calls = 0, last_bytes = 0;
static bool fails = false;
static cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
static cudaError_t cudaFuncSetAttribute(const void*, int, int bytes) { ++calls; last_bytes = bytes; return fails ? cudaErrorInvalidValue : cudaSuccess; }
@@
int main() {
  std::atomic<uint64_t> done{0};
  int n = 0;
  auto check = [&](bool ok) { ++n; if (!ok) { printf("check %d failed\n", n); return false; } return true; };
  fails = true;
  if (!check(allow_smem(done, nullptr, 90000) == cudaErrorInvalidValue && calls == 1)) return 1;  // the failure is reported ..
  fails = false;
  if (!check(allow_smem(done, nullptr, 90000) == cudaSuccess && calls == 2 && last_bytes == 90000)) return 1;  // .. and tried again
  if (!check(allow_smem(done, nullptr, 90000) == cudaSuccess && calls == 2)) return 1;
  device = 1;  // another device of the same process has an attribute of its own
  if (!check(allow_smem(done, nullptr, 90000) == cudaSuccess && calls == 3)) return 1;
  device = 0;
  if (!check(allow_smem(done, nullptr, 90000) == cudaSuccess && calls == 3)) return 1;
  printf("ok\n");
  return 0;
}
"""


def test_set_once_per_device_and_failures_reported(tmp_path):
    text = open(os.path.join(CSRC, "common.cuh")).read()
    at = text.index("inline cudaError_t allow_smem(")
    src = tmp_path / "a.cpp"
    src.write_text(FAKE.replace("@@", text[at:text.index("\n}\n", at) + 3]))
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(tmp_path / "a"), str(src)], check=True)
    run = subprocess.run([str(tmp_path / "a")], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout == "ok\n", run.stdout


def test_the_kernels_with_limited_waits_use_it():
    """a flag per process or per thread misses the second device"""
    for name in ("gemm_skinny.cu", "moe_grouped.cu", "latent_attention_tc.cu"):
        text = open(os.path.join(CSRC, name)).read()
        assert "allow_smem(" in text and "cudaFuncSetAttribute" not in text, name
    for name, fn in (("recurrent_mixers.cu", "launch_delta_t"), ("recurrent_mixers.cu", "launch_delta_chunk"),
                     ("qwen35_ops.cu", "pk_b200_gated_delta_rule_prefill_recurrent")):
        text = open(os.path.join(CSRC, name)).read()
        body = re.search(r"\b" + fn + r"\([^;{]*\) \{(.*?)\n\}\n", text, re.S).group(1)
        assert "allow_smem(" in body and "cudaFuncSetAttribute" not in body, fn
