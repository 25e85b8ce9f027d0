"""Nothing that one device answers is kept for the process: contexts on several
devices may be alive at once (include/xg.h), and a kernel's attributes and a
device's limits are the device's own.  allow_smem's own text runs against a
runtime that notes what it was asked for."""

import os
import re

import host_kernel as hk

CODE = r"""
#include <atomic>
struct xg_ctx { int device; };
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize };
static int current, fails, asked[3][80];
template <int I> void kernel() {}
template <class F>
cudaError_t cudaFuncSetAttribute(F* f, int, int bytes) {
  if (fails) return --fails, cudaErrorInvalidValue;
  ++asked[f == kernel<1> ? 1 : 2][current];
  return bytes == 100 ? cudaSuccess : cudaErrorInvalidValue;
}
%s
extern "C" int call(int k, int device, int fail) {
  xg_ctx c{current = device};
  fails = fail;
  return k == 1 ? allow_smem<kernel<1>>(&c, 100) : allow_smem<kernel<2>>(&c, 100);
}
extern "C" int count(int k, int device) { return asked[k][device]; }
"""


def test_smem_is_allowed_once_per_kernel_and_device(tmp_path):
    lib = hk.build(tmp_path, CODE % hk.cut(hk.source("xg_internal.hpp"), "allow_smem"))
    assert lib.call(1, 0, 1) == 1  # a failure is not taken for done
    for _ in range(3):
        for device in (0, 1, 63):
            assert lib.call(1, device, 0) == 0
    assert [lib.count(1, d) for d in (0, 1, 63, 2)] == [1, 1, 1, 0]
    assert lib.call(2, 1, 0) == 0 and lib.count(2, 1) == 1  # each kernel for itself
    for _ in range(2):  # past the last bit: every time, never left out
        assert lib.call(1, 70, 0) == 0
    assert lib.count(1, 70) == 2


def test_no_device_answers_at_file_scope():
    """No variable of a source file's scope but constants, kernels' own arrays and
    the once-per-device look-up of the allocation-free time step."""
    known = {"xg_noalloc.cu": {"g_dt_scratch", "g_scratch_ptr", "g_scratch_once", "g_scratch_err"}}
    for f in sorted(os.listdir(hk.CSRC)):
        found = set()
        for d in hk.definitions(hk.source(f)):
            head = re.sub(r"//[^\n]*", "", d).strip()
            if "(" in head.split("=")[0].replace("__align__(256)", "") or re.match(
                    r"(template|struct|class|enum|constexpr|using|typedef|static constexpr|#)",
                    head):
                continue
            m = re.match(r"[\w:*<>\s]*?[\s*](\w+)\s*(\[[^\]]*\])?\s*(=|;|\{)",
                         head.replace("__align__(256)", ""))
            if m:
                found.add(m.group(1))
        assert found == known.get(f, set()), f
