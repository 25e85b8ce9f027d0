"""Pieces of a CUDA source compiled for the host, to run a kernel's own text on
the CPU where the GPU cannot show what a test asks for: the named top-level
definitions are cut out of the file and compiled by g++ behind stand-ins for
CUDA's keywords, vector types and bit casts, one thread at a time."""

import ctypes
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xyst_gb300",
                    "csrc")

SHIM = r"""
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <initializer_list>
#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __shared__ static
using std::fabs;
using std::fmax;
using std::fmin;
struct Dim3 { unsigned x = 0, y = 0, z = 0; };
static Dim3 threadIdx, blockIdx, blockDim, gridDim;
#define XG_VEC(T, B) struct T##2 { B x, y; }; struct T##4 { B x, y, z, w; };          \
  static inline T##2 make_##T##2(B x, B y) { return T##2{x, y}; }                     \
  static inline T##4 make_##T##4(B x, B y, B z, B w) { return T##4{x, y, z, w}; }
XG_VEC(int, int) XG_VEC(uint, unsigned) XG_VEC(float, float) XG_VEC(double, double)
XG_VEC(longlong, long long) XG_VEC(ulonglong, unsigned long long)
template <class T> static inline T __ldg(const T* p) { return *p; }
template <class T, class S> static inline T bits_of(S s) {
  static_assert(sizeof(T) == sizeof(S), "same size");
  T t;
  std::memcpy(&t, &s, sizeof(t));
  return t;
}
static inline long long __double_as_longlong(double v) { return bits_of<long long>(v); }
static inline double __longlong_as_double(long long v) { return bits_of<double>(v); }
static inline unsigned __float_as_uint(float v) { return bits_of<unsigned>(v); }
static inline int __float_as_int(float v) { return bits_of<int>(v); }
static inline float __uint_as_float(unsigned v) { return bits_of<float>(v); }
static inline int __double2hiint(double v) { return int(bits_of<uint64_t>(v) >> 32); }
static inline int __double2loint(double v) { return int(bits_of<uint64_t>(v)); }
static inline void __syncwarp() {}
"""


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def definitions(text):
    """The file's top-level definitions, in order (namespaces do not indent)."""
    out, cur, depth = [], [], 0
    for line in text.split("\n"):
        code = line.split("//")[0].rstrip()
        if depth == 0 and not cur and (not code or code[0] in "# }" or
                                       code.startswith(("namespace", "using namespace",
                                                        "extern"))):
            continue
        cur.append(line)
        depth += code.count("{") - code.count("}")
        if depth == 0 and code.endswith(("}", ";")):
            out.append("\n".join(cur))
            cur = []
    return out


def cut(text, *names):
    """The definitions of the given functions, types and constants."""
    got = []
    for d in definitions(text):
        head = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", re.sub(r"//.*", "", d))
        head = re.split(r"[({;=]", head, maxsplit=1)[0]
        if any(re.search(rf"\b{n}\b", head) for n in names):
            got.append(d)
    for n in names:
        assert any(re.search(rf"\b{n}\b", d) for d in got), f"{n} not found"
    return "\n".join(got)


def build(tmp_path, code, name="piece"):
    """The shared library of SHIM + code, loaded."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, lib = tmp_path / f"{name}.cpp", tmp_path / f"{name}.so"
    src.write_text(SHIM + code)
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-shared", "-fPIC",
                        str(src), "-o", str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(lib))
