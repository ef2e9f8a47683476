"""The device arithmetic of apophis_gb300/csrc/aph_math.cuh (and aph_adjoint_math.cuh) compiled by the
host's C++ compiler, so that its integer sequences can be compared with the processor's IEEE
arithmetic without a GPU.

The header text is taken as it is, except for its four one-line assembler statements, which become
calls of functions written here: the two sign masks, and the FP32 approximations of 1/x and 1/sqrt(x),
which host_approx moves to either end of the error that the PTX documentation states (2^-23 and
2^-22.9 relative).  The device intrinsics are functions of the same names.
"""
import os
import re
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "apophis_gb300", "csrc")

SHIM = r"""
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
using std::abs;
using std::fma;
using std::max;
using std::min;
using std::sqrt;
template <class To, class From> static inline To bits_as(From x) {
  static_assert(sizeof(To) == sizeof(From), "");
  To r;
  std::memcpy(&r, &x, sizeof r);
  return r;
}
static inline int __double2hiint(double x) { return (int)(unsigned)(bits_as<uint64_t>(x) >> 32); }
static inline int __double2loint(double x) { return (int)(unsigned)bits_as<uint64_t>(x); }
static inline double __hiloint2double(int hi, int lo) {
  return bits_as<double>(((uint64_t)(unsigned)hi << 32) | (unsigned)lo);
}
static inline long long __double_as_longlong(double x) { return bits_as<long long>(x); }
static inline double __longlong_as_double(long long x) { return bits_as<double>(x); }
static inline unsigned __float_as_uint(float x) { return bits_as<unsigned>(x); }
static inline float __uint_as_float(unsigned x) { return bits_as<float>(x); }
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __ddiv_rn(double a, double b) { return a / b; }
static inline double __drcp_rn(double a) { return 1.0 / a; }
static inline double __dsqrt_rn(double a) { return std::sqrt(a); }
static inline double rsqrt(double a) { return 1.0 / std::sqrt(a); }
// where the approximations lie in their error: -1 and 1 the ends, 0 the middle
static double host_approx = 0.0;
static inline float host_rcp(float x) { return (float)((1.0 / x) * (1.0 + host_approx * 1.19209290e-7)); }
static inline float host_rsqrt(float x) {
  return (float)((1.0 / std::sqrt((double)x)) * (1.0 + host_approx * 1.27765998e-7));
}
extern "C" void set_approx(double where) { host_approx = where; }
"""

ASM = [
    (r'asm\("and\.b32 %0, %1, 0x7fffffff;"\s*:\s*"=r"\(r\)\s*:\s*"r"\((.*?)\)\);\n', r"r = (unsigned)(\1) & 0x7fffffffu;\n"),
    (r'asm\("xor\.b32 %0, %1, %2;"\s*:\s*"=r"\(hi\)\s*:\s*"r"\((.*?)\),\s*"r"\((.*?)\)\);\n', r"hi = (\1) ^ (int)(\2);\n"),
    (r'asm\("rcp\.approx\.ftz\.f32 %0, %1;"\s*:\s*"=f"\(r\)\s*:\s*"f"\((.*?)\)\);\n', r"r = host_rcp(\1);\n"),
    (r'asm\("rsqrt\.approx\.ftz\.f32 %0, %1;"\s*:\s*"=f"\(r\)\s*:\s*"f"\((.*?)\)\);\n', r"r = host_rsqrt(\1);\n"),
]


def compiler():
    return shutil.which("g++") or shutil.which("c++")


def build(folder, exact, body, includes=("aph_math.cuh",)):
    """The path of a shared library of body, which sees the device arithmetic of the mode."""
    folder = str(folder)
    for name in ("aph_math.cuh", "aph_adjoint_math.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        if name == "aph_math.cuh":
            for pattern, call in ASM:
                text, n = re.subn(pattern, call, text, flags=re.S)
                assert n == 1, pattern
        assert "asm(" not in text and "asm volatile" not in text
        with open(os.path.join(folder, name), "w") as f:
            f.write(text)
    with open(os.path.join(folder, "cuda_runtime.h"), "w") as f:
        f.write(SHIM)
    tag = "exact" if exact else "fast"
    src, so = os.path.join(folder, tag + ".cpp"), os.path.join(folder, tag + ".so")
    with open(src, "w") as f:
        f.write("#define APH_EXACT %d\n" % exact)
        for name in includes:
            f.write('#include "%s"\n' % name)
        f.write("using namespace aph;\n" + body)
    subprocess.check_call([compiler(), "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-w", "-shared",
                           "-fPIC", "-I", folder, src, "-o", so])
    return so
