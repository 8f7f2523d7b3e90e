"""Runs parts of the CUDA sources on the CPU: a piece of a source file, cut out
by its text, compiled by the host compiler with stand-ins for the CUDA names it
uses. Index arithmetic, choices and which loads a kernel issues are then the
code's own, not a restatement of it."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flowlab_gb300", "csrc")

PRELUDE = r"""
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#define __device__
#define __host__
#define __global__
#define __restrict__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
template <class To, class From> inline To bits_as(From v) { To t; std::memcpy(&t, &v, sizeof t); return t; }
inline unsigned __float_as_uint(float v) { return bits_as<unsigned>(v); }
inline int __float_as_int(float v) { return bits_as<int>(v); }
inline float __int_as_float(int v) { return bits_as<float>(v); }
inline float __uint_as_float(unsigned v) { return bits_as<float>(v); }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __fadd_rd(float a, float b) {  // exact in double for a in [0, 2^23) and b = 2^23, then rounded down
  const double s = (double)a + (double)b;
  float f = (float)s;
  return (double)f > s ? std::nextafterf(f, -INFINITY) : f;
}
using std::max;
using std::min;
"""


def source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return fh.read()


def between(text, start, end):
    """The text from `start` up to (not including) `end`."""
    a = text.index(start)
    return text[a:text.index(end, a)]


def block(text, start):
    """The definition that begins with `start`, to its closing brace (and the
    semicolon after it, if there is one)."""
    a = text.index(start)
    depth = 0
    for k in range(text.index("{", a), len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[a:k + 1] + (";" if text[k + 1:k + 2] == ";" else "")
    raise ValueError(start)


def launches_as_calls(text):
    """kernel<<<grid, block, shared, stream>>>(args) as kernel(args)."""
    return re.sub(r"<<<.*?>>>", "", text, flags=re.S)


def run(tmp_path, code):
    """Compiles and runs a C++ program; its standard output."""
    src, exe = tmp_path / "host.cpp", tmp_path / "host"
    src.write_text(PRELUDE + code)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, "exit %d\n%s%s" % (out.returncode, out.stdout, out.stderr)
    return out.stdout
