"""Device headers compiled for the host: the few CUDA names that their
arithmetic uses, so that a CPU test can call the kernels' own functions."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "harm_finalwham_b200", "csrc")

STUB = r"""
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
using std::max;
using std::min;
static inline int __double2hiint(double x) { uint64_t u; memcpy(&u, &x, 8); return (int)(u >> 32); }
static inline int __double2loint(double x) { uint64_t u; memcpy(&u, &x, 8); return (int)(uint32_t)u; }
static inline double __hiloint2double(int h, int l) {
  const uint64_t u = (uint64_t)(uint32_t)h << 32 | (uint32_t)l;
  double x;
  memcpy(&x, &u, 8);
  return x;
}
"""


def build(d, source):
    """Compile a program that includes device headers; returns its path."""
    (d / "cuda_runtime.h").write_text(STUB)
    (d / "t.cc").write_text('#include <random>\n#include <stdio.h>\n#include <stdlib.h>\n#include <cuda_runtime.h>\n' + source)
    exe = str(d / "t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-ffp-contract=off", "-I", str(d), "-I", CSRC, "-o", exe,
                    str(d / "t.cc")], check=True)
    return exe
