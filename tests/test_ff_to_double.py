"""The float-float pair to double conversion of the mixed form's kernels
(ff_to_d, compiled for the host from its source): the double that an FP64
addition of the two parts gives, at the edges of its integer form (powers of
two, where the units change; parts of exactly half a unit; ties to even; the
smallest high part it takes) and at random."""
import ctypes
import pathlib
import re
import subprocess

import numpy as np
import pytest

CSRC = next(pathlib.Path(__file__).resolve().parents[1].glob("4d-*/csrc"))

SHIM = """
#include <math.h>
#include <string.h>
#define __device__
#define __forceinline__ inline
struct ff { float h, l; };
static unsigned __float_as_uint(float f) { unsigned u; memcpy(&u, &f, 4); return u; }
static float __uint_as_float(unsigned u) { float f; memcpy(&f, &u, 4); return f; }
static int __float2int_rn(float f) { return (int)lrintf(f); }
static double __longlong_as_double(long long v) { double d; memcpy(&d, &v, 8); return d; }
static double __hiloint2double(int h, int l) { return __longlong_as_double((long long)(((unsigned long long)(unsigned)h << 32) | (unsigned)l)); }
%s
extern "C" void convert(long long n, const float *h, const float *l, double *out)
{
    for (long long q = 0; q < n; ++q)
        out[q] = ff_to_d(ff{h[q], l[q]});
}
"""


def _function(text, name):
    start = re.search(r"__device__ __forceinline__ double %s\(" % name, text).start()
    return text[start:text.index("\n}\n", start) + 3]


@pytest.fixture(scope="module")
def convert(tmp_path_factory):
    d = tmp_path_factory.mktemp("ff")
    src = _function((CSRC / "ss4d_sweep.cuh").read_text(), "f2d_bits") + \
        _function((CSRC / "ss4d_ff.cuh").read_text(), "ff_to_d")
    (d / "c.cpp").write_text(SHIM % src)
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "c.so"), str(d / "c.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "c.so"))

    def run(h, l):
        h, l = np.ascontiguousarray(h, np.float32), np.ascontiguousarray(l, np.float32)
        out = np.empty(h.size)
        p = [ctypes.c_void_p(a.ctypes.data) for a in (h, l, out)]
        lib.convert(ctypes.c_longlong(h.size), *p)
        return out
    return run


def test_pair_to_double_is_the_fp64_sum(convert):
    rng = np.random.default_rng(1)
    h = [np.float32(2.0) ** np.arange(-125, 127, dtype=np.float32)]
    h.append(np.nextafter(h[0], np.float32(0)))
    h.append(np.nextafter(h[0], np.float32(np.inf)))
    h.append((rng.uniform(1, 2, 20000) * 2.0 ** rng.integers(-100, 100, 20000)).astype(np.float32))
    h = np.concatenate(h)
    unit = np.spacing(h)
    for part in (0.0, 0.5, -0.5, 0.25, -0.25, 2.0 ** -29, -(2.0 ** -29), 1.5 * 2.0 ** -29, -2.5 * 2.0 ** -29, 2.0 ** -60,
                 1.0, -1.0, None):
        f = rng.uniform(-0.5, 0.5, h.size) if part is None else part
        with np.errstate(under="ignore"):
            l = (unit.astype(np.float64) * f).astype(np.float32)
        l[np.abs(l) < np.finfo(np.float32).tiny] = 0.0  # the conversions drop subnormal parts
        assert np.array_equal(convert(h, l), h.astype(np.float64) + l.astype(np.float64)), part
        assert np.array_equal(convert(-h, l), -h.astype(np.float64) + l.astype(np.float64)), part
    assert np.array_equal(convert([0.0, np.inf], [0.0, 0.0]), [0.0, np.inf])
    assert np.isnan(convert([np.nan, 1.0], [0.0, np.nan])).all()
