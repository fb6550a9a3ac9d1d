"""The rows that a warp of the forward projection marches over and their parts
(csrc/row_parts.h, compiled here for the host), for every warp of fan geometries
whose outer rays miss the image and include some nearly parallel to its columns:
a part lies within the image's rows or is empty, the parts of a range follow one
another without gaps, and no row in which a ray comes within half + 2 of the
image's centre column is left out."""
import ctypes
import subprocess

import numpy as np
import pytest

from imgrecsrc_b200 import build

# (n, W, P, d): unit pitch and beam, every view
GEOMS = [(1136, 1617, 668, 3408.0), (944, 1465, 716, 2360.0), (950, 1859, 504, 3800.0), (933, 2288, 672, 1866.0),
         (812, 2290, 940, 2436.0), (512, 1024, 360, 2048.0)]
SOURCE = r"""
#include "row_parts.h"
using namespace ctprj;
// rows of the warps of 32 rays (A[i], S[i]), as the kernel's reduction forms
// them, and their parts: out[warp][0] all rows, [1 + s] part s of R
extern "C" void warp_parts(const float *A, const float *S, int rays, int half, int R, int *out)
{
    for (int w = 0; w * 32 < rays; ++w) {
        RowRange all = no_rows(half);
        for (int i = w * 32; i < rays && i < w * 32 + 32; ++i) {
            const RowRange r = ray_rows(A[i], S[i], half);
            all.bottom = r.bottom < all.bottom ? r.bottom : all.bottom;
            all.top = r.top > all.top ? r.top : all.top;
        }
        int *o = out + w * 2 * (R + 1);
        o[0] = all.bottom; o[1] = all.top;
        for (int s = 0; s < R; ++s) {
            const RowRange p = part_rows(all, s, R);
            o[2 + 2 * s] = p.bottom; o[3 + 2 * s] = p.top;
        }
    }
}
"""


@pytest.fixture(scope="module")
def warp_parts(tmp_path_factory):
    d = tmp_path_factory.mktemp("row_parts")
    (d / "p.cpp").write_text(SOURCE)
    # -ftrapv: an overflow of the row arithmetic ends the test
    subprocess.run(["g++", "-std=c++17", "-O2", "-ftrapv", "-shared", "-fPIC", "-I", build.CSRC, str(d / "p.cpp"),
                    "-o", str(d / "p.so")], check=True)
    f = ctypes.CDLL(str(d / "p.so")).warp_parts

    def call(A, S, half, R):
        A, S = np.ascontiguousarray(A, np.float32), np.ascontiguousarray(S, np.float32)
        out = np.zeros(((len(A) + 31) // 32, R + 1, 2), np.int32)
        ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        f(ptr(A), ptr(S), len(A), half, R, ptr(out))
        return out
    return call


def rays(n, W, P, d, b):
    """A and S of the rays' crossings xc = A - y S in base view b."""
    th = float((np.float32(2) * np.float32(b) * np.float32(3.14159265359)) / np.float32(P))
    c, s = np.cos(th), np.sin(th)
    k0 = 1 if W % 2 == 0 else 0
    t = np.arange(k0, W) - W // 2 + 0.0
    A, S = [], []
    for edge, sg in ((t - 0.5, 0.5), (t + 0.5, -0.5)):
        qx, qy = edge * c + d * s, -edge * s + d * c
        A.append(((d * edge - np.where(qx > 0, sg, -sg) * qx) / qy).astype(np.float32))
        S.append((qx / qy).astype(np.float32))
    return np.float32(0.5) * (A[0] + A[1]), np.float32(0.5) * (S[0] + S[1])


@pytest.mark.parametrize("n, W, P, d", GEOMS)
def test_parts_stay_in_the_image(warp_parts, n, W, P, d):
    half = (n - 1) // 2
    y = np.arange(-half, half + 1)
    empty = 0
    for b in range(P // 8 + 1):
        A, S = rays(n, W, P, d, b)
        for R in (1, 2, 4, 8):
            out = warp_parts(A, S, half, R)
            lo, hi = out[:, 1:, 0].astype(np.int64), out[:, 1:, 1].astype(np.int64)
            some = hi >= lo
            assert (lo[some] >= -half).all() and (hi[some] <= half).all()
            # together the warp's rows, each once, from the top down
            bottom, top = out[:, 0, 0].astype(np.int64), out[:, 0, 1].astype(np.int64)
            rows = np.maximum(top - bottom + 1, 0)
            assert (np.where(some, hi - lo + 1, 0).sum(1) == rows).all()
            full = rows > 0
            assert (hi[full, 0] == top[full]).all() and (lo[full, -1] == bottom[full]).all()
            assert (lo[full, :-1] == hi[full, 1:] + 1).all()
            assert not some[~full].any()
            empty += (~full).sum()
        if b % 8 == 0:
            xc = A[:, None] - y[None, :] * S[:, None]
            near = np.abs(xc) <= half + 2
            i, j = np.nonzero(near)
            assert (bottom[i // 32] <= y[j]).all() and (y[j] <= top[i // 32]).all()
    assert empty > 0
