"""The wavelet map's workspace when there is no memory for more partial sums: it
keeps what it has, since the reconstruction loop uses it again and counts on a
buffer of the first size.  WvltProx::reserve_parts compiled for the host with an
allocator that fails on demand."""
import os
import re
import subprocess

from imgrecsrc_b200 import build

SOURCE = r"""
#include <cstdlib>
typedef void *cudaStream_t;
enum { CTPRJ_OK = 0 };
static bool full = false;
static int cudaMallocAsync(void **p, size_t bytes, cudaStream_t) { if (full) return 2; *p = malloc(bytes); return 0; }
static int cudaFreeAsync(void *p, cudaStream_t) { free(p); return 0; }
static int cuda_error(int e, const char *) { return e; }
struct WvltProx { double *part = nullptr; size_t part_cap = 0; int reserve_parts(size_t need, cudaStream_t s); };
@FUNCTION@
int main()
{
    WvltProx w;
    if (w.reserve_parts(100, nullptr) || w.part_cap != 100) return 1;
    double *first = w.part;
    full = true;
    if (!w.reserve_parts(200, nullptr)) return 2;
    if (w.part != first || w.part_cap != 100) return 3;      // still there
    if (w.reserve_parts(50, nullptr) || w.part != first) return 4;
    full = false;
    if (w.reserve_parts(200, nullptr) || !w.part || w.part_cap != 200) return 5;
    w.part[199] = 1.0;
    free(w.part);
    return 0;
}
"""


def test_a_failed_allocation_keeps_the_buffer(tmp_path):
    text = open(os.path.join(build.CSRC, "wavelet.cu")).read()
    function = re.search(r"^int WvltProx::reserve_parts\(.*?^}\n", text, re.S | re.M).group(0)
    (tmp_path / "w.cpp").write_text(SOURCE.replace("@FUNCTION@", function))
    subprocess.run(["g++", "-std=c++17", str(tmp_path / "w.cpp"), "-o", str(tmp_path / "w")], check=True)
    assert subprocess.run([str(tmp_path / "w")]).returncode == 0
