"""The shared-memory rule of the one-launch loops' meetings (grid_sums.cuh): a
buffer that every warp of a block reads (sums_post, sums_of_block) is not folded
into again before a barrier.  Checked on the source of each loop, its body taken
twice in a row so that the step from one iteration to the next is covered;
barriers that only some plans reach (inside a lambda) do not count."""
import os
import re
import subprocess

import pytest

from imgrecsrc_b200 import build

STEP = re.compile(r"(sums_fold|sums_post|sums_wait|sums_of_block|__syncthreads)\(((?:[^()]|\([^()]*\))*)\)")


def loop_body(source, kernel):
    """Text of the iteration loop (`for` with round or without a condition) of a kernel."""
    text = open(os.path.join(build.CSRC, source)).read()
    at = text.index("\n" + kernel) if "\n" + kernel in text else text.index(kernel)
    at = re.compile(r"for \((unsigned round = 1; !st\.done; \+\+round|;;)\) \{").search(text, at).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return re.sub(r"//[^\n]*", "", text[at:end - 1])


@pytest.mark.parametrize("source, kernel", [("tv.cu", "k_tv_loop(const TvArgs"), ("wavelet.cu", "k_admm_loop(const AdmmLoopArgs")])
def test_no_fold_into_a_buffer_that_is_being_read(source, kernel):
    steps = [(m.group(1), m.group(2).split(",")[-1].strip()) for m in STEP.finditer(loop_body(source, kernel))]
    names = [s for s, _ in steps]
    assert names.count("sums_fold") == 2 and names.count("sums_post") == names.count("sums_of_block") == 1
    reading, folded = set(), set()
    for step, buf in steps + steps:
        if step in ("__syncthreads", "sums_wait"):   # sums_wait ends with a barrier
            reading.clear()
            folded.clear()
        elif step == "sums_fold":
            assert buf not in reading, "%s folds into %s while it is being read" % (kernel, buf)
            folded.add(buf)
        else:
            assert buf not in folded, "%s reads %s before a barrier" % (kernel, buf)
            reading.add(buf)


def test_a_block_that_gave_up_voids_the_result(tmp_path):
    """Block 0 may finish the last round while another block gives up: the state
    then says done, and only the failure word tells.  The rule (loop_met) run on
    the host, and that both loops' hosts go by it."""
    (tmp_path / "met.cu").write_text('#include "ctprj_internal.h"\n#include "grid_sums.cuh"\nusing namespace ctprj;\n'
                                     "int main() { return loop_met(1, 0) && !loop_met(1, 1) && !loop_met(0, 0) && "
                                     "!loop_met(0, 1) ? 0 : 1; }\n")
    subprocess.run([build.nvcc(), "-std=c++17", "-I", build.CSRC, str(tmp_path / "met.cu"), "-o",
                    str(tmp_path / "met")] + build.ARCH, check=True)
    assert subprocess.run([str(tmp_path / "met")]).returncode == 0
    for source in ("tv.cu", "wavelet.cu"):
        text = open(os.path.join(build.CSRC, source)).read()
        assert len(re.findall(r"started && loop_met\(h\.st\.done, h\.failed\)", text)) == 1


def test_the_count_of_arrivals_may_wrap(tmp_path):
    """Arrivals are counted in 32 bits: in the rounds around 2^32 / blocks a wait
    still ends when the round's last block is in, and not before."""
    (tmp_path / "count.cu").write_text(r"""
#include "ctprj_internal.h"
#include "grid_sums.cuh"
using namespace ctprj;
int main()
{
    for (unsigned blocks : {1u, 148u, 592u}) {
        const unsigned long long wrap = (1ull << 32) / blocks;
        for (unsigned long long round = 1; round < wrap + 3; round = round == 3 ? wrap - 3 : round + 1) {
            const unsigned want = (unsigned)round * blocks;
            for (unsigned long long in = (round - 1) * blocks; in < (round + 1) * blocks; ++in)
                if (all_in((unsigned)in, want) != (in >= round * blocks)) return 1;
        }
    }
    return 0;
}
""")
    subprocess.run([build.nvcc(), "-std=c++17", "-I", build.CSRC, str(tmp_path / "count.cu"), "-o",
                    str(tmp_path / "count")] + build.ARCH, check=True)
    assert subprocess.run([str(tmp_path / "count")]).returncode == 0
    text = open(os.path.join(build.CSRC, "grid_sums.cuh")).read()
    assert re.search(r"const unsigned want = round \* nblocks;", text) and "if (all_in(r, want)) break;" in text
