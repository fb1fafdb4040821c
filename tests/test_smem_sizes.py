"""Shared memory of the register passes, on the host: every copy that a pass makes into it ends inside
what its launch asks for, and starts on the 16 bytes an asynchronous copy needs, for every line length
and tile width."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-wave-julia_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "kwb_fast_impl.cuh"
using namespace kwb::fast;
template <class F>
void show(int n, int L, int width) {
  const size_t lines = (size_t)L * F::LP * sizeof(float2);
  printf("%d %d %d %zu %zu %zu %zu %zu\n", n, width, L, lines, lines + image_tw_bytes<F>(), eos_smem<F>(L),
         lines + image_line_bytes<F>(), pline_offset<F>(L));
}
template <int N>
void sizes() {
  using P = LinePolicy<N>;
  constexpr int G = P::template F<true>::G;
  constexpr int BIG = P::THREADS / G, SMALL = (32 / G > 2 ? 32 / G : 2);
  constexpr int MID = ((128 / G) & ~1) > SMALL ? ((128 / G) & ~1) : SMALL;
  for (int L : {BIG, MID, SMALL}) {
    show<typename P::template F<true>>(N, L, 0);
    show<typename P::template F<false>>(N, L, 1);
  }
}
int main() {
  sizes<64>(); sizes<128>(); sizes<256>(); sizes<512>(); sizes<1024>();
  sizes<96>(); sizes<160>(); sizes<192>(); sizes<320>(); sizes<80>(); sizes<640>();
  sizes<144>(); sizes<288>(); sizes<432>(); sizes<576>(); sizes<864>(); sizes<400>();
  sizes<500>(); sizes<800>(); sizes<1000>(); sizes<384>(); sizes<768>();
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_copies_stay_inside_the_shared_memory_of_a_launch(tmp_path):
    src, exe = tmp_path / "sizes.cu", tmp_path / "sizes"
    src.write_text(PROGRAM)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True, text=True)
    rows = [tuple(map(int, r.split())) for r in subprocess.run([str(exe)], check=True, capture_output=True,
                                                              text=True).stdout.splitlines()]
    assert len({r[0] for r in rows}) == 22
    for n, _, L, lines, tw_end, eos, image_end, stage in rows:
        assert lines % 16 == 0, (n, L)
        assert tw_end <= eos, (n, L, tw_end, eos)
        assert image_end <= stage, (n, L, image_end, stage)
