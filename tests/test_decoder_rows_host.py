"""Host-side parts of the projections of 9 to 64 rows (csrc/decoder_rows.cuh), compiled with g++; no GPU."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, source: str) -> list:
    path, exe = tmp_path / "host.cpp", tmp_path / "host"
    path.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "sps_b200", "csrc"), str(path), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [[int(x) for x in line.split()] for line in out.splitlines()]


def test_every_copy_has_landed_however_the_loads_end(tmp_path):
    """A step that is given up (by the loading lane at its `stop`-th wait, or by another thread while the
    loading lane got through) leaves no copy in flight: the last copy into each stage is waited for, by
    the parity of its own turn."""
    lines = _run(tmp_path, r"""
#include "decoder_rows_ring.h"
#include <cstdio>
int main() {
  for (int stages = 1; stages <= 5; ++stages)
    for (int chunks = 1; chunks <= 13; ++chunks)
      for (int stop = 0; stop <= chunks; ++stop) {
        const int first = chunks < stages ? chunks : stages;
        int turn[5] = {}, waits = 0, next = first, bad = 0, open = 0;
        bool landed[5];
        for (int s = 0; s < stages; ++s) landed[s] = s >= first;
        const int asked = spsattn::rows_feed(first, chunks, stages,
          [&](int st, int phase) {                       // the products' turns of a stage: 0, 1, ...
            bad += phase != (turn[st] & 1) || st != next % stages;
            return waits++ != stop;
          },
          [&](int st, int j) { bad += j != next++ || st != j % stages; ++turn[st]; landed[st] = false; });
        spsattn::rows_landed(asked, stages, [&](int st, int phase) { bad += phase != (turn[st] & 1); landed[st] = true; });
        for (int s = 0; s < stages; ++s) open += !landed[s];
        const int want = first + (stop < chunks - first ? stop : chunks - first);
        std::printf("%d %d %d %d\n", bad, open, asked - want, next - want);
      }
}
""")
    assert len(lines) > 500
    assert all(line == [0, 0, 0, 0] for line in lines)
    # and the kernel asks for them whenever a wait of the block has expired, not only one of the loading lane
    kernel = open(os.path.join(ROOT, "sps_b200", "csrc", "decoder_rows.cuh")).read()
    teardown = kernel[kernel.rindex("if (*abort_flag != 0) {"):]
    assert teardown.index("rows_give_up(full0, s_asked, p.stages") < teardown.index("__syncthreads();") < teardown.index("tmem_dealloc")
