"""Host-side parts of the projections of 9 to 64 rows (csrc/decoder_rows.cuh), compiled with g++; no GPU."""

import os
import subprocess

import pytest

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


@pytest.mark.parametrize("weight_rows,step,most", [(64, 8, 64), (768, 8, 64), (2304, 8, 64), (4096, 16, 128), (2048, 8, 64), (22016, 16, 128)])
def test_blocks_are_planned_as_they_are_launched(tmp_path, weight_rows, step, most):
    """The plan counts the blocks of its own grid (33 to 48 rows in tiles of 16 are three tiles, not four), and no
    other sizes of a block are cheaper by the rule that it states."""
    lines = _run(tmp_path, r"""
#include "decoder_rows_plan.h"
#include <cstdio>
int main() {
  for (int rows = 1; rows <= 64; ++rows) {
    const spsattn::RowsTiles t = spsattn::rows_tiles(%d, rows, 148, %d, %d);
    std::printf("%%d %%d %%d %%lld\n", rows, t.bn, t.bm, t.blocks);
  }
}
""" % (weight_rows, step, most))
    for rows, bn, bm, blocks in lines:
        def launched(n, m):
            return -(-weight_rows // n) * -(-rows // m)

        def cost(n, m):
            return -(-launched(n, m) // 148) * (n + m + 16)

        assert blocks == launched(bn, bm)
        assert bn % step == 0 and bn <= most and bm % 16 == 0 and bm <= -(-rows // 16) * 16
        assert cost(bn, bm) == min(cost(n, m) for n in range(step, most + 1, step) for m in (16, 32, 48, 64) if m < rows + 16)


def test_steps_of_few_rows_keep_the_projections_that_are_faster(tmp_path):
    """Up to 8 rows, up to 16 below 384 columns, and where launches are not captured up to more rows the less a layer
    weighs, decoder_step.cuh is ahead (figures beside the rule)."""
    lines = _run(tmp_path, r"""
#include "decoder_rows_plan.h"
#include <cstdio>
#include <initializer_list>
int main() {
  for (int captured : {0, 1})
    for (int rows = 1; rows <= 16; ++rows)
      for (int hidden : {64, 256, 320, 384, 512, 768, 1024, 2048})
        std::printf("%d %d %d %d\n", captured, rows, hidden, spsattn::rows_faster(rows, hidden, hidden * 8 / 3 / 64 * 64, captured));
}
""")
    first = {384: 17, 512: 17, 768: 13, 1024: 9, 2048: 9}
    for captured, rows, hidden, faster in lines:
        assert faster == (hidden >= 384 and rows >= (9 if captured else first[hidden]))


@pytest.mark.parametrize("rows,hidden,inter,slower", [(64, 4096, 11008, True), (49, 2560, 10240, True), (64, 8192, 28672, True),
                                                      (48, 4096, 11008, False), (64, 3072, 8192, False), (64, 2048, 8192, False), (1, 8192, 28672, False)])
def test_wide_steps_of_many_rows_keep_the_library_projections(rows, hidden, inter, slower):
    from sps_b200.generation import row_tiles_slower
    assert row_tiles_slower(rows, hidden, inter) is slower
