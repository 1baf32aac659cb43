"""The converters' waits of the MX prefill kernel (csrc/mx_rings.h): a wait by parity for a phase of a slot is sound only where
the phase before is known to be complete, from the group's own waits or from stages known to have retired."""

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jax_metallib_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include <initializer_list>
#include "mx_rings.h"
int main() {
  using namespace qmm::mxp;
  for (int bits : {4, 8})
    for (int rows : {32, 64, 96}) {
      const Rings r = rings(bits, rows);
      printf("%d %d %d %d %d %d %d %d\\n", bits, rows, kGroups, kConsumed, r.slots, r.x_stages, r.raw_boxes, r.stages_per_box);
    }
}
"""


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    path = tmp_path_factory.mktemp("mx_rings")
    (path / "main.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(path / "main.cc"), "-o", str(path / "main")], check=True)
    rows = [tuple(map(int, line.split())) for line in subprocess.run([path / "main"], capture_output=True, text=True, check=True).stdout.splitlines()]
    return {row[:2]: row[2:] for row in rows}


def unsound_waits(config, stages, tiles):
    """Waits of the converters that pass while the phase before may be incomplete, in tiles of `stages` stages each."""
    groups, consumed, slots, x_stages, raw_boxes, per_box = config
    boxes = -(-stages // per_box)
    box_of = [tile * boxes + stage // per_box for tile in range(tiles) for stage in range(stages)]   # of a stage, counted over the launch
    found = []
    for group in range(groups):
        seen_x, seen_raw, asked, retired = set(), set(), set(), -1
        for c in range(group, stages * tiles, groups):
            def landed_raw(box):
                return box in seen_raw or retired >= 0 and box <= box_of[retired]

            box = box_of[c]
            if box >= raw_boxes and not landed_raw(box - raw_boxes):
                found.append(("raw", group, c))
            seen_raw.add(box)
            if c >= slots:
                before = c - slots - consumed
                if before >= 0 and before not in asked and before > retired:
                    found.append(("consumed", group, c))
                asked.add(c - slots)
                retired = max(retired, c - slots)   # MMAs retire in order
            if c >= x_stages and c - x_stages not in seen_x and c - x_stages > retired:
                found.append(("x", group, c))
            seen_x.add(c)
    return found


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("rows", [32, 64, 96])
def test_waits_by_parity_are_sound(table, bits, rows):
    for stages in range(1, 41):
        assert unsound_waits(table[bits, rows], stages, max(3, 80 // stages)) == []
