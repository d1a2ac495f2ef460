"""How the F32 matvecs share out a block's shared memory (csrc/mv_room.h), on the host: a small program is compiled against the
header and asked for widths a model has and for widths that 32-bit arithmetic cannot hold. Skipped where g++ is missing."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "mv_room.h"
using namespace osmos::mv_room;
int main(int argc, char** argv) {
  for (int i = 1; i + 2 < argc; i += 3) {  // columns, tokens, bytes of 256 values
    const uint32_t cols = (uint32_t) strtoul(argv[i], 0, 10), n = (uint32_t) strtoul(argv[i + 1], 0, 10);
    const uint64_t stretch = strtoull(argv[i + 2], 0, 10);
    const Passes p = pair_passes(225 * 1024, 8, 8, n, cols, [&](uint32_t seg) {
      const uint32_t k = cols / 256 < seg ? cols / 256 : seg;
      return 2 * 16 * 2 * ((k * (uint32_t) stretch + 46u + 63u) / 128u * 128u + 64u);
    });
    printf("%u %u %u\n", p.seg, p.fit, staged_slots(226 * 1024 - 16, 16, 4, cols / 256 * stretch, n, cols));
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def room(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("room")
    src, exe = d / "room.cpp", d / "room"
    src.write_text(PROGRAM)
    r = subprocess.run([gxx, "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "libosmos_b200", "csrc"), "-o", str(exe), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def ask(cases):
        r = subprocess.run([str(exe)] + [str(v) for c in cases for v in c], capture_output=True, text=True)
        assert r.returncode == 0, "the program ended with %d" % r.returncode
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return ask


STRETCHES = [136, 144, 176, 210, 272]  # bytes of 256 values, over the types


def test_widths_of_models(room):
    cases = [(c, n, b) for c in (256, 2048, 4096, 7168, 16384) for n in (1, 5, 8) for b in STRETCHES]
    for (cols, n, stretch), (seg, fit, slots) in zip(cases, room(cases)):
        assert seg in (1, 2, 4, 8) and 1 <= fit <= 8 and fit * cols * 4 < 225 * 1024, (cols, n, stretch)
        x = (n * cols * 4 + 127) // 128 * 128
        want = min(4, (226 * 1024 - 16 - x) // (16 * (cols // 256 * stretch))) if x < 226 * 1024 - 16 else 0
        assert slots == want, (cols, n, stretch)


def test_widths_past_32_bits(room):
    """x of eight tokens, of one, a ring's bytes: each past 4 GB at some of these; there is room for none"""
    cols = [2 ** 16, 2 ** 26, 2 ** 27, 2 ** 28, 2 ** 29, 2 ** 30 - 4096, 2 ** 30 - 512, 2 ** 30 - 256, 2 ** 30, 2 ** 31, 2 ** 32 - 256]
    cases = [(c, n, b) for c in cols for n in (1, 2, 4, 8) for b in STRETCHES + [1024]]
    assert room(cases) == [(0, 0, 0)] * len(cases)
