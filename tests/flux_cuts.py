"""The cuts of the flux launches (csrc/device/flux_cut.hpp), from a small host
program: what a grid takes, whatever machine asks."""
import functools
import subprocess
import tempfile
from pathlib import Path

from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "device/flux_cut.hpp"
using namespace ostc;
// kind (air, mixture or the variant of the FP32-bulk passes), SMs, then mx my mz per block
int main(int argc, char **argv) {
  std::vector<BlockDims> blocks;
  for (int q = 3; q + 2 < argc; q += 3) blocks.push_back({std::atoi(argv[q]), std::atoi(argv[q + 1]), std::atoi(argv[q + 2])});
  const char kind = argv[1][0];
  const int sms = std::atoi(argv[2]);
  if (kind == 'a' || kind == 'm') {
    const Fp64Cut c = fp64_flux_cut(blocks, sms, kind == 'a');
    std::printf("%d %d\n", c.rows ? 1 : 0, c.kc);
  } else {
    const FluxVariant v = kFluxVariant[kind - '0'];
    std::printf("%d %d\n", march_cut(blocks, 1, v, sms), march_cut(blocks, 2, v, sms));
  }
}
"""
B200_SMS = 148


@functools.lru_cache(maxsize=None)
def _program():
    d = Path(tempfile.mkdtemp(prefix="flux_cuts_"))
    (d / "cut.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "openstc_b200" / "csrc"), str(d / "cut.cpp"), "-o",
                    str(d / "cut")], check=True)
    return str(d / "cut")


def _ask(kind, blocks, sms):
    out = subprocess.run([_program(), str(kind), str(sms), *[str(v) for b in blocks for v in b]], check=True,
                         capture_output=True, text=True).stdout.split()
    return int(out[0]), int(out[1])


def fp64_cut(*blocks, air=False, sms=B200_SMS):
    """"rows" or the planes per column."""
    rows, kc = _ask("a" if air else "m", blocks, sms)
    return "rows" if rows else kc


def march_cut(variant, *blocks, sms=B200_SMS):
    """The cells a thread of the y and of the z pass marches over."""
    return _ask(variant, blocks, sms)

# Grids on which the launches take every cut on a B200, most with a last segment
# that is not full; the FP64 ones against the per-cell kernel, the FP32-bulk ones
# against the other variants, which cut them otherwise (y and z march per variant).
FP64_GRIDS = {(33, 9, 7): "rows", (65, 37, 19): 1, (129, 65, 33): 2, (128, 64, 33): 4, (97, 61, 31): 8}
MIXED_GRIDS = {(33, 9, 7): [(1, 1)] * 4, (65, 45, 27): [(1, 1), (1, 1), (2, 2), (2, 2)],
               (97, 61, 31): [(2, 2), (2, 2), (4, 4), (4, 4)], (33, 61, 131): [(4, 4), (4, 4), (8, 8), (8, 8)],
               (129, 131, 61): [(4, 4), (4, 16), (4, 4), (4, 8)], (129, 61, 131): [(4, 4), (16, 4), (4, 4), (8, 4)]}
