"""The table of kept tensor maps, compiled for the host: once every cache of a model has been seen, none is encoded again,
however the caches' addresses are spaced."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyquant_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <memory>
#include "hq_kept.h"
// misses of the third round over `layers` caches `stride` bytes apart (0: anywhere); -1 if a wrong value came back
static int misses(int layers, uint64_t stride, uint64_t first, int stale) {
  std::unique_ptr<hq::Kept<hq::PlanesKey, long>> kept(new hq::Kept<hq::PlanesKey, long>());
  auto key_of = [&](uint64_t address) {
    hq::PlanesKey k; k.base = (const void*)address; k.tokens = 4096; k.planes = 16; k.row = 64; k.unit = 32; return k;
  };
  uint64_t x = first | 1;
  auto next = [&] { x = x * 6364136223846793005ull + 1442695040888963407ull; return (x >> 20) & 0x7FFFFFFFFF00ull; };
  for (int i = 0; i < stale; ++i) kept->keep(key_of(next()), -7);              // caches of programs gone by
  uint64_t base[256];
  for (int i = 0; i < layers; ++i) base[i] = stride ? first + stride * i : next();
  int n = 0;
  for (int round = 0; round < 3; ++round) {
    n = 0;
    for (int i = 0; i < layers; ++i) {
      const hq::PlanesKey k = key_of(base[i]);
      const long* v = kept->find(k);
      if (v == nullptr) { ++n; kept->keep(k, (long)i); }
      else if (*v != i) return -1;
      hq::PlanesKey other = k; other.tokens += 128;                            // a cache that has grown is another entry
      if (kept->find(other) != nullptr) return -1;
    }
  }
  return n;
}
int main(int argc, char** argv) {
  std::printf("%d\n", misses(std::atoi(argv[1]), std::strtoull(argv[2], nullptr, 0), std::strtoull(argv[3], nullptr, 0), std::atoi(argv[4])));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("kept")
    (d / "kept.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, "-o", str(d / "kept"), str(d / "kept.cpp")], check=True)
    return str(d / "kept")


def misses(program, layers, stride, first, stale=0):
    return int(subprocess.run([program, str(layers), hex(stride), hex(first), str(stale)], check=True, capture_output=True, text=True).stdout)


@pytest.mark.parametrize("layers,stale", [(8, 0), (32, 0), (32, 500), (48, 0)])
@pytest.mark.parametrize("stride", [0, 1 << 20, 2 << 20, 0x2C0000, 0x1300000, 33 << 20, 512])
def test_a_models_caches_all_stay(program, layers, stale, stride):
    bad = [first for first in range(0x7F0000000000, 0x7F0000000000 + 40 * 0x1234500, 0x1234500)
           if misses(program, layers, stride, first, stale) != 0]
    assert not bad


def test_more_caches_than_places_still_give_the_right_map(program):
    assert misses(program, 200, 1 << 21, 0x7F0000000000) > 0
