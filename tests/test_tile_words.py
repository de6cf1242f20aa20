"""The debug tap of the tile lists reads what the raster reads: the bins'
ranges and the tiles' words (csrc/bins.cuh), on the CPU; on the GPU the taps
equal the oracle's lists at pair counts around a word (32 positions) and a
group of words (256)."""

import subprocess

import numpy as np
import pytest

import build as native
import gsplat_scenes
from test_gpu_parity import _compare_stages, _render

# Reads n, first, end and n lists of 16 tile bits; writes their words as the
# range build lays them out, flips bit `flip` of the words (-1: none) and
# prints every tile's positions in [first, end).
PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "bins.cuh"
using namespace gsr;
int main() {
  unsigned n, first, end;
  long flip;
  if (std::scanf("%u %u %u %ld", &n, &first, &end, &flip) != 4) return 1;
  std::vector<uint32_t> words(tile_words(n));
  for (unsigned i = 0; i < n; ++i) {
    unsigned tiles;
    if (std::scanf("%u", &tiles) != 1) return 1;
    for (unsigned t = 0; t < kBinTiles; ++t)
      if (tiles >> t & 1u) words.at(tile_word(i / 32, t)) |= 1u << i % 32;
  }
  if (flip >= 0) words.at(flip / 32) ^= 1u << flip % 32;
  for (unsigned t = 0; t < kBinTiles; ++t) {
    each_tile_position(words.data(), first, end, t, [](uint32_t i) { std::printf("%u ", i); });
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("words")
    (d / "words.cpp").write_text(PROGRAM)
    subprocess.run([native.CXX, "-std=c++17", "-O1", "-I", native.CSRC, str(d / "words.cpp"), "-o",
                    str(d / "words")], check=True)

    def lists(tiles, first, end, flip=-1):
        text = f"{len(tiles)} {first} {end} {flip}\n" + " ".join(map(str, tiles))
        out = subprocess.run([str(d / "words")], input=text, capture_output=True, text=True,
                             check=True).stdout
        return [list(map(int, line.split())) for line in out.split("\n")[:16]]

    return lists


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 600])
def test_tile_lists_are_read_from_the_words(walk, n):
    tiles = np.random.default_rng(n).integers(0, 1 << 16, n)
    first, end = n // 5, n - n // 7
    want = [[i for i in range(first, end) if tiles[i] >> t & 1] for t in range(16)]
    assert walk(tiles, first, end) == want
    # a wrong word and a wrong range both show
    assert walk(tiles, first, end, flip=32 * 8 * 3 + first % 32 + 32 * (first // 32 % 8)
                + 32 * 128 * (first // 256)) != want
    assert walk(tiles, first, end - 1) != want or not (tiles[end - 1] & 0xffff)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(64, 64), (65, 64)])  # one bin, two bins
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 511, 1023, 1025])
def test_tile_lists_around_words_and_groups(oracle, w, h, n):
    rng = np.random.default_rng(n)
    means = rng.normal(0.0, 0.1, (n, 3)).astype(np.float32)
    scene = gsplat_scenes.make_scene(rng, means, -2.0, 0.5, 0.0, 1.0, 0)
    cam = gsplat_scenes.camera((0.0, 0.0, -4.0), (0, 0, 0), 55.0)
    sv = oracle.SceneView(scene)
    fr = oracle.Frame(sv, cam, w, h)
    assert fr.drawn == n
    ctx = _render(scene, cam, w, h)
    _compare_stages(ctx, fr, sv)
