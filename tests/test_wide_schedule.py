"""Tiles of 256 x 512 (gemm2w_kernel.cuh): how they are dealt out to the SM pairs, on the CPU, and on the GPU the kinds of
schedule that small results do not have: whole tiles of the least K, cut tiles behind whole ones, the phase lock of several
rounds."""
import ctypes
import random
import subprocess

import pytest

from cute_mma_b200 import build, ops

PAIRS = 74  # of a B200

# the kernel's own schedule and launch geometry, compiled for the host; 0, or the number of the rule that does not hold
HARNESS = r"""
#include <vector>
#include "gemm2w_kernel.cuh"
using namespace b200;
extern "C" int walk(int m, int n, int raster, int gpu_pairs, int* kinds) {
  const long long tiles_m = (m + 255) / 256, tiles_n = (n + 255) / 256, halves = tiles_m * tiles_n;
  const WideGrid g = wide_grid(m, n, gpu_pairs);
  if (g.pairs < 1 || g.pairs > static_cast<unsigned>(gpu_pairs)) return 1;
  std::vector<int> seen(halves);
  const WideSchedule s(m, n, g.wide, raster, g.pairs);
  long long longest = 0, whole = 0, cut = 0, single = 0;
  for (unsigned pair = 0; pair < g.pairs; ++pair) {
    long long load = 0;
    WideItem w;
    unsigned j = 0;
    for (; s.item(pair, j, w); ++j) {
      if (j < s.full_rounds && w.halves != 2) return 2;  // the phase lock counts on every pair in these rounds
      if (w.tm >= tiles_m || w.n0 % 256 || w.n0 < 0 || w.n0 / 256 + w.halves > tiles_n || w.halves < 1 || w.halves > 2) return 3;
      for (int h = 0; h < w.halves; ++h)
        if (seen[w.tm * tiles_n + w.n0 / 256 + h]++) return 4;
      load += w.halves;
      (w.halves == 2 ? whole : (tiles_n % 2 && w.n0 / 256 == tiles_n - 1) ? single : cut) += 1;
    }
    if (j < 1 || j < s.full_rounds) return 5;  // a pair without work
    longest = load > longest ? load : longest;
  }
  for (int x : seen)
    if (x != 1) return 6;
  if (longest != (halves + gpu_pairs - 1) / gpu_pairs) return 7;
  kinds[0] = static_cast<int>(whole), kinds[1] = static_cast<int>(cut), kinds[2] = static_cast<int>(single), kinds[3] = static_cast<int>(s.full_rounds);
  return 0;
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("wide")
    (d / "walk.cu").write_text(HARNESS)
    subprocess.run([build.nvcc_path(), *build.NVCC_FLAGS, f"-I{build.CSRC}", f"-I{build.DEFAULT_CONFIG}", str(d / "walk.cu"), "-o", str(d / "walk.so"), "-lcudart"],
                   check=True)
    fn = ctypes.CDLL(str(d / "walk.so")).walk

    def call(m, n, raster=16, pairs=PAIRS):
        kinds = (ctypes.c_int * 4)()
        assert fn(m, n, raster, pairs, kinds) == 0, (m, n, raster, pairs)
        return tuple(kinds)

    return call


# (m, n): whole tiles, halves of cut tiles, halves that have no neighbour, full rounds
SCHEDULES = [((256, 512), (0, 2, 0, 0)), ((129, 257), (0, 2, 0, 0)), ((300, 700), (0, 4, 2, 0)), ((5000, 9000), (360, 0, 0, 4)), ((2048, 6656), (74, 60, 0, 1)),
             ((7308, 5888), (297, 44, 29, 4)), ((1734, 2723), (3, 64, 7, 0)), ((20000, 1100), (158, 0, 79, 2)), ((512, 26624), (74, 60, 0, 1))]


@pytest.mark.parametrize("shape,kinds", SCHEDULES, ids=lambda s: "x".join(map(str, s)))
def test_kinds_of_schedule(walk, shape, kinds):
    assert walk(*shape) == kinds


@pytest.mark.parametrize("pairs", [1, 2, 10, 66, 74])
def test_every_half_once_and_the_longest_pair_as_short_as_can_be(walk, pairs):
    rng = random.Random(pairs)
    for _ in range(3000):
        tiles = rng.choice([8, 4 * pairs, 2000])
        m = rng.randint(1, 256 * rng.randint(1, tiles))
        n = rng.randint(257, 257 + 256 * max(1, tiles * 256 // m))
        walk(m, n, rng.choice([0, 1, 8, 16]), pairs)


def bits_of_pair_tiles(shape, kind):
    import test_wide_gpu

    test_wide_gpu.test_wide_tiles_have_the_bits_of_pair_tiles(shape, kind)


KINDS = [("half", "half", "TN", 1.0, 0.0), ("half", "float", "NT", 1 / 128, 0.0), ("half", "half", "TN", 0.5, 2.0), ("float", "float", "NT", 1.0, 0.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS, ids=lambda k: "-".join(map(str, k[:3])) + ("-beta" if k[4] else ""))
@pytest.mark.parametrize("m,n,steps", [(5000, 9000, 4), (2048, 6656, 4), (2048, 6656, 5), (7308, 5888, 7), (1734, 2723, 4), (1734, 2723, 9)])
def test_whole_and_cut_tiles(lib, pair_build, m, n, steps, kind):
    """The kinds of schedule above: the least K of whole tiles (both ends, nothing between them), cut tiles behind them."""
    if not pair_build:
        pytest.skip("tiles of 256 x 512 belong to the CTA-pair build")
    bk = 64 if kind[0] == "half" else 32
    bits_of_pair_tiles((m, n, steps * bk - (24 if steps % 2 else 0)), kind)


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [0, 1], ids=["256", "512"])
def test_phase_lock_on_two_streams(lib, cuda, pair_build, wide):
    """Several rounds of whole tiles (three of 256 x 512, six of 256 x 256), started together, on two streams without a
    synchronisation between them: every launch has round counters of its own, so both finish with the bits of launches
    without the lock."""
    import torch

    if not pair_build:
        pytest.skip("the phase lock is a feature of the CTA-pair kernels")
    m, n, k = 4096, 8192, 1024
    gen = torch.Generator(device=cuda).manual_seed(78)
    A, B = (torch.randn((r, k), generator=gen, device=cuda).half() for r in (m, n))
    C = [torch.full((n, m), -7.0, dtype=torch.float16, device=cuda) for _ in range(3)]
    with ops.option("gemm_wide", wide, lib), ops.option("small_tiles", 0, lib):
        with ops.option("gemm_tile_sync", 0, lib):
            ops.gemm_tn(m, n, k, A, k, B, k, C[0], m, lib=lib)
        torch.cuda.synchronize()
        streams = torch.cuda.Stream(), torch.cuda.Stream()
        with ops.option("gemm_tile_sync", 1, lib):
            for _ in range(3):
                for s, c in zip(streams, C[1:]):
                    ops.gemm_tn(m, n, k, A, k, B, k, c, m, s.cuda_stream, lib=lib)
    torch.cuda.synchronize()
    assert ops.device_status(lib)[0] == 0
    assert torch.equal(C[0], C[1]) and torch.equal(C[0], C[2])


@pytest.mark.gpu
@pytest.mark.parametrize("t_in,t_out", [("half", "half"), ("half", "float"), ("float", "float")])
def test_ragged_edges_are_stored_as_fast(lib, cuda, pair_build, t_in, t_out):
    """One row and one column less than whole tiles, in the same C: a warp of the last tiles has 128 columns to store with checks,
    at 4 instructions a column about 1 us more than without, at 16 more than 4."""
    import torch

    from test_beta_gpu import us

    if not pair_build:
        pytest.skip("tiles of 256 x 512 belong to the CTA-pair build")
    m, n, k = 2304, 2048, 512
    A, B = (torch.randn((r, k), device=cuda).to(torch.float16 if t_in == "half" else torch.float32) for r in (m, n))
    C = torch.empty((n, m), device=cuda, dtype=torch.float16 if t_out == "half" else torch.float32)

    def call(rows, cols):
        ops.gemm_ex("T", "N", rows, cols, k, 1.0, A, k, B, k, 0.0, C, m, in_type=ops.F16 if t_in == "half" else ops.TF32,
                    out_type=ops.F16 if t_out == "half" else ops.F32, lib=lib)

    with ops.option("gemm_wide", 1, lib), ops.option("small_tiles", 0, lib):
        whole, ragged = us(lambda: call(m, n)), us(lambda: call(m - 1, n - 1))
    assert ragged - whole <= 2.5, (whole, ragged)
