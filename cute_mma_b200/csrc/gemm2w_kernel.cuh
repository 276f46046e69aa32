// Plain GEMM on CTA pairs with tiles of 256 x 512: the pair tile of gemm2_kernel.cuh twice over, side by side.  Same operator,
// layouts and sums (gemm_sm80_tc.cu:95-228): every element of C is accumulated over K in the same order, bit for bit.
//
// Bound: the 1 kW power cap.  The pair kernels reach it whenever launches follow one another for more than some tens of
// milliseconds, and from there on the energy of a launch is its time (970 to 990 W on every large product, whatever the clock;
// 8192^3 half on gemm2_kernel 880 mJ, of which moving the operands without a single MMA takes about a third).  A 256 x 256
// tile loads 32 KB per CTA and 64 columns of K, 9.9 TB/s from L2 at 8192^3; two accumulators of 256 columns that share the rows
// of A load 48 KB for twice the work (8.6 -> 6.4 GB in all), and the A operand of a pair of MMAs is fetched from shared memory
// once (collector buffer, 1 %).  Long runs, us on tiles of 256 / 512: 8192^3 half 864 / 831, 4096 x 4096 x 16384 half NT 471 /
// 436, 4096^3 TF32 NT 221 / 209, 11008 x 3001 x 4096 half 252 / 219, 16384 x 4096 x 1024 half 130 / 119.  Per 64 columns of K and
// tile the pipe needs 1024 cycles, which the middle steps keep to; 2300 cycles a tile go into its two ends.
//
// Tensor memory (512 columns) holds the two accumulators of ONE tile, so nothing is left for the next one.  The halves are
// therefore run kSkew K steps apart at both ends of a tile: at the end, half 0 finishes its last kSkew steps first and its
// accumulator is drained under the last kSkew steps of half 1; the next tile starts with kSkew steps of half 0, under which
// half 1 is drained.  Eight epilogue warps take an accumulator into registers (as packed fp16 or as float), hand it back, and
// store it under the next MMAs.
//
// Roles (320 threads): warp 0 TMA producer, warp 1 tensor memory and MMA issuer (leader CTA), warps 2..9 epilogue (quadrant
// warp % 4 of the lanes, 128 columns of an accumulator each).  Barriers as in gemm2_kernel.cuh, one unit = one accumulator
// of 256 columns: unit u of a pair lives in accumulator u % 2, so a pair may also take single halves (last round).
#pragma once
#include "gemm2_kernel.cuh"

namespace b200 {

template <typename TIn_, typename TOut_, bool kMn_>
struct Gemm2WTraits {
  using TIn = TIn_;
  using TOut = TOut_;
  static constexpr bool kMn = kMn_;
  static constexpr int kBM = 128;                  // rows of C per CTA; the pair covers 256
  static constexpr int kBN = 256;                  // columns of C per accumulator (tcgen05 N); a tile has two
  static constexpr int kBNHalf = kBN / 2;          // rows of an accumulator's B tile each CTA loads
  static constexpr int kElem = sizeof(TIn);
  static constexpr int kBK = 128 / kElem;
  static constexpr int kUmmaK = 32 / kElem;
  static constexpr int kChunk = 128 / kElem;
  static constexpr int kStages = 4;
  static constexpr int kSkew = 2;                  // K steps by which the halves are apart at both ends of a tile
  static constexpr int kMinSteps = 2 * kSkew;      // least K steps of a tile
  static constexpr int kABytes = kBM * 128;
  static constexpr int kBBytes = kBNHalf * 128;    // per accumulator
  static constexpr int kStageBytes = kABytes + 2 * kBBytes;
  static constexpr int kTmemCols = 512;
  static constexpr int kEpiWarps = 8;
  static constexpr int kThreads = 64 + 32 * kEpiWarps;
  static constexpr int kNumBars = 2 * kStages + 4;
  static constexpr int kSmemBytes = kStages * kStageBytes + kNumBars * 8 + 64 + 1024;
  static constexpr int kFmt = (kElem == 2) ? kFmtF16 : kFmtTF32;
  static constexpr bool k32Atom = kMn && kElem == 4;
  static_assert(kStages >= 2 * kSkew, "the next tile's first steps must fit beside the last ones of this");
  static_assert(kSmemBytes <= 232448, "shared memory ring too large");
};

struct Gemm2WArgs {
  int m, n, k;
  void* C;
  long long ldC;
  int* status;
  int raster;                         // 0: z-curve tile order; g > 0: bands of g tile rows (tiles of 256 x 512)
  int tile_sync;                      // producers of all CTAs start each round of whole tiles together
  int* rounds;                        // 4 zeroed counters (tile_sync only)
  int a3d, b3d;                       // MN-major operand described by a 3-D map
  unsigned long long hint_a, hint_b;  // L2 eviction priority of the K-major tile loads
  unsigned wide;                      // this many tiles run whole, the halves of the others are items of their own (wide_grid)
  float alpha, beta;
};

// The work of a pair: `halves` accumulators of 256 columns from column n0 on, in row block tm.
struct WideItem {
  unsigned tm;
  int n0, halves;
};
// Items of the pairs.  C is cut into tiles of 256 x 512 and, where its 256-column tiles are odd in number, a last column of
// single halves.  Whole tiles first, a round of one per pair after the other; in the last, part-filled round the pairs that
// get no whole tile take up to two halves each, and what is left goes round singly.  The longest pair then has
// ceil(h / pairs) of the h halves of C, the same as if every half were an item of its own (wide_tiles_whole).
struct WideSchedule {
  unsigned tiles_m, tiles_w, wide, full_rounds, part, split, halves, pairs;
  int raster, last_n0;
  __host__ __device__ WideSchedule(int m, int n, unsigned wide_, int raster_, unsigned num_pairs) {
    const unsigned tiles_n = (n + 255u) / 256;
    tiles_m = (m + 255u) / 256;
    tiles_w = tiles_n / 2;
    wide = wide_;
    pairs = num_pairs;
    full_rounds = wide / pairs;
    part = wide % pairs;
    split = 2 * (tiles_m * tiles_w - wide);  // halves that come from cut tiles
    halves = split + (tiles_n & 1 ? tiles_m : 0);
    raster = raster_;
    last_n0 = static_cast<int>(tiles_n - 1) * 256;
  }
  __host__ __device__ WideItem tile(unsigned t) const {
    unsigned tm, tw;
    tile_coord_r(raster, tiles_m, tiles_w, t, tm, tw);
    return {tm, static_cast<int>(tw) * 512, 2};
  }
  // item j of pair `pair`; false when there is none any more
  __host__ __device__ bool item(unsigned pair, unsigned j, WideItem& w) const {
    if (j < full_rounds) {
      w = tile(j * pairs + pair);
      return true;
    }
    j -= full_rounds;
    unsigned h;
    if (part == 0) {
      h = j * pairs + pair;
    } else if (pair < part) {
      if (j == 0) {
        w = tile(full_rounds * pairs + pair);
        return true;
      }
      h = 2 * (pairs - part) + (j - 1) * pairs + pair;
    } else {
      h = j < 2 ? j * (pairs - part) + pair - part : 2 * (pairs - part) + (j - 2) * pairs + pair;
    }
    if (h >= halves) return false;
    if (h < split) {
      w = tile(wide + h / 2);
      w.n0 += static_cast<int>(h & 1) * 256;
      w.halves = 1;
    } else {
      w = {h - split, last_n0, 1};
    }
    return true;
  }
};
// How many of the whole tiles run whole.  Those of full rounds do.  Of the rest none if all that is left fits into one round of
// halves; only as many as the pairs need to get by with two halves each if few pairs need a second one (while the whole tile
// of a pair runs, the others have finished half of one and leave it the memory system: 1734 x 2723 x 4418 NT half, 77 halves on 74
// pairs, 61.6 -> 51.9 us, 7308 x 5888 x 4000 TN, 667 halves, 296 -> 287); else all (4096 x 4096 x 16384 NT, 256 halves: 428
// us, cut up like that 441: idle pairs draw no power).
inline unsigned wide_tiles_whole(long long tiles, long long single_halves, long long pairs) {
  const long long rest = tiles % pairs, left = 2 * rest + single_halves;
  if (left <= pairs) return static_cast<unsigned>(tiles - rest);
  if (4 * left <= 5 * pairs && left - pairs < rest) return static_cast<unsigned>(tiles - rest + left - pairs);
  return static_cast<unsigned>(tiles);
}
// What a launch for an m x n result on a GPU of `pairs` SM pairs needs: the tiles that run whole and the pairs that get work.
struct WideGrid {
  unsigned wide, pairs;
};
inline WideGrid wide_grid(int m, int n, long long pairs) {
  const long long tiles_m = (m + 255ll) / 256, tiles_n = (n + 255ll) / 256;
  const unsigned wide = wide_tiles_whole(tiles_m * (tiles_n / 2), tiles_n % 2 ? tiles_m : 0, pairs);
  const long long items = tiles_m * tiles_n - wide;
  return {wide, static_cast<unsigned>(items < pairs ? items : pairs)};
}

// MMAs of one K step (128 bytes of K): accumulator d0 over the first B tile, d1 over the second, or both with A kept in the
// collector buffer between the two.  kHalf: 0, 1 or 2 (both).  One elected lane.
template <class T, int kHalf>
__device__ __forceinline__ void wide_issue(uint32_t d0, uint32_t d1, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool first) {
  constexpr uint32_t adv = T::kMn ? T::kUmmaK * 128 : 32;
#pragma unroll
  for (int kk = 0; kk < T::kBK / T::kUmmaK; ++kk) {
    const uint32_t acc = (!first || kk > 0) ? 1u : 0u;
    const uint64_t a = a_desc + ((kk * adv) >> 4), b0 = b_desc + ((kk * adv) >> 4), b1 = b0 + (T::kBBytes >> 4);
    if constexpr (kHalf == 2) umma_ss_pair_keep_a<T::kFmt>(d0, d1, a, b0, b1, idesc, acc);
    else if constexpr (T::kFmt == kFmtF16) umma_f16_ss_pair(kHalf == 0 ? d0 : d1, a, kHalf == 0 ? b0 : b1, idesc, acc);
    else umma_tf32_ss_pair(kHalf == 0 ? d0 : d1, a, kHalf == 0 ? b0 : b1, idesc, acc);
  }
}

// The issuing warp's walk over the K steps of one item.  `it` counts ring slots, `unit` accumulators.
template <class T>
__device__ __forceinline__ bool wide_issue_item(int halves, int k_steps, uint32_t& it, uint32_t& unit, uint32_t tmem_base, uint64_t a_desc0, uint64_t b_desc0,
                                                uint32_t idesc, uint32_t full, uint32_t empty, uint32_t accfull, uint32_t accempty, const WaitCtx& ctx) {
  auto off = [](uint32_t i) { return static_cast<uint64_t>((i % T::kStages) * (T::kStageBytes >> 4)); };
  auto wait_full = [&](uint32_t i) { return mbar_wait_warp_spin(full + 8 * (i % T::kStages), (i / T::kStages) & 1, ctx, 3); };
  auto wait_acc = [&](uint32_t u) { return mbar_wait_warp_spin(accempty + 8 * (u & 1), ((u >> 1) & 1) ^ 1, ctx, 2); };
  const uint32_t a0 = unit & 1, d0 = tmem_base + a0 * T::kBN, d1 = tmem_base + (a0 ^ 1) * T::kBN;
  if (!wait_acc(unit)) return false;
  if (halves == 1) {
    for (int ks = 0; ks < k_steps; ++ks, ++it) {
      if (!wait_full(it)) return false;
      tc_fence_after();
      if (elect_one()) {
        wide_issue<T, 0>(d0, d1, a_desc0 + off(it), b_desc0 + off(it), idesc, ks == 0);
        umma_commit_pair(empty + 8 * (it % T::kStages), 3);
        if (ks + 1 == k_steps) umma_commit_pair(accfull + 8 * a0, 3);
      }
      __syncwarp();
    }
    unit += 1;
    return true;
  }
  // both ends: half 0 of kSkew steps, then half 1 of the same steps
  auto end_steps = [&](bool first) -> bool {
#pragma unroll
    for (int j = 0; j < T::kSkew; ++j) {
      if (!wait_full(it + j)) return false;
      tc_fence_after();
      if (elect_one()) {
        wide_issue<T, 0>(d0, d1, a_desc0 + off(it + j), b_desc0 + off(it + j), idesc, first && j == 0);
        if (!first && j + 1 == T::kSkew) umma_commit_pair(accfull + 8 * a0, 3);
      }
      __syncwarp();
    }
    if (first && !wait_acc(unit + 1)) return false;
    tc_fence_after();
    if (elect_one()) {
#pragma unroll
      for (int j = 0; j < T::kSkew; ++j) {
        wide_issue<T, 1>(d0, d1, a_desc0 + off(it + j), b_desc0 + off(it + j), idesc, first && j == 0);
        umma_commit_pair(empty + 8 * ((it + j) % T::kStages), 3);
        if (!first && j + 1 == T::kSkew) umma_commit_pair(accfull + 8 * (a0 ^ 1), 3);
      }
    }
    __syncwarp();
    it += T::kSkew;
    return true;
  };
  if (!end_steps(true)) return false;
  bool have_full = false;
  for (int ks = 2 * T::kSkew; ks < k_steps; ++ks, ++it) {
    if (!have_full && !wait_full(it)) return false;
    tc_fence_after();
    if (elect_one()) wide_issue<T, 2>(d0, d1, a_desc0 + off(it), b_desc0 + off(it), idesc, false);
    // is the next stage there already?  (never waits; the commit below waits for nothing either)
    have_full = mbar_test_warp(full + 8 * ((it + 1) % T::kStages), ((it + 1) / T::kStages) & 1);
    if (elect_one()) umma_commit_pair(empty + 8 * (it % T::kStages), 3);  // frees the stage in both CTAs
  }
  if (!end_steps(false)) return false;
  unit += 2;
  return true;
}

// One epilogue warp's 32 rows x 128 columns of an accumulator: into registers, `release` hands the accumulator back, then
// to column-major C (c: the lane's row, first column; `cols` of the columns exist, none if the row does not).  `whole`, the
// same for all lanes: every row and column exists and C is only written.
template <typename TOut, class Release>
__device__ __forceinline__ void wide_store(uint32_t t_row, TOut* c, long long ld, int cols, bool whole, float alpha, float beta, Release release) {
  constexpr int kChunks = 4;
  if (!whole) {  // straight from tensor memory; whole blocks of 32 columns in the fast loop, a tile's last rows and columns hold up
                 // the accumulator (us 2542 x 3175 x 2752 half 37.8 -> 34.0, 2388 x 2312 x 4032 53.8 -> 49.7, 256-column tiles 34.1 and 48.1)
#pragma unroll 1
    for (int i = 0; i < kChunks; ++i) {
      uint32_t v[32];
      tmem_ld_x32(t_row + i * 32, v);
      tmem_wait_ld();
      if (cols > 32 * i) store_columns<TOut>(v, c + 32ll * i * ld, ld, cols - 32 * i, alpha, beta, true);
    }
    __syncwarp();
    release();
    return;
  }
  if constexpr (sizeof(TOut) == 2) {
    uint32_t p[kChunks * 16];
#pragma unroll
    for (int i = 0; i < kChunks; i += 2) {
      uint32_t v0[32], v1[32];
      tmem_ld_x32(t_row + i * 32, v0);
      tmem_ld_x32(t_row + i * 32 + 32, v1);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const __half2 a = __floats2half2_rn(alpha * __uint_as_float(v0[2 * j]), alpha * __uint_as_float(v0[2 * j + 1]));
        const __half2 b = __floats2half2_rn(alpha * __uint_as_float(v1[2 * j]), alpha * __uint_as_float(v1[2 * j + 1]));
        p[i * 16 + j] = *reinterpret_cast<const uint32_t*>(&a);
        p[i * 16 + 16 + j] = *reinterpret_cast<const uint32_t*>(&b);
      }
    }
    release();
    TOut *d0 = c, *d1 = c + ld;
#pragma unroll
    for (int j = 0; j < kChunks * 16; ++j) {
      const __half2 h = *reinterpret_cast<const __half2*>(&p[j]);
      *d0 = __low2half(h);
      *d1 = __high2half(h);
      d0 += 2 * ld;
      d1 += 2 * ld;
    }
  } else {
    uint32_t v[kChunks][32];
#pragma unroll
    for (int i = 0; i < kChunks; ++i) tmem_ld_x32(t_row + i * 32, v[i]);
    tmem_wait_ld();
    release();
    TOut* d = c;
#pragma unroll
    for (int j = 0; j < kChunks * 32; ++j) {
      *d = alpha * __uint_as_float(v[j / 32][j % 32]);
      d += ld;
    }
  }
}

template <class T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(T::kThreads, 1)
gemm2w_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const Gemm2WArgs args) {
  using TOut = typename T::TOut;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t full = smem_base + T::kStages * T::kStageBytes, empty = full + 8 * T::kStages, accfull = empty + 8 * T::kStages, accempty = accfull + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_gen + T::kStages * T::kStageBytes + T::kNumBars * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx ctx{abort_flag, args.status, kWaitLimitNs};

  const int warp = warp_id_uniform(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader (issues the MMAs), 1 = peer
  const unsigned pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const WideSchedule sched(args.m, args.n, args.wide, args.raster, num_pairs);
  const int k_steps = (args.k + T::kBK - 1) / T::kBK;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < T::kStages; ++s) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(accfull + 8 * a, 1); mbar_init(accempty + 8 * a, 2 * 32 * T::kEpiWarps); }
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), T::kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the pair's barriers exist before anything arrives on them from the other CTA
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();  // nothing above touches memory that an earlier kernel of the stream may still be writing

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      WideItem w;
      for (unsigned j = 0; ok && sched.item(pair, j, w); ++j) {
        if (args.tile_sync && j > 0 && j < sched.full_rounds) {
          if (!(ok = tile_round_sync(args.rounds + rank, j * num_pairs, ctx, 5))) break;
        }
        const int m0 = w.tm * 2 * T::kBM + rank * T::kBM;  // this CTA's rows of A and C
        const int nb = w.n0 + rank * T::kBNHalf;           // this CTA's half of an accumulator's B tile
        const uint32_t bytes = 2u * (T::kABytes + w.halves * T::kBBytes);
        for (int ks = 0; ks < k_steps; ++ks, ++it) {
          const uint32_t s = it % T::kStages, bar = full + 8 * s;
          if (!(ok = mbar_wait(empty + 8 * s, ((it / T::kStages) & 1) ^ 1, ctx, 1))) break;
          if (rank == 0) mbar_expect_tx(bar, bytes);  // both CTAs' bytes land on this barrier
          const uint32_t a_dst = smem_base + s * T::kStageBytes, b_dst = a_dst + T::kABytes;
          const int k0 = ks * T::kBK;
          if constexpr (!T::kMn) {
            tma_load_2d_pair_hint(a_dst, &tmap_a, bar, k0, m0, args.hint_a);
            tma_load_2d_pair_hint(b_dst, &tmap_b, bar, k0, nb, args.hint_b);
            if (w.halves == 2) tma_load_2d_pair_hint(b_dst + T::kBBytes, &tmap_b, bar, k0, nb + T::kBN, args.hint_b);
          } else {
            if (args.a3d) {
              tma_load_3d_pair(a_dst, &tmap_a, bar, 0, k0, m0 / T::kChunk);
            } else {
#pragma unroll
              for (int c = 0; c < T::kBM / T::kChunk; ++c) tma_load_2d_pair(a_dst + c * (T::kBK * 128), &tmap_a, bar, m0 + c * T::kChunk, k0);
            }
            for (int hh = 0; hh < w.halves; ++hh) {
              const uint32_t dst = b_dst + hh * T::kBBytes;
              const int n0 = nb + hh * T::kBN;
              if (args.b3d) {
                tma_load_3d_pair(dst, &tmap_b, bar, 0, k0, n0 / T::kChunk);
              } else {
#pragma unroll
                for (int c = 0; c < T::kBNHalf / T::kChunk; ++c) tma_load_2d_pair(dst + c * (T::kBK * 128), &tmap_b, bar, n0 + c * T::kChunk, k0);
              }
            }
          }
        }
      }
      pdl_launch_dependents();  // all loads are on their way: the next kernel's launch may start under the last tile
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc(T::kFmt, T::kMn, T::kMn, 2 * T::kBM, T::kBN);
      constexpr uint32_t lbo = T::kMn ? T::kBK * 128 : 16, sbo = T::k32Atom ? 512 : 1024, type = T::k32Atom ? 1 : 2;
      const uint64_t a_desc0 = umma_desc_sw128(smem_base, lbo, sbo, type), b_desc0 = umma_desc_sw128(smem_base + T::kABytes, lbo, sbo, type);
      uint32_t it = 0, unit = 0;
      WideItem w;
      for (unsigned j = 0; sched.item(pair, j, w); ++j)
        if (!wide_issue_item<T>(w.halves, k_steps, it, unit, tmem_base, a_desc0, b_desc0, idesc, full, empty, accfull, accempty, ctx)) break;
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9, both CTAs)
    const int quad = warp & 3, cgroup = (warp - 2) >> 2;
    uint32_t unit = 0;
    bool ok = true;
    TOut* C = reinterpret_cast<TOut*>(args.C);
    WideItem w;
    for (unsigned j = 0; ok && sched.item(pair, j, w); ++j) {
      const int row = w.tm * 2 * T::kBM + rank * T::kBM + quad * 32 + lane;
      for (int hh = 0; hh < w.halves; ++hh, ++unit) {
        const uint32_t a = unit & 1;
        if (!(ok = mbar_wait_warp_spin(accfull + 8 * a, (unit >> 1) & 1, ctx, 4))) break;
        tc_fence_after();
        const int col0 = w.n0 + hh * T::kBN + cgroup * 128;
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + a * T::kBN + cgroup * 128;
        const bool whole = row - lane + 32 <= args.m && col0 + 128 <= args.n && args.beta == 0.f;
        wide_store<TOut>(t_row, C + row + static_cast<long long>(col0) * args.ldC, args.ldC, row < args.m ? args.n - col0 : 0, whole, args.alpha,
                         args.beta, [&]() {
                           tc_fence_before();
                           mbar_arrive_cluster(mapa_shared(accempty + 8 * a, 0));  // the leader's barrier collects both CTAs
                         });
      }
    }
  }

  // ---------------------------------------------------------------------- teardown
  wait_profile_flush(ctx);
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  tc_fence_before();
  cluster_sync_all();  // neither CTA frees tensor memory or exits while its pair may still use it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, T::kTmemCols);
  }
}

}  // namespace b200
