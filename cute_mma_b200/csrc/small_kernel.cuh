// Products that do not fill the GPU with 256 x 256 pair tiles: one CTA per 128 x (16..128) tile of C and per piece of K.
//
//   C(i, j) = alpha * sum_l P(i, l) * Q(j, l) + beta * C(i, j),  C(i, j) at C[i + j * ldC]
//
// P (the M side, 128 rows per tile) and Q (the N side) are the operands of the plain GEMM, or, for the OFT product
// Y^T = W . (X.R)^T, P = W and Q = X with every 64-column slice of Q rotated by R on its way to the tensor core (the
// same Y row-major).  The pair kernels give a problem with few tiles to few SMs (8 x 4096 x 4096: 32 of 148); here
//   * a tile covers 128 x n_tile of C, n_tile = 16..128 chosen for the problem (a decode step of 8 tokens multiplies
//     16 columns, not 256),
//   * the tiles are cut along K into `split` pieces (the CTAs of one cluster), so that every SM streams part of P;
//     the pieces' fp32 partial tiles meet in distributed shared memory, summed in piece order by the CTA that owns
//     the columns: no scratch in global memory, no counters, the same bits on every run,
//   * CTAs hold half of an SM's tensor memory and, where a ring of the least depth fits, half of its shared memory: plain
//     products always, rotated ones with tiles of at most 80 columns (48 with 64 x 64 blocks, never with 128 x 128).  Two
//     are resident then, and one's prologue and epilogue run under the other's main loop.
// Bound: small M reads P once from HBM (8 x 4096 x 4096: 33.5 MB); the rest is launch and pipeline latency.
//
// Roles (256 threads): warp 0 TMA producer, warp 1 issues the product, warp 2 owns tensor memory, warp 3 issues the
// rotation and warps 4..7 convert its slices (OFT only); all eight warps write C.  Rotation of slice j:
//   MMA1  XR [128 x 64] fp32 (TMEM) = X[128 x 64] . Rblk^T   (rows past n_tile are whatever shared memory holds: they
//         only ever reach rows of XR that nobody reads)
//   cvt   fp16 (RNE) into a K-major, 128-byte-swizzled tile in shared memory: the N-side operand of
//   MMA2  acc[128 x n_tile] += W[128 x 64] . XR^T
// MMA1 runs up to xbufs slices ahead of MMA2, so the conversion is off the tensor pipe's path.
#pragma once
#include <type_traits>

#include "gemm_kernel.cuh"

namespace b200 {

__device__ __forceinline__ float4 ld_dsmem_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

template <typename TIn_, typename TOut_, bool kMn_, int kB_>
struct SmallTraits {
  using TIn = TIn_;
  using TOut = TOut_;
  static constexpr bool kMn = kMn_;        // operands stored with M / N contiguous (NT), else K contiguous
  static constexpr int kB = kB_;           // block edge of the rotation of Q; 0: plain product
  static constexpr bool kRot = kB > 0;
  static constexpr int kElem = sizeof(TIn);
  static constexpr int kBM = 128;
  static constexpr int kMaxN = 128;
  static constexpr int kBK = 128 / kElem;
  static constexpr int kUmmaK = 32 / kElem;
  static constexpr int kChunk = 128 / kElem;
  static constexpr int kFmt = (kElem == 2) ? kFmtF16 : kFmtTF32;
  static constexpr bool k32Atom = kMn && kElem == 4;
  static constexpr int kPBytes = kBM * 128;
  static constexpr int kRBytes = kB * 128;
  static constexpr int kMaxStages = 12;
  static constexpr int kMaxXr = 3;
  static constexpr int kTmemCols = 256;    // accumulator (n_tile) and up to three 64-column rotation results
  static constexpr int kThreads = 256;
  static constexpr int kNumBars = 2 * kMaxStages + 3 * kMaxXr + 1;
  static constexpr int kTailBytes = kNumBars * 8 + 64;
  static_assert(!kRot || (!kMn && kElem == 2 && (kB == 16 || kB == 32 || kB == 64 || kB == 128)), "rotation: fp16, K contiguous, block edge 16 to 128");
};

struct SmallArgs {
  int m, n, k;             // rows of P, rows of Q, columns of both
  void* C;
  long long ldC;
  int* status;
  int n_tile;              // columns of C per tile: a multiple of 16 (of the 128-byte chunk for NT operands), <= 128
  int tiles_n;             // tiles along n; the tiles that share rows of P run side by side
  int split;               // pieces along K = cluster size
  int stages, xbufs;       // ring depth, rotation buffers
  int group_size;          // rows of P that share one R (rotation only)
  int p3d, q3d;            // NT operands described by a 3-D map (chunk, K, chunk index)
  int vec;                 // four rows of a column of C (and of further destinations) may be stored at once
  float alpha, beta;
};
// The same with further destinations of the result, laid out as C; they may be a peer's memory.  A type (and a kernel
// instance) of its own: with the loop over destinations in every launch 8 x 4096 x 4096 took 10.4 us instead of 10.1 and
// 647 x 4096 x 512 15.2 instead of 14.2.
struct SmallArgsMore : SmallArgs {
  int n_more;
  void* C_more[7];
};

template <class T, bool kMore = false>
__global__ void __launch_bounds__(T::kThreads, 2)
small_kernel(const __grid_constant__ CUtensorMap tmap_p, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_r,
             const std::conditional_t<kMore, SmallArgsMore, SmallArgs> args) {
  using TOut = typename T::TOut;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  // stage: [Q tile][R tile][P tile]; MMA1 reads 128 rows from the start of the Q tile, which stay inside the stage
  const uint32_t q_bytes = static_cast<uint32_t>(args.n_tile) * 128u;
  const uint32_t stage_bytes = q_bytes + T::kRBytes + T::kPBytes;
  const uint32_t xr_stage = smem_base + args.stages * stage_bytes;
  const uint32_t bars = xr_stage + (T::kRot ? args.xbufs * q_bytes : 0u);
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (T::kMaxStages + s); };
  auto x_acc = [&](int i) { return bars + 8u * (2 * T::kMaxStages + i); };
  auto x_ready = [&](int i) { return bars + 8u * (2 * T::kMaxStages + T::kMaxXr + i); };
  auto x_free = [&](int i) { return bars + 8u * (2 * T::kMaxStages + 2 * T::kMaxXr + i); };
  const uint32_t acc_full = bars + 8u * (T::kNumBars - 1);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_gen + (bars - smem_base) + T::kNumBars * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx ctx{abort_flag, args.status, kWaitLimitNs};

  const int warp = warp_id_uniform(), lane = threadIdx.x & 31;
  const int split = args.split;
  const unsigned piece = blockIdx.x % split, tile = blockIdx.x / split;  // piece = rank in the cluster
  const int tm = tile / args.tiles_n, tn = tile % args.tiles_n;
  const int m0 = tm * T::kBM, n0 = tn * args.n_tile;
  // pieces of whole K steps; 128 x 128 blocks span two steps, which stay together
  constexpr int kUnit = T::kB == 128 ? 2 : 1;
  const int units = (args.k + T::kBK * kUnit - 1) / (T::kBK * kUnit);
  const int ks0 = static_cast<int>(static_cast<long long>(units) * piece / split) * kUnit;
  const int steps = static_cast<int>(static_cast<long long>(units) * (piece + 1) / split) * kUnit - ks0;
  const int active_quads = (args.n_tile + 31) / 32;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < args.stages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), T::kB == 128 ? 2 : 1); }
    for (int i = 0; i < T::kMaxXr; ++i) { mbar_init(x_acc(i), 1); mbar_init(x_ready(i), 32 * active_quads); mbar_init(x_free(i), 1); }
    mbar_init(acc_full, 1);
    fence_mbar_init();
    fence_proxy_async_smem();
    prefetch_tmap(&tmap_p);
    prefetch_tmap(&tmap_q);
    if (T::kRot) prefetch_tmap(&tmap_r);
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(tmem_slot), T::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // From here on the next kernel of the stream may start its own prologue (every CTA of this launch is resident and
  // holds its tensor memory); nothing above touches memory that an earlier kernel may still be writing.
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    const int r_row = T::kRot ? (m0 / args.group_size) * T::kB : 0;
    int s = 0;
    uint32_t ph = 1;
    for (int i = 0; i < steps; ++i) {
      if (!mbar_wait_warp_spin(empty_bar(s), ph, ctx, 1)) break;
      const uint32_t q_dst = smem_base + s * stage_bytes, p_dst = q_dst + q_bytes + T::kRBytes;
      const int k0 = (ks0 + i) * T::kBK;
      if (elect_one()) {
        mbar_expect_tx(full_bar(s), stage_bytes);
        if constexpr (!T::kMn) {
          tma_load_2d(p_dst, &tmap_p, full_bar(s), k0, m0);
          tma_load_2d(q_dst, &tmap_q, full_bar(s), k0, n0);
          if constexpr (T::kRot) tma_load_2d(q_dst + q_bytes, &tmap_r, full_bar(s), k0, r_row);
        } else {
          if (args.p3d) {
            tma_load_3d(p_dst, &tmap_p, full_bar(s), 0, k0, m0 / T::kChunk);
          } else {
            for (int c = 0; c < T::kBM / T::kChunk; ++c) tma_load_2d(p_dst + c * (T::kBK * 128), &tmap_p, full_bar(s), m0 + c * T::kChunk, k0);
          }
          if (args.q3d) {
            tma_load_3d(q_dst, &tmap_q, full_bar(s), 0, k0, n0 / T::kChunk);
          } else {
            for (int c = 0; c < args.n_tile / T::kChunk; ++c) tma_load_2d(q_dst + c * (T::kBK * 128), &tmap_q, full_bar(s), n0 + c * T::kChunk, k0);
          }
        }
      }
      __syncwarp();
      if (++s == args.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ issuer of the product
    const uint32_t idesc = umma_idesc(T::kFmt, T::kMn, T::kMn, T::kBM, 16) + (static_cast<uint32_t>((args.n_tile - 16) >> 3) << 17);
    constexpr uint32_t adv = T::kMn ? T::kUmmaK * 128 : 32, lbo = T::kMn ? T::kBK * 128 : 16;
    constexpr uint32_t sbo = T::k32Atom ? 512 : 1024, type = T::k32Atom ? 1 : 2;
    const uint64_t p_desc0 = umma_desc_sw128(smem_base + q_bytes + T::kRBytes, lbo, sbo, type);
    // Q comes from the ring, or, rotated, from the tiles the converters fill
    const uint64_t q_desc0 = umma_desc_sw128(T::kRot ? xr_stage : smem_base, lbo, sbo, type);
    const uint32_t q_slot_bytes = T::kRot ? q_bytes : stage_bytes;
    const int q_slots = T::kRot ? args.xbufs : args.stages;
    int s = 0, x = 0;
    uint32_t ph = 0, ph_x = 0;
    for (int j = 0; j < steps; ++j) {
      if (T::kRot && !mbar_wait_warp_spin(x_ready(x), ph_x, ctx, 4)) break;
      if (!mbar_wait_warp_spin(full_bar(s), ph, ctx, 3)) break;
      tc_fence_after();
      const uint64_t p_desc = p_desc0 + ((s * stage_bytes) >> 4), q_desc = q_desc0 + ((x * q_slot_bytes) >> 4);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < T::kBK / T::kUmmaK; ++kk) {
          if constexpr (T::kFmt == kFmtF16) umma_f16_ss(tmem_base, p_desc + ((kk * adv) >> 4), q_desc + ((kk * adv) >> 4), idesc, (j > 0 || kk > 0) ? 1u : 0u);
          else umma_tf32_ss(tmem_base, p_desc + ((kk * adv) >> 4), q_desc + ((kk * adv) >> 4), idesc, (j > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(s));
        if constexpr (T::kRot) umma_commit(x_free(x));
        if (j + 1 == steps) umma_commit(acc_full);
      }
      __syncwarp();
      if (++s == args.stages) { s = 0; ph ^= 1; }
      if (++x == q_slots) { x = 0; ph_x ^= 1; }
    }
  } else if (T::kRot && warp == 3) {
    // ------------------------------------------------------------------ issuer of the rotation
    constexpr uint32_t idesc1 = umma_idesc(kFmtF16, 0, 0, T::kBM, T::kB == 0 ? 16 : (T::kB > 64 ? 64 : T::kB));
    const uint64_t x_desc0 = umma_desc_sw128(smem_base, 16, 1024), r_desc0 = umma_desc_sw128(smem_base + q_bytes, 16, 1024);
    int s = 0, x = 0, prev = 0;
    uint32_t ph = 0, ph_x = 0;
    for (int j = 0; j < steps; ++j) {
      // the converters have read the buffer's last result (their x_ready of slice j - xbufs)
      if (j >= args.xbufs && !mbar_wait_warp_spin(x_ready(x), ph_x ^ 1, ctx, 8)) break;
      if (T::kB != 128 || (j & 1) == 0) {
        if (!mbar_wait_warp_spin(full_bar(s), ph, ctx, 9)) break;
      }
      const uint32_t d = tmem_base + args.n_tile + x * 64;
      if constexpr (T::kB == 128) {
        // a block spans two steps and gives two slices: slice h = j & 1 is X's two steps times rows [64 h, 64 h + 64) of R
        const int next = s + 1 == args.stages ? 0 : s + 1;
        if ((j & 1) == 0 && !mbar_wait_warp_spin(full_bar(next), next == 0 ? ph ^ 1 : ph, ctx, 9)) break;
        tc_fence_after();
        const int h = j & 1, s_even = h ? prev : s, s_odd = h ? s : next;
        if (elect_one()) {
#pragma unroll
          for (int su = 0; su < 2; ++su) {
            const uint64_t off = ((su ? s_odd : s_even) * stage_bytes) >> 4;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_f16_ss(d, x_desc0 + off + kk * 2, r_desc0 + off + ((h * 64 * 128) >> 4) + kk * 2, idesc1, (su > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(x_acc(x));
          if (h) {  // both slices of the block have read both stages
            umma_commit(empty_bar(s_even));
            umma_commit(empty_bar(s_odd));
          }
        }
      } else {
        tc_fence_after();
        const uint64_t off = (s * stage_bytes) >> 4;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {  // slice kk of the step belongs to block (16 kk) / b: columns [blk b, blk b + b) of XR
            constexpr int b = T::kB == 0 ? 16 : T::kB;
            umma_f16_ss(d + (kk * 16) / b * b, x_desc0 + off + kk * 2, r_desc0 + off + kk * 2, idesc1, ((kk * 16) % b) != 0 ? 1u : 0u);
          }
          umma_commit(x_acc(x));
        }
      }
      __syncwarp();
      prev = s;
      if (++s == args.stages) { s = 0; ph ^= 1; }
      if (++x == args.xbufs) { x = 0; ph_x ^= 1; }
    }
  } else if (T::kRot && warp >= 4 && warp - 4 < active_quads) {
    // ------------------------------------------------------------------ rotated slice: fp32 (TMEM) -> fp16 tile (shared memory)
    const int quad = warp & 3, r = quad * 32 + lane;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + args.n_tile;
    int x = 0;
    uint32_t ph = 0;
    for (int j = 0; j < steps; ++j) {
      if (!mbar_wait_warp_spin(x_acc(x), ph, ctx, 5)) break;
      tc_fence_after();
      uint32_t v0[32], v1[32];
      tmem_ld_x32(t_row + x * 64, v0);
      tmem_ld_x32(t_row + x * 64 + 32, v1);
      tmem_wait_ld();
      uint32_t p[32];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const __half2 a = __floats2half2_rn(__uint_as_float(v0[2 * i]), __uint_as_float(v0[2 * i + 1]));
        const __half2 b = __floats2half2_rn(__uint_as_float(v1[2 * i]), __uint_as_float(v1[2 * i + 1]));
        p[i] = *reinterpret_cast<const uint32_t*>(&a);
        p[16 + i] = *reinterpret_cast<const uint32_t*>(&b);
      }
      if (!mbar_wait_warp_spin(x_free(x), ph ^ 1, ctx, 6)) break;  // the product of slice j - xbufs has read the tile
      const uint32_t row = xr_stage + x * q_bytes + r * 128;
      if (r < args.n_tile) {
#pragma unroll
        for (int c = 0; c < 8; ++c) st_shared_v4(row + ((c ^ (r & 7)) << 4), p[4 * c], p[4 * c + 1], p[4 * c + 2], p[4 * c + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(x_ready(x));
      if (++x == args.xbufs) { x = 0; ph ^= 1; }
    }
    __syncwarp();
  }

  // ---------------------------------------------------------------------- C (all warps)
  TOut* C = reinterpret_cast<TOut*>(args.C);
  const bool scaled = args.alpha != 1.f || args.beta != 0.f;
  const int cols = args.n - n0 < args.n_tile ? args.n - n0 : args.n_tile;
  int more = 0;  // destinations beside C
  if constexpr (kMore) more = args.n_more;
  auto dst_of = [&](int d) {
    if constexpr (kMore) return d == 0 ? C : static_cast<TOut*>(args.C_more[d - 1]);
    else return C;
  };
  auto store = [&](float f, TOut* dst) {
    if (scaled) {
      f *= args.alpha;
      if (args.beta != 0.f) f += args.beta * static_cast<float>(*dst);
    }
    if constexpr (sizeof(TOut) == 2) *dst = __float2half_rn(f);
    else *dst = f;
  };
  {
    const bool ok = mbar_wait_warp_spin(acc_full, 0, ctx, 7);
    tc_fence_after();
    const int quad = warp & 3, r = quad * 32 + lane;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    for (int d = 0; ok && d <= (split > 1 ? 0 : more); ++d) {  // tensor memory is read again for each destination: kept values cost 38 registers
      TOut* base = dst_of(d);
      for (int c = (warp >> 2) * 32; c < cols; c += 64) {
        uint32_t v[32];
        tmem_ld_x32(t_row + c, v);
        tmem_wait_ld();
        if (split > 1) {  // park the partial tile: [column][128 rows] over the ring, whose stages have all been read
          const uint32_t dst = smem_base + (c * 128 + r) * 4;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c + j < cols) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + j * 512), "r"(v[j]) : "memory");
        } else if (m0 + r < args.m) {
          store_columns<TOut>(v, base + (m0 + r) + static_cast<long long>(n0 + c) * args.ldC, args.ldC, cols - c, args.alpha, args.beta, true);
        }
      }
    }
  }
  tc_fence_before();
  if (split > 1) {
    cluster_sync_all();
    // this CTA adds up its share of the columns over all pieces, in piece order
    const int c0 = cols * static_cast<int>(piece) / split, c1 = cols * (static_cast<int>(piece) + 1) / split;
    const int row = m0 + 4 * lane;
    for (int c = c0 + warp; c < c1; c += T::kThreads / 32) {
      const uint32_t src = smem_base + (c * 128 + 4 * lane) * 4;
      float4 x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = q < split ? ld_dsmem_f4(mapa_shared(src, q)) : make_float4(0.f, 0.f, 0.f, 0.f);
      float o[4] = {x[0].x, x[0].y, x[0].z, x[0].w};
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < split) { o[0] += x[q].x; o[1] += x[q].y; o[2] += x[q].z; o[3] += x[q].w; }
      const long long at = row + static_cast<long long>(n0 + c) * args.ldC;
      for (int d = 0; d <= more; ++d) {
        TOut* dst = dst_of(d) + at;
        if (args.vec && !scaled && row + 4 <= args.m) {
          if constexpr (sizeof(TOut) == 2) {
            const __half2 a = __floats2half2_rn(o[0], o[1]), b = __floats2half2_rn(o[2], o[3]);
            *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
          } else {
            *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (row + e < args.m) store(o[e], dst + e);
        }
      }
    }
    cluster_sync_all();  // nobody leaves while another CTA may still read its partial tile
  } else {
    __syncthreads();
  }

  // ---------------------------------------------------------------------- teardown
  if (*abort_flag) {  // a wait ran out: let the copies in flight land before shared and tensor memory go away
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, T::kTmemCols);
  }
}

}  // namespace b200
