// W4A16 projection  y[M,N] = half(x[M,K] W^T + bias),  W[n][k] = half((code - 8) * scale[n][k/g]).
//
// Weights arrive in the interchange format unchanged: uint8 [N, ceil(K/2)], low nibble = even k.
// A 16-byte load therefore carries 32 consecutive-k codes of one output column, and because every
// legal group size is a multiple of 32 those codes share one scale.  Codes are unpacked in
// registers with the FP16 "magic number" trick (or-ing a nibble into the mantissa of 1024.0 gives
// 1024 + code exactly), turned into code - 8 exactly, and multiplied by the FP16 scale with one
// FP16 rounding -- bit-identical to the format's definition half(float(q) * float(scale)), since
// that FP32 product is exact.  Products with x accumulate in FP32.
//
// Compute paths (they share the unpack; the dispatcher at the end of the file picks one):
//   * small M, K % 1024 == 0: mma.m16n8k16 with the operands swapped -- 16 weight columns are the MMA's rows, the rows of
//     x its columns -- fed from direct 16-byte loads (w4a16_mma_kernel).
//   * M >= 9 on widths that suit its strips (and any M with a strided or multi-rank output), K % 256 == 0, group >= 64:
//     tcgen05 kind::f16 with the dequantised weights in tensor memory (w4a16_umma_kernel).
//   * the other M >= 3, K % 128 == 0: the same MMAs with x kept in registers and K shared by the warps of a CTA or the
//     CTAs of a cluster (w4a16_rx_kernel).
//   * the rest: a TMA-fed mma.sync stream kernel (short K of M >= 9, K > 32768), a SIMT kernel (lanes stride over the packed row,
//     mixed-precision FMAs, warp shuffle per column) and a generic kernel for any K.
// The k order inside an MMA fragment is free as long as both operands use the same order, so x is stored in shared
// memory pre-permuted to the order the unpack produces and no weight ever moves between lanes.
#include <cooperative_groups.h>
#include <stdlib.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "umma.cuh"

namespace cg = cooperative_groups;

namespace xdk {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

struct W4Args {
  const __half* x;
  const uint8_t* packed;
  const __half* scales;
  const __half* bias;
  __half* y;
  PeerOut out;        // where y goes for the tcgen05 kernel: y itself, or the same place in every rank's buffer
  int m, k, n;
  int group, groups;  // group size and scales per row
  int col_groups, groups_per_cta;
};

// Eight codes of one 32-bit word -> four half2 of dequantised weights, ordered
// (k0,k4) (k1,k5) (k2,k6) (k3,k7) relative to the word's first k.
__device__ __forceinline__ void dequant8(uint32_t word, __half2 scale2, __half2 (&w)[4]) {
  constexpr uint32_t kMagic = 0x64006400u;  // half2(1024, 1024)
  const uint32_t hi = word >> 8;
  uint32_t t0, t1, t2, t3;
  asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xea;" : "=r"(t0) : "r"(word), "r"(kMagic));  // (a & b) | c
  asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xea;" : "=r"(t1) : "r"(word), "r"(kMagic));
  asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xea;" : "=r"(t2) : "r"(hi), "r"(kMagic));
  asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xea;" : "=r"(t3) : "r"(hi), "r"(kMagic));
  const __half2 k1032 = __floats2half2_rn(1032.0f, 1032.0f);
  const __half2 k16th = __floats2half2_rn(0.0625f, 0.0625f);
  const __half2 km72 = __floats2half2_rn(-72.0f, -72.0f);
  // low nibbles: (1024 + c) - 1032 = c - 8;  high nibbles: (1024 + 16 c) / 16 - 72 = c - 8; both exact
  const __half2 q0 = __hsub2(*reinterpret_cast<__half2*>(&t0), k1032);
  const __half2 q1 = __hfma2(*reinterpret_cast<__half2*>(&t1), k16th, km72);
  const __half2 q2 = __hsub2(*reinterpret_cast<__half2*>(&t2), k1032);
  const __half2 q3 = __hfma2(*reinterpret_cast<__half2*>(&t3), k16th, km72);
  w[0] = __hmul2(q0, scale2);
  w[1] = __hmul2(q1, scale2);
  w[2] = __hmul2(q2, scale2);
  w[3] = __hmul2(q3, scale2);
}

// acc += a * b with FP16 operands and an FP32 accumulator in one instruction (sm_100 mixed FMA).
__device__ __forceinline__ void fma_h(float& acc, __half a, __half b) {
  asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc) : "h"(__half_as_ushort(a)), "h"(__half_as_ushort(b)));
}

// 16-byte units of x are XOR-swizzled in shared memory so that lanes reading consecutive
// 64-byte spans (32 halves each) hit distinct banks.
__device__ __forceinline__ int swz(int unit) { return unit ^ ((unit >> 3) & 3); }

// Fast SIMT path: K % 32 == 0, 16-byte aligned rows.  A warp owns CW columns at a time and lanes
// stride over the 16-byte vectors of the packed rows; x (all M rows, whole K) sits in shared memory.
template <int MT, int CW>
__global__ void __launch_bounds__(kThreads)
w4a16_simt_kernel(W4Args a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  U4* xs = reinterpret_cast<U4*>(smem_raw);  // [MT][K/8] swizzled 16-byte units
  const int units = a.k / 8;
  for (int i = threadIdx.x; i < MT * units; i += kThreads) {
    const int r = i / units, u = i - r * units;
    U4 v = U4{0u, 0u, 0u, 0u};
    if (r < a.m) v = ld_cached16(a.x + static_cast<size_t>(r) * a.k + u * 8);
    xs[r * units + swz(u)] = v;
  }
  __syncthreads();

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int vecs = a.k / 32;         // 16-byte vectors per packed row
  const int row_bytes = a.k / 2;
  for (int gi = 0; gi < a.groups_per_cta; ++gi) {
    const int cg = blockIdx.x * a.groups_per_cta + gi;
    if (cg >= a.col_groups) break;
    const int col0 = (cg * kWarps + warp) * CW;
    float acc[MT][CW];
#pragma unroll
    for (int r = 0; r < MT; ++r)
#pragma unroll
      for (int c = 0; c < CW; ++c) acc[r][c] = 0.0f;

    for (int v0 = 0; v0 < vecs; v0 += 32 * 2) {
      U4 wv[2][CW];
      __half sc[2][CW];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int v = v0 + u * 32 + lane;
#pragma unroll
        for (int c = 0; c < CW; ++c) {
          const bool ok = v < vecs && col0 + c < a.n;
          wv[u][c] = U4{0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u};  // code 8 == weight 0
          sc[u][c] = __float2half(0.0f);
          if (ok) {
            wv[u][c] = ld_stream16(a.packed + static_cast<size_t>(col0 + c) * row_bytes + v * 16);
            sc[u][c] = __ldg(a.scales + static_cast<size_t>(col0 + c) * a.groups + (v * 32) / a.group);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int v = v0 + u * 32 + lane;
        if (v0 + u * 32 < vecs) {
          const int vv = v < vecs ? v : 0;  // out-of-range lanes multiply zeros by valid x
#pragma unroll
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // the four 32-bit words of the vector, 8 k each
            __half2 w[CW][4];
#pragma unroll
            for (int c = 0; c < CW; ++c) {
              const uint32_t word = j == 0 ? wv[u][c].x : (j == 1 ? wv[u][c].y : (j == 2 ? wv[u][c].z : wv[u][c].w));
              dequant8(word, __half2half2(sc[u][c]), w[c]);
            }
#pragma unroll
            for (int r = 0; r < MT; ++r) {
              const U4 xv = xs[r * units + swz(vv * 4 + j)];
              const __half* xh = reinterpret_cast<const __half*>(&xv);
#pragma unroll
              for (int c = 0; c < CW; ++c) {
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                  fma_h(acc[r][c], __low2half(w[c][p]), xh[p]);
                  fma_h(acc[r][c], __high2half(w[c][p]), xh[p + 4]);
                }
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < MT; ++r)
#pragma unroll
      for (int c = 0; c < CW; ++c) {
        const float total = warp_sum(acc[r][c]);
        if (lane == 0 && r < a.m && col0 + c < a.n) {
          const float b = a.bias ? __half2float(a.bias[col0 + c]) : 0.0f;
          a.y[static_cast<size_t>(r) * a.n + col0 + c] = __float2half_rn(total + b);
        }
      }
  }
}

// ------------------------------------------------------------------------------------------------
// Tensor-core building blocks.  A warp works on blocks of 8 columns in steps of 128 k: in a step
// lane (g = lane/4, j = lane%4) holds the 16 bytes with k in [32j, 32j+32) of column g of the block.
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Physical position of 16-byte unit `unit` of x row `row`: the XOR spreads the eight units a
// quarter-warp reads in one shared-memory phase (2 rows x 4 lanes) over all eight bank groups.
__device__ __forceinline__ int xunit(int unit, int row) { return unit ^ ((((unit >> 3) & 1) << 1) | (row & 1)); }

// ------------------------------------------------------------------------------------------------
// Streaming tensor-core path (M >= 3, K % 128 == 0: a short K of M >= 9, and K too long for the paths below).
//
// One persistent CTA per SM.  The N/8 column blocks are dealt out evenly to clusters of S CTAs
// (S = split-K factor, 1/2/4); inside a cluster CTA r takes the K chunks r, r+S, ... of 1024 k, and
// inside a CTA warp w takes blocks w, w+8, ...  A (chunk, block) tile is 8 column rows of 512 packed
// bytes plus their scales.  Every warp runs its own software pipeline: an elected lane keeps the TMA
// box copies (one op for the weights, one for the scales) of the warp's next three tiles in flight
// into a private four-slot shared-memory ring, completing on per-slot mbarriers, while the warp
// unpacks the current tile in registers and feeds mma.m16n8k16.  (A warp can only keep a handful
// of ordinary load instructions in flight; one TMA op moves a whole 4 KB tile.)  x for the current chunk sits in shared memory, pre-permuted and swizzled
// as in the path above and double-buffered across chunks.  Partial sums of the S CTAs meet through
// distributed shared memory in rank order.
constexpr int kStreamWarps = 8;
constexpr int kStreamThreads = kStreamWarps * 32;
constexpr int kChunkK = 1024;                       // k per chunk
constexpr int kRowStride = kChunkK / 2;             // a tile is a dense TMA box: 8 column rows x 512 B
constexpr int kSlotBytes = 8 * kRowStride + 512;    // + up to 8 x 64 B of scales (dense box, 8 rows)
// ring slots per warp: all but one hold tiles in flight; 16 staged x rows leave room for 3, 8 rows for 4
// MR = rows of x staged per chunk (8 for M <= 8, else 16)
template <int MR> struct StreamDepth { static constexpr int value = MR == 16 ? 3 : 4; };
constexpr int kMaxNB = 8;                           // column blocks per warp per pass

__device__ unsigned int g_w4_fault;  // set when a bounded wait gives up

struct StreamPlan {
  int clusters;        // number of clusters (grid = clusters * splits)
  int splits;          // CTAs per cluster = split-K factor
  int total_blocks;    // ceil(N / 8)
  int chunks;          // ceil(K / 1024)
  int ring_scales;     // 1: the chunk's scales travel through the ring with the weights
};

template <int MR>
__global__ void __launch_bounds__(kStreamThreads, 1)
w4a16_stream_kernel(W4Args a, StreamPlan plan, const __grid_constant__ CUtensorMap wmap,
                    const __grid_constant__ CUtensorMap smap) {
  constexpr bool ROWS16 = MR == 16;
  constexpr int kRows = MR;
  constexpr int kXUnits = kChunkK / 8;  // 16-byte units per staged x row
  constexpr int kPassBlocks = kStreamWarps * kMaxNB;
  constexpr int kDepth = StreamDepth<MR>::value;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, j = lane & 3;
  unsigned char* ring = smem_raw + warp * kDepth * kSlotBytes;                          // this warp's slots
  U4* xs = reinterpret_cast<U4*>(smem_raw + kStreamWarps * kDepth * kSlotBytes);       // [2][kRows][kXUnits]
  float* part = reinterpret_cast<float*>(smem_raw + kStreamWarps * kDepth * kSlotBytes + 2 * kRows * kChunkK * 2);
  uint64_t* full = reinterpret_cast<uint64_t*>(part + 16 * kStreamWarps * kMaxNB * 8) + warp * kDepth;  // this warp's barriers
  if (lane == 0) {
    for (int i = 0; i < kDepth; ++i) mbar_init(full + i, 1);
    mbar_fence_init();
  }
  __syncwarp();

  const int rank = plan.splits > 1 ? static_cast<int>(cg::this_cluster().block_rank()) : 0;
  const int cluster_id = blockIdx.x / plan.splits;
  // even deal of column blocks to clusters
  const int blk_begin = static_cast<int>(static_cast<int64_t>(cluster_id) * plan.total_blocks / plan.clusters);
  const int blk_end = static_cast<int>(static_cast<int64_t>(cluster_id + 1) * plan.total_blocks / plan.clusters);
  const int nblk = blk_end - blk_begin;
  const int my_chunks = plan.chunks > rank ? (plan.chunks - rank + plan.splits - 1) / plan.splits : 0;
  const int row_bytes = a.k / 2;
  const int scale_shift = 31 - __clz(a.group);  // group is a power of two

  // ---- prefetch side: walks the same (pass, chunk, block) sequence as the compute loop, ahead of it
  int pf_p0 = 0, pf_ci = 0, pf_b = warp, pf_q = 0;
  bool pf_valid = my_chunks > 0 && nblk > 0;
  auto pf_normalize = [&]() {
    while (pf_valid && pf_b >= min(kPassBlocks, nblk - pf_p0)) {
      pf_b = warp;
      if (++pf_ci >= my_chunks) {
        pf_ci = 0;
        pf_p0 += kPassBlocks;
        if (pf_p0 >= nblk) pf_valid = false;
      }
    }
  };
  const unsigned tile_bytes = 8 * kRowStride + (plan.ring_scales ? 8u * ((kChunkK >> scale_shift) * 2) : 0u);
  auto pf_issue = [&]() {  // TMA ops for the next tile of this warp (if any) into slot pf_q % kDepth
    pf_normalize();
    if (pf_valid) {
      if (lane == 0) {
        const int kc = rank + pf_ci * plan.splits;
        const int col0 = (blk_begin + pf_p0 + pf_b) * 8;
        unsigned char* dst = ring + (pf_q % kDepth) * kSlotBytes;
        uint64_t* bar = full + pf_q % kDepth;
        mbar_expect_tx(bar, tile_bytes);  // out-of-range parts of a box are zero-filled and still counted
        tma_box_2d(dst, &wmap, kc * (kChunkK / 8), col0, bar);
        if (plan.ring_scales) tma_box_2d(dst + 8 * kRowStride, &smap, kc * (kChunkK >> scale_shift), col0, bar);
      }
      pf_b += kStreamWarps;
      ++pf_q;
    }
  };
#pragma unroll
  for (int d = 0; d < kDepth - 1; ++d) pf_issue();

  int q = 0;  // tiles this warp has consumed
  for (int p0 = 0; p0 < nblk; p0 += kPassBlocks) {
    const int nb_pass = min(kPassBlocks, nblk - p0);
    const int cols = nb_pass * 8;  // width of part[16][cols] for this pass

    // x staging.  A thread owns kStage 16-byte units of every chunk.  The first chunk of a pass is
    // staged at once; the next chunk is staged two units at a time around the tiles of the current
    // one (loads issued before a tile, permuted and stored after it) so that only two units are
    // ever live in registers during the unpack/mma loop.
    constexpr int kStage = (kRows * kXUnits + kStreamThreads - 1) / kStreamThreads;  // units per thread per chunk
    auto x_load = [&](int kc, int i) -> U4 {
      const int idx = threadIdx.x + i * kStreamThreads;
      const int r = idx / kXUnits, u = idx - r * kXUnits;
      const int k0 = kc * kChunkK + u * 8;
      U4 v = U4{0u, 0u, 0u, 0u};
      if (idx < kRows * kXUnits && r < a.m && k0 < a.k) v = ld_cached16(a.x + static_cast<size_t>(r) * a.k + k0);
      return v;
    };
    auto x_store = [&](int buf, int i, const U4& t) {
      const int idx = threadIdx.x + i * kStreamThreads;
      if (idx >= kRows * kXUnits) return;
      const int r = idx / kXUnits, u = idx - r * kXUnits;
      U4 v;  // the unpack's k order (0,4,1,5,2,6,3,7) inside every 8-block
      v.x = __byte_perm(t.x, t.z, 0x5410);
      v.y = __byte_perm(t.x, t.z, 0x7632);
      v.z = __byte_perm(t.y, t.w, 0x5410);
      v.w = __byte_perm(t.y, t.w, 0x7632);
      xs[(buf * kRows + r) * kXUnits + xunit(u, r)] = v;
    };
    if (my_chunks > 0) {
      U4 first[kStage];
#pragma unroll
      for (int i = 0; i < kStage; ++i) first[i] = x_load(rank, i);
#pragma unroll
      for (int i = 0; i < kStage; ++i) x_store(0, i, first[i]);
    }
    __syncthreads();

    for (int ci = 0; ci < my_chunks; ++ci) {
      const int kc = rank + ci * plan.splits;
      const int steps = min(kChunkK, a.k - kc * kChunkK) / 128;
      const bool more = ci + 1 < my_chunks;
      const bool last = !more;
      int staged = more ? 0 : kStage;  // units of the next chunk this thread has staged so far
      const U4* xb = xs + (ci & 1) * kRows * kXUnits;
      for (int b = warp; b < nb_pass; b += kStreamWarps, ++q) {
        const bool stage_now = staged < kStage;
        U4 nx0 = U4{0u, 0u, 0u, 0u}, nx1 = U4{0u, 0u, 0u, 0u};
        if (stage_now) {
          nx0 = x_load(kc + plan.splits, staged);
          nx1 = x_load(kc + plan.splits, staged + 1);
        }
        {
          const int col = (blk_begin + p0 + b) * 8 + g;
          // Slow path only (scales not in the ring): this lane's scale for every step, fetched before the wait
          __half sc[8];
          if (!plan.ring_scales) {
  #pragma unroll
            for (int st = 0; st < 8; ++st) {
              sc[st] = __float2half(0.0f);
              if (st < steps && col < a.n)
                sc[st] = __ldg(a.scales + static_cast<size_t>(col) * a.groups + ((kc * kChunkK + st * 128 + j * 32) >> scale_shift));
            }
          }
          pf_issue();  // refill the slot freed by the previous tile
          const bool landed = mbar_wait(full + q % kDepth, (q / kDepth) & 1);
          const unsigned char* slot = ring + (q % kDepth) * kSlotBytes;
          const unsigned char* tile = slot + g * kRowStride + j * 16;
          const __half* tile_scales =
              reinterpret_cast<const __half*>(slot + 8 * kRowStride + g * ((kChunkK >> scale_shift) * 2));
          if (!landed) atomicOr(&g_w4_fault, 1u);
          float part4[8][4];  // eight independent accumulator chains hide the mma latency
  #pragma unroll
          for (int w = 0; w < 8; ++w)
  #pragma unroll
            for (int e = 0; e < 4; ++e) part4[w][e] = 0.0f;
  #pragma unroll
          for (int st = 0; st < 8; ++st) {
            if (st >= steps || !landed) break;
            U4 wv = U4{0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u};
            __half s1 = __float2half(0.0f);
            if (col < a.n) {
              wv = *reinterpret_cast<const U4*>(tile + st * 64);
              s1 = plan.ring_scales ? tile_scales[(st * 128 + j * 32) >> scale_shift] : sc[st];
            }
            const __half2 s2 = __half2half2(s1);
  #pragma unroll
            for (int w = 0; w < 4; ++w) {
              const int unit = st * 16 + j * 4 + w;
              const U4 xa = xb[g * kXUnits + xunit(unit, g)];
              U4 xc = U4{0u, 0u, 0u, 0u};
              if constexpr (ROWS16) xc = xb[(g + 8) * kXUnits + xunit(unit, g + 8)];
              const uint32_t word = w == 0 ? wv.x : (w == 1 ? wv.y : (w == 2 ? wv.z : wv.w));
              __half2 h[4];
              dequant8(word, s2, h);
              mma16816(part4[2 * w], xa.x, xc.x, xa.y, xc.y, *reinterpret_cast<uint32_t*>(&h[0]),
                       *reinterpret_cast<uint32_t*>(&h[1]));
              mma16816(part4[2 * w + 1], xa.z, xc.z, xa.w, xc.w, *reinterpret_cast<uint32_t*>(&h[2]),
                       *reinterpret_cast<uint32_t*>(&h[3]));
            }
          }
          __syncwarp();  // every lane is done reading the slot before the next pf_issue overwrites it

          // C[row g][2j], C[g][2j+1], C[g+8][2j], C[g+8][2j+1] of this block for this chunk
          float c4[4];
  #pragma unroll
          for (int e = 0; e < 4; ++e)
            c4[e] = ((part4[0][e] + part4[1][e]) + (part4[2][e] + part4[3][e])) + ((part4[4][e] + part4[5][e]) + (part4[6][e] + part4[7][e]));
          float* mine = part + g * cols + b * 8 + 2 * j;  // rows g and g+8 of part[16][cols]; only this lane touches them
          if (ci > 0) {
            c4[0] += mine[0], c4[1] += mine[1];
            c4[2] += mine[8 * cols], c4[3] += mine[8 * cols + 1];
          }
          if (last && plan.splits == 1) {
  #pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int row = g + (e >> 1) * 8, oc = (blk_begin + p0 + b) * 8 + 2 * j + (e & 1);
              if (row < a.m && oc < a.n) {
                const float bv = a.bias ? __half2float(a.bias[oc]) : 0.0f;
                a.y[static_cast<size_t>(row) * a.n + oc] = __float2half_rn(c4[e] + bv);
              }
            }
          } else {
            mine[0] = c4[0], mine[1] = c4[1];
            mine[8 * cols] = c4[2], mine[8 * cols + 1] = c4[3];
          }
        }
        if (stage_now) {
          x_store((ci + 1) & 1, staged, nx0);
          x_store((ci + 1) & 1, staged + 1, nx1);
          staged += 2;
        }
      }
      for (; staged < kStage; ++staged) x_store((ci + 1) & 1, staged, x_load(kc + plan.splits, staged));
      __syncthreads();
    }
  }
  if (plan.splits > 1) {
    // The host guarantees a single pass when K is split, so part[16][nblk * 8] is complete here.
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int cols = nblk * 8;
    const int total = 16 * cols;
    const int share = (total + plan.splits - 1) / plan.splits;
    for (int i = threadIdx.x; i < share; i += kStreamThreads) {
      const int o = rank * share + i;
      if (o < total) {
        const int row = o / cols, c = o - row * cols;
        const int col = blk_begin * 8 + c;
        float v = 0.0f;
        for (int sidx = 0; sidx < plan.splits; ++sidx) v += *cluster.map_shared_rank(part + o, sidx);
        if (row < a.m && col < a.n) {
          const float bv = a.bias ? __half2float(a.bias[col]) : 0.0f;
          a.y[static_cast<size_t>(row) * a.n + col] = __float2half_rn(v + bv);
        }
      }
    }
    cluster.sync();
  }
}

template <int MR>
int launch_stream(const W4Args& a, cudaStream_t stream) {
  const int sms = xdk::sm_count();
  StreamPlan plan;
  plan.total_blocks = (a.n + 7) / 8;
  plan.chunks = (a.k + kChunkK - 1) / kChunkK;
  plan.ring_scales = (a.group <= 128 && a.k % kChunkK == 0 && aligned16(a.scales)) ? 1 : 0;
  constexpr int kDepth = StreamDepth<MR>::value;
  const size_t smem = static_cast<size_t>(kStreamWarps) * kDepth * kSlotBytes + 2 * MR * kChunkK * 2 +
                      16 * kStreamWarps * kMaxNB * 8 * sizeof(float) + kStreamWarps * kDepth * sizeof(uint64_t);
  CUtensorMap wmap, smap;
  {
    // packed weights as a [N][K/8] matrix of 32-bit words; box = 8 rows x 128 words (1024 k)
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(a.k / 8), static_cast<cuuint64_t>(a.n)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(a.k / 2)};
    const cuuint32_t box[2] = {kChunkK / 8, 8};
    if (!encode_tiled(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, a.packed, dims, strides, box, false)) return XDK_ERR_LAUNCH;
    smap = wmap;
    if (plan.ring_scales) {
      const cuuint64_t sdims[2] = {static_cast<cuuint64_t>(a.groups), static_cast<cuuint64_t>(a.n)};
      const cuuint64_t sstrides[1] = {static_cast<cuuint64_t>(a.groups) * 2};
      const cuuint32_t sbox[2] = {static_cast<cuuint32_t>(kChunkK / a.group), 8};
      if (!encode_tiled(&smap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, a.scales, sdims, sstrides, sbox, false)) return XDK_ERR_LAUNCH;
    }
  }
  auto kernel = w4a16_stream_kernel<MR>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return note_launch(err);
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kStreamThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;

  // How many clusters of S CTAs fit on the device at once (1 CTA per SM; a cluster must sit inside
  // one GPC, so this is not simply SMs / S).  Asked once per S, then cached.
  static int resident[3] = {0, 0, 0};  // S = 1, 2, 4
  auto resident_clusters = [&](int s_log2) {
    if (resident[s_log2] == 0) {
      const int sz = 1 << s_log2;
      int n = 0;
      if (sz == 1) {
        n = sms;
      } else {
        cfg.gridDim = dim3(sms / sz * sz);
        attr[0].val.clusterDim.x = sz;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
          (void)cudaGetLastError();
          n = 0;
        }
      }
      resident[s_log2] = n > 0 ? n : -1;
    }
    return resident[s_log2] > 0 ? resident[s_log2] : 0;
  };
  // Split K over a cluster so that each CTA stages only 1/S of x, as long as (a) the whole grid stays
  // resident in one wave, (b) it does not idle more than ~6 % of the SMs, and (c) the cluster can
  // finish its blocks in one pass (partial sums are parked in shared memory).
  int best_log2 = 0;
  for (int s_log2 = 2; s_log2 >= 1; --s_log2) {
    const int sz = 1 << s_log2;
    if (sz > plan.chunks) continue;
    const int fit = resident_clusters(s_log2);
    if (fit * sz * 100 < sms * 94) continue;
    const int clusters = min(fit, plan.total_blocks);
    if ((plan.total_blocks + clusters - 1) / clusters > kStreamWarps * kMaxNB) continue;
    best_log2 = s_log2;
    break;
  }
  plan.splits = 1 << best_log2;
  plan.clusters = min(resident_clusters(best_log2), plan.total_blocks);
  if (plan.clusters <= 0) plan.clusters = min(sms, plan.total_blocks), plan.splits = 1;
  cfg.gridDim = dim3(plan.clusters * plan.splits);
  attr[0].val.clusterDim.x = plan.splits;
  cfg.numAttrs = plan.splits > 1 ? 1 : 0;
  return note_launch(cudaLaunchKernelEx(&cfg, kernel, a, plan, wmap, smap));
}


// ------------------------------------------------------------------------------------------------
// tcgen05 path (M > 8, K % 256 == 0, group >= 64): the contraction runs on the 5th-generation tensor
// cores.  Operands are swapped so that the UMMA "M" dimension (128 TMEM lanes) carries output columns:
//     D[128 lanes x 16 S] += A[128 x 16 k] * B[16 k x 16 S],   A = dequantised W,  B = x^T
// and A lives in TENSOR MEMORY: the unpack warps write the dequantised weights straight from registers
// into TMEM (tcgen05.st), so they never pass through shared memory.  (With A in shared memory every
// M=128,N=16 MMA re-reads 4 KB of A for 16 columns of use, which by itself saturates the 128 B/clk
// shared-memory port and starves the unpack warps that share it.)
//
// One persistent CTA per SM owns a contiguous, evenly dealt range of 32-column units and walks it in
// strips of <= 4 units, full K each (no cross-CTA reduction).  A warp may touch only the TMEM lane quarter
// warp % 4, so a strip narrower than 128 columns would leave unpack warps idle.  Instead K is split S ways
// over the lane quarters (S = 4 for a 1-unit strip, 2 for 2 units, 1 otherwise): quarter lq holds columns
// of unit lq % (4/S) for the k range lq / (4/S), and B gets 16 S rows, rows 16 ks .. 16 ks + 15 being x over
// k range ks.  An MMA then multiplies every lane with every k range; lane quarter lq keeps only the block of
// 16 accumulator columns that belongs to its own range, and the S partial sums of a column meet in shared
// memory in a fixed order.  (N = 64 costs the tensor pipe no more than N = 16 here: the MMA rate is bound by
// issue, see below.)
//   TMA warp, one lane : box copies of the packed codes of a (strip, 256-k step): one 4 KB, 128-byte swizzled
//                        box per live lane quarter, into a ring of step buffers; plus the strip's scales
//   x warps (2)        : one lane issues one TMA box per k range ([16 rows][256 k], 512-byte rows; a box whose
//                        inner extent is one 16-byte unit would land the operand layout directly, but TMA moves
//                        such boxes unit by unit and was slower than the whole unpack); both warps then move every
//                        16-byte unit to its place in the canonical K-major core-matrix layout ([k group][8 rows]
//                        [8 k]), reordering its 8 k to the order the unpack produces, and hand the buffer to the MMAs
//   unpack warps (8)   : thread = one TMEM lane; warp w owns lane quarter w % 4 and k half w / 4 of every step:
//                        16-byte shared loads of codes -> dequant -> tcgen05.st
//   MMA warps (4)      : one lane each.  A warp gets a tcgen05.mma out only every ~100 cycles, whatever the shape
//                        (measured: 94-118 cycles per M=128 MMA for N = 16 .. 128), while four warps issuing side
//                        by side reach one per ~29 cycles.  So the 16 K=16 blocks of a step are dealt round-robin
//                        to 4 issuers, each accumulating into its OWN accumulator, then tcgen05.commit onto the
//                        barriers (count 4) that hand the stage / x buffer back and announce the finished strip
//   unpack warps 0-3   : epilogue -- tcgen05.ld of the four accumulators, summed in fixed order, (S > 1: the
//                        k-range partials through shared memory,) bias, FP16 store
// TMEM columns (512 allocated; the kernel is alone on its SM): 64 i .. accumulator of issuer i (16 S used),
// 256 + 128 s .. A stage s.
// Every wait is time-bounded; on a timeout the kernel raises g_w4_fault, stops issuing work, and still
// frees its TMEM columns before it returns.
constexpr int kUStepK = 256;                   // k per step: one packed box row (128 bytes), one A stage
constexpr int kUPackedBufs = 4;                // packed steps in flight (16 KB each)
constexpr int kUMaxStages = 3;                 // A operand stages in TMEM: 3 while the accumulators fit 128 columns, else 2
constexpr int kUMaxXBufs = 4;                  // x step buffers (raw and operand layout each): 4 unless a strip splits K four ways
constexpr int kUIssuers = 4;                   // MMA-issuing warps, one accumulator each
constexpr int kUTmemCols = 512;                // allocation (power of two): accumulators first, then the stages
constexpr int kUStageCols = kUStepK / 2;       // 32-bit TMEM columns per stage (two FP16 k per column)
constexpr int kUXLbo = 128, kUXSbo = (kUStepK / 8) * kUXLbo;  // x: [row group of 8][32 k groups][8 rows x 16 B]
constexpr int kUXBytes = 8 * kUXSbo;           // an x buffer for 64 rows (S = 4); the x region is 2 x 2 of these
constexpr int kUXRegion = 2 * kUXBytes;        // bytes of all operand images (and again of all raw buffers)
constexpr int kUPackedBytes = 4 * 32 * (kUStepK / 2);  // 4 lane quarters x 32 rows x 128 B
constexpr int kURedBytes = 128 * 16 * 4;       // k-range partials: [lane][16] floats
constexpr int kWTma = 8, kWMma0 = 9, kWX0 = 10, kWMma1 = 12;  // warp roles; 0-7 unpack, 10-11 x, 12-14 MMA
constexpr int kUThreads = 15 * 32;

struct UmmaPlan {
  int ctas, total_units;  // 32-column units
  int smax;               // widest K split (lane quarters) any strip of the launch uses: sizes the x buffers
  int xdepth;             // x buffers in flight: the x region cut into buffers of smax x 8 KB, at most kUMaxXBufs
  int stages;             // A stages in TMEM
};

__global__ void __launch_bounds__(kUThreads, 1)
w4a16_umma_kernel(W4Args a, UmmaPlan plan, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap smap,
                  const __grid_constant__ CUtensorMap xmap) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* packed = smem_raw;                                 // [kUPackedBufs][kUPackedBytes]
  // A step's x is smax k ranges of [16 rows][256 k] = smax x 8 KB, raw as TMA lands it and again as operand image.
  // With a small smax the same memory holds more steps: the x path (TMA -> x warps -> MMA -> buffer free) is a loop of
  // ~1.4 us, which with two buffers set the step time of the whole kernel.
  const int xstride = plan.smax * 2 * kUXSbo, xdepth = plan.xdepth;
  const int kUStages = plan.stages;
  const int kUAccCols = (kUTmemCols - kUStages * kUStageCols) / kUIssuers, kUTmemA = kUIssuers * kUAccCols;
  unsigned char* xbuf = packed + kUPackedBufs * kUPackedBytes;      // [xdepth][xstride] operand images
  unsigned char* xraw = xbuf + kUXRegion;                           // [xdepth][smax k ranges][16 rows][256 k] as TMA lands it
  unsigned char* scbuf = xraw + kUXRegion;                          // [128 lanes][scale_row_bytes]
  const int scale_row_bytes = a.groups * 2;
  float* red = reinterpret_cast<float*>(scbuf + 128 * scale_row_bytes);  // [128 lanes][16]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(red) + kURedBytes);
  uint64_t* pk_full = bars;                       // [kUPackedBufs]  TMA bytes of a packed step landed
  uint64_t* pk_empty = pk_full + kUPackedBufs;    // [kUPackedBufs]  the 8 unpack warps are done with the step
  uint64_t* a_full = pk_empty + kUPackedBufs;     // [kUMaxStages] the 8 unpack warps wrote the stage to TMEM
  uint64_t* a_empty = a_full + kUMaxStages;       // [kUMaxStages] every issuer's MMAs that read the stage completed
  uint64_t* x_raw = a_empty + kUMaxStages;        // [kUMaxXBufs] TMA bytes of an x step landed
  uint64_t* x_full = x_raw + kUMaxXBufs;          // [kUMaxXBufs] both x warps reordered their share
  uint64_t* x_empty = x_full + kUMaxXBufs;        // [kUMaxXBufs] every issuer's MMAs that read the buffer completed
  uint64_t* sc_full = x_empty + kUMaxXBufs;       // [1]
  uint64_t* acc_full = sc_full + 1;               // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int scale_shift = 31 - __clz(a.group);
  UmmaCursor cur;
  cur.init(blockIdx.x, plan.ctas, plan.total_units, a.k, kUStepK);

  if (threadIdx.x == 0) {
    pdl_launch_dependents();  // the next kernel of the stream may be scheduled (it waits for this one's data itself)
    for (int i = 0; i < kUPackedBufs; ++i) {
      mbar_init(pk_full + i, 1);
      mbar_init(pk_empty + i, 8);   // one arrival per unpack warp
    }
    for (int i = 0; i < xdepth; ++i) {
      mbar_init(x_raw + i, 1);
      mbar_init(x_full + i, 1);     // one x thread, after the x warps met
      mbar_init(x_empty + i, kUIssuers);
    }
    for (int i = 0; i < kUStages; ++i) {
      mbar_init(a_full + i, 8);
      mbar_init(a_empty + i, kUIssuers);
    }
    mbar_init(sc_full, 1);
    mbar_init(acc_full, kUIssuers);
    mbar_fence_init();
  }
  if (warp == kWMma0) {  // TMEM: accumulators + A stages
    tmem_alloc<kUTmemCols>(tmem_slot);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kWTma) {
    // ------------------------------------------------------------ TMA producer: packed codes and scales
    {  // the whole warp runs the loop (waits included), one elected lane issues: operands stay warp-uniform
      bool ok = true;
      int strip_i = 0;
      while (ok && cur.begin_strip()) {
        const int qpk = 4 / cur.split;  // lane quarters per k range = units the strip can hold
        // scales of the strip (whole K, once per live lane quarter): the buffer is free once the unpack warps
        // have released the last packed step of the previous strip
        if (strip_i > 0) {
          const int prev = cur.q - 1;
          ok = __all_sync(0xffffffffu, mbar_wait(pk_empty + prev % kUPackedBufs, (prev / kUPackedBufs) & 1));
          if (!ok) break;
        }
        if (elect_one()) {
          mbar_expect_tx(sc_full, static_cast<unsigned>(cur.units * cur.split * 32 * scale_row_bytes));
          for (int lq = 0; lq < 4; ++lq)
            if (lq % qpk < cur.units) tma_box_2d(scbuf + lq * 32 * scale_row_bytes, &smap, 0, (cur.unit + lq % qpk) * 32, sc_full);
        }
        __syncwarp();
        do {
          const int buf = cur.q % kUPackedBufs;
          if (cur.q >= kUPackedBufs) {
            ok = __all_sync(0xffffffffu, mbar_wait(pk_empty + buf, ((cur.q / kUPackedBufs) - 1) & 1));
            if (!ok) break;
          }
          if (elect_one()) {
            mbar_expect_tx(pk_full + buf, static_cast<unsigned>(cur.units * cur.split * 32 * (kUStepK / 2)));
            for (int lq = 0; lq < 4; ++lq)  // 32-row boxes; the 128-byte swizzle depends on (row & 7) only
              if (lq % qpk < cur.units)
                tma_box_2d(packed + buf * kUPackedBytes + lq * 32 * (kUStepK / 2), &wmap,
                           ((lq / qpk) * cur.kper + cur.kc * kUStepK) / 8, (cur.unit + lq % qpk) * 32, pk_full + buf);
          }
          __syncwarp();
        } while (cur.next_step());
        ++strip_i;
      }
      if (!ok && lane == 0) atomicOr(&g_w4_fault, 4u);
    }
  } else if (warp == kWMma0 || warp >= kWMma1) {
    // ------------------------------------------------------------ MMA issuers
    {  // whole warp, one elected lane issues (a lane-0-only loop issued a tcgen05.mma only every ~120 ns)
      const int issuer = warp == kWMma0 ? 0 : warp - kWMma1 + 1;
      const uint32_t acc = tmem_base + issuer * kUAccCols;
      // x descriptor: only the 14-bit start-address field changes from MMA to MMA
      const uint64_t xd0 = umma_desc(smem_u32(xbuf), kUXLbo, kUXSbo);
      const uint32_t xd_lo = static_cast<uint32_t>(xd0), xd_hi = static_cast<uint32_t>(xd0 >> 32);
      bool ok = true;
      RingPos xp, sp;
      while (ok && cur.begin_strip()) {
        // D = F32, A = B = F16 K-major, N = 16 S, M = 128
        const uint32_t idesc = umma_idesc(16 * cur.split, 0u);
        do {
          const int xb = xp.slot, s = sp.slot;
          ok = __all_sync(0xffffffffu, mbar_wait(x_full + xb, xp.parity) && mbar_wait(a_full + s, sp.parity));
          if (!ok) break;
          xp.advance(xdepth), sp.advance(kUStages);
          tc_fence_after();
          const uint32_t a_base = tmem_base + kUTmemA + s * kUStageCols + issuer * 8;
          const uint32_t x_lo = xd_lo + ((xb * xstride + issuer * 2 * kUXLbo) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < kUStepK / 16 / kUIssuers; ++j) {  // K blocks issuer, issuer + 4, ...
              uint64_t xd;
              asm("mov.b64 %0, {%1, %2};" : "=l"(xd) : "r"(x_lo + ((j * kUIssuers * 2 * kUXLbo) >> 4)), "r"(xd_hi));
              umma_f16_ta(acc, a_base + j * kUIssuers * 8, xd, idesc, !(cur.kc == 0 && j == 0));
            }
            umma_commit(a_empty + s);   // the TMEM stage is free once every issuer's MMAs have read it
            umma_commit(x_empty + xb);
          }
          __syncwarp();
        } while (cur.next_step());
        if (ok && elect_one()) umma_commit(acc_full);
        __syncwarp();
      }
      if (!ok && lane == 0) atomicOr(&g_w4_fault, 8u);
    }
  } else if (warp >= kWX0) {
    // ------------------------------------------------------------ x warps
    const int t = threadIdx.x - kWX0 * 32;  // 0 .. 63
    bool ok = true;
    UmmaCursor ahead = cur;  // issues the loads, xdepth steps in front of `cur`
    bool ahead_live = ahead.begin_strip();
    RingPos xi, xs;          // of the load being issued, of the step being reordered
    auto issue = [&]() {  // raw buffer xi.slot is free: its last readers passed the x-warp barrier
      if (!ahead_live) return;
      if (t == 0) {
        const int xb = xi.slot;
        mbar_expect_tx(x_raw + xb, static_cast<unsigned>(ahead.split * 16 * kUStepK * 2));
        for (int ks = 0; ks < ahead.split; ++ks)  // rows >= M are out of range: zero-filled, still counted
          tma_box_2d(xraw + xb * xstride + ks * 16 * kUStepK * 2, &xmap, ks * ahead.kper + ahead.kc * kUStepK, 0, x_raw + xb);
      }
      xi.advance(xdepth);
      if (!ahead.next_step()) ahead_live = ahead.begin_strip();
    };
    if (t == 0) pdl_wait();  // x is the preceding kernel's output; packed codes and scales (issued already) are not
    for (int i = 0; i < xdepth; ++i) issue();
    // A quarter warp moves an 8-row x 8-k-group block per pass along its diagonals: lane i takes k group i of row
    // (i + r) & 7, so the eight 16-byte loads (row pitch 512 B) and the eight stores (k-group pitch 128 B) each hit
    // eight different bank groups.
    const int qw = t >> 3, li = t & 7;        // 8 quarter warps: (row group, quarter of the 32 k groups)
    const int mg = qw >> 2, kg = (qw & 3) * 8 + li;
    while (cur.begin_strip()) {
      do {
        const int xb = xs.slot;
        if (ok) ok = mbar_wait(x_raw + xb, xs.parity);
        if (ok) ok = mbar_wait(x_empty + xb, xs.parity ^ 1u);  // a fresh barrier passes: nothing has read the buffer yet
        xs.advance(xdepth);
        if (ok) {
          auto fetch = [&](int ks, U4 (&v)[8]) {
            const unsigned char* src = xraw + xb * xstride + ks * 16 * kUStepK * 2 + kg * 16;
#pragma unroll
            for (int r = 0; r < 8; ++r) v[r] = *reinterpret_cast<const U4*>(src + (mg * 8 + ((li + r) & 7)) * (kUStepK * 2));
          };
          auto place = [&](int ks, const U4 (&v)[8]) {
            unsigned char* dst = xbuf + xb * xstride + (ks * 2 + mg) * kUXSbo + kg * kUXLbo;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              U4 o;  // k 0..7 of one row -> 0,4,1,5,2,6,3,7, the order the unpack produces
              o.x = __byte_perm(v[r].x, v[r].z, 0x5410);
              o.y = __byte_perm(v[r].x, v[r].z, 0x7632);
              o.z = __byte_perm(v[r].y, v[r].w, 0x5410);
              o.w = __byte_perm(v[r].y, v[r].w, 0x7632);
              *reinterpret_cast<U4*>(dst + ((li + r) & 7) * 16) = o;
            }
          };
          if (cur.split == 1) {
            U4 v[8];
            fetch(0, v);
            place(0, v);
          } else {
            // a step of a strip that splits K carries 2 or 4 k ranges of x: two at a time, so that the two x warps
            // have sixteen loads in flight instead of eight (the x path sets the step time of these strips)
            for (int ks = 0; ks < cur.split; ks += 2) {
              U4 va[8], vb[8];
              fetch(ks, va);
              fetch(ks + 1, vb);
              place(ks, va);
              place(ks + 1, vb);
            }
          }
          fence_async_smem();
        }
        asm volatile("bar.sync 2, 64;" ::: "memory");  // both x warps are done with the raw buffer and wrote their share
        if (t == 0) mbar_arrive_cta(x_full + xb);
        issue();
      } while (cur.next_step());
    }
    if (!ok && lane == 0) atomicOr(&g_w4_fault, 32u);
  } else {
    // ------------------------------------------------------------ unpack warps (+ epilogue)
    const int lq = warp & 3, kh = warp >> 2;  // TMEM lane quarter this warp may touch, k half of a step
    const int c = lq * 32 + lane;             // this thread's TMEM lane
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(lq * 32) << 16);
    const uint32_t a_lane_base = lane_base + kUTmemA + kh * (kUStageCols / 2);
    const __half* sc_row = reinterpret_cast<const __half*>(scbuf + c * scale_row_bytes);
    int strip_i = 0;
    bool ok = true;
    RingPos sp;
    while (cur.begin_strip()) {
      const int qpk = 4 / cur.split;
      const int ks = lq / qpk, uq = lq % qpk;   // this quarter's k range and unit of the strip
      const bool warp_live = uq < cur.units;    // warp-uniform: a quarter without columns writes nothing
      const int col = (cur.unit + uq) * 32 + lane;  // output column of this thread
      const int k_range0 = ks * cur.kper;
      const int split = cur.split;
      if (ok) ok = mbar_wait(sc_full, strip_i & 1);
      do {
        const int buf = cur.q % kUPackedBufs, s = sp.slot;
        if (ok) ok = mbar_wait(pk_full + buf, (cur.q / kUPackedBufs) & 1);
        if (ok) ok = mbar_wait(a_empty + s, sp.parity ^ 1u);
        sp.advance(kUStages);
        if (ok && warp_live) {
          tc_fence_after();
          // packed tiles arrive 128-byte swizzled: 16-byte piece p of row r sits at piece p ^ (r & 7), so the
          // lanes of a warp, which read the same piece of 32 different rows, spread over all bank groups
          const unsigned char* row = packed + buf * kUPackedBytes + c * (kUStepK / 2);
          const int k_half = k_range0 + cur.kc * kUStepK + kh * (kUStepK / 2);
#pragma unroll
          for (int pp = 0; pp < kUStepK / 128; ++pp) {  // two pieces = 64 k = 32 TMEM columns per store
            // (a tcgen05.st costs the warp ~125 ns whatever its width, so 32 columns go out at once)
            uint32_t r[32];
            // two pieces = 64 k lie inside one group (group >= 64)
            const __half2 s2 = __half2half2(sc_row[(k_half + pp * 64) >> scale_shift]);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int piece = kh * (kUStepK / 64) + pp * 2 + half;
              const U4 wv = *reinterpret_cast<const U4*>(row + ((piece ^ (c & 7)) << 4));  // rows past N are zero-filled: harmless
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                const uint32_t word = w == 0 ? wv.x : (w == 1 ? wv.y : (w == 2 ? wv.z : wv.w));
                __half2 h[4];
                dequant8(word, s2, h);
#pragma unroll
                for (int i = 0; i < 4; ++i) r[16 * half + 4 * w + i] = *reinterpret_cast<uint32_t*>(&h[i]);
              }
            }
            tmem_st32(a_lane_base + s * kUStageCols + pp * 32, r);
          }
          tmem_wait_st();
          tc_fence_before();
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_cta(a_full + s);
          mbar_arrive_cta(pk_empty + buf);
        }
      } while (cur.next_step());
      // ---- epilogue of the strip: warps 0-3 read their own lane quarter of the four accumulators
      float sum[16];
      if (warp < 4) {
        if (ok) ok = mbar_wait(acc_full, strip_i & 1);
        if (ok && warp_live) {
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < kUIssuers; ++i) {
            uint32_t r[16];
            tmem_ld16(lane_base + i * kUAccCols + ks * 16, r);  // the 16 accumulator columns of this quarter's own k range
#pragma unroll
            for (int m = 0; m < 16; ++m) sum[m] = i == 0 ? __uint_as_float(r[m]) : __fadd_rn(sum[m], __uint_as_float(r[m]));
          }
          tc_fence_before();
          if (split > 1) {
#pragma unroll
            for (int m = 0; m < 16; m += 4)
              *reinterpret_cast<float4*>(red + c * 16 + m) = make_float4(sum[m], sum[m + 1], sum[m + 2], sum[m + 3]);
          }
        }
      }
      if (split > 1) {
        asm volatile("bar.sync 1, 256;" ::: "memory");  // strip-uniform: the k-range partials are in shared memory
        if (warp < 4 && ok && warp_live && ks == 0) {
          for (int j = 1; j < split; ++j)  // fixed order: k range 0 + 1 + 2 + 3
#pragma unroll
            for (int m = 0; m < 16; ++m) sum[m] = __fadd_rn(sum[m], red[(c + j * qpk * 32) * 16 + m]);
        }
      }
      if (warp < 4 && ok && warp_live && ks == 0 && col < a.n) {
        const float bv = a.bias ? __half2float(a.bias[col]) : 0.0f;
#pragma unroll
        for (int m = 0; m < 16; ++m)
          if (m < a.m) peer_store(a.out, m, col, __float2half_rn(sum[m] + bv));
      }
      // all 256 threads meet before the next strip's stages can reach the MMA warps (a_full needs all of them),
      // so the next strip's first MMAs cannot overwrite TMEM (nor its partials the shared buffer) while they are read
      asm volatile("bar.sync 1, 256;" ::: "memory");
      ++strip_i;
    }
    if (!ok && lane == 0) atomicOr(&g_w4_fault, 16u);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kWMma0) {
    tc_fence_after();
    tmem_dealloc<kUTmemCols>(tmem_base);
  }
}

int launch_umma(const W4Args& a, bool dependent, cudaStream_t stream) {
  UmmaPlan plan;
  plan.total_units = (a.n + 31) / 32;
  plan.ctas = plan.total_units < sm_count() ? plan.total_units : sm_count();
  plan.smax = 1;
  for (int cta = 0; cta < plan.ctas; ++cta) {  // a CTA's strips: whole ones of four units, then the rest
    const int units = static_cast<int>(static_cast<int64_t>(cta + 1) * plan.total_units / plan.ctas - static_cast<int64_t>(cta) * plan.total_units / plan.ctas);
    if (units % 4 != 0) plan.smax = max(plan.smax, umma_split(units % 4, a.k, kUStepK));
  }
  plan.xdepth = 8 / plan.smax < kUMaxXBufs ? 8 / plan.smax : kUMaxXBufs;
  plan.stages = plan.smax <= 2 ? kUMaxStages : 2;  // 16 smax accumulator columns per issuer must fit beside the stages
  const size_t smem = kUPackedBufs * kUPackedBytes + 2 * kUXRegion + 128 * a.groups * 2 + kURedBytes + 48 * sizeof(uint64_t);
  if (smem > 225 * 1024) return XDK_ERR_LIMIT;
  CUtensorMap wmap, smap, xmap;
  {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(a.k / 8), static_cast<cuuint64_t>(a.n)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(a.k / 2)};
    const cuuint32_t box[2] = {kUStepK / 8, 32};
    const cuuint64_t sdims[2] = {static_cast<cuuint64_t>(a.groups), static_cast<cuuint64_t>(a.n)};
    const cuuint64_t sstrides[1] = {static_cast<cuuint64_t>(a.groups) * 2};
    const cuuint32_t sbox[2] = {static_cast<cuuint32_t>(a.groups), 32};
    static_assert(kUStepK / 2 == 128, "the packed box is one 128-byte swizzle span wide");
    if (!encode_tiled(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, a.packed, dims, strides, box, true) ||
        !encode_tiled(&smap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, a.scales, sdims, sstrides, sbox, false))
      return XDK_ERR_LAUNCH;
    const cuuint64_t xdims[2] = {static_cast<cuuint64_t>(a.k), static_cast<cuuint64_t>(a.m)};
    const cuuint64_t xstrides[1] = {static_cast<cuuint64_t>(a.k) * 2};
    const cuuint32_t xbox[2] = {kUStepK, 16};
    if (!encode_tiled(&xmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, a.x, xdims, xstrides, xbox, false)) return XDK_ERR_LAUNCH;
  }
  cudaError_t err = cudaFuncSetAttribute(w4a16_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return note_launch(err);
  return launch_opts(w4a16_umma_kernel, dim3(plan.ctas), dim3(kUThreads), smem, stream, 1u, dependent, a, plan, wmap, smap, xmap);
}

// Any K (odd included), any alignment: warp per column, lane per byte (two codes), rows one at a
// time.  Slow; it exists so that every shape the format allows has a GPU path.
__global__ void __launch_bounds__(kThreads)
w4a16_generic_kernel(W4Args a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * kWarps + warp;
  if (col >= a.n) return;
  const int row_bytes = (a.k + 1) / 2;
  for (int r = 0; r < a.m; ++r) {
    float acc = 0.0f;
    for (int b = lane; b < row_bytes; b += 32) {
      const uint32_t byte = a.packed[static_cast<size_t>(col) * row_bytes + b];
      const int k0 = 2 * b;
      const float s0 = __half2float(a.scales[static_cast<size_t>(col) * a.groups + k0 / a.group]);
      const float w0 = __half2float(__float2half_rn(__fmul_rn(static_cast<float>(static_cast<int>(byte & 15u) - 8), s0)));
      acc = fmaf(w0, __half2float(a.x[static_cast<size_t>(r) * a.k + k0]), acc);
      if (k0 + 1 < a.k) {
        const float s1 = __half2float(a.scales[static_cast<size_t>(col) * a.groups + (k0 + 1) / a.group]);
        const float w1 = __half2float(__float2half_rn(__fmul_rn(static_cast<float>(static_cast<int>(byte >> 4) - 8), s1)));
        acc = fmaf(w1, __half2float(a.x[static_cast<size_t>(r) * a.k + k0 + 1]), acc);
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      const float b = a.bias ? __half2float(a.bias[col]) : 0.0f;
      a.y[static_cast<size_t>(r) * a.n + col] = __float2half_rn(acc + b);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Direct-load tensor-core path for M <= 8 and K % 1024 == 0.
//
// The SIMT kernel spends five thread instructions per code (the exact unpack, then an FMA per code and row with
// both operands taken out of their half2 pairs) and is issue-bound at a third of the HBM rate on this part.  Here
// the unpack's half2 pairs go to mma.m16n8k16 as they are, with the operands swapped so that no row of the MMA is
// wasted on small M: the 16 rows of the MMA are 16 columns of W, its 8 columns are the (up to 8) rows of x.  Lane
// (n = lane / 4, q = lane % 4) loads the 16-byte vectors (32 codes) of columns n and n + 8 that start at
// k = chunk + 32 q.  An MMA does not care which k a fragment slot stands for as long as A and B agree, so slot pairs
// are simply "the pairs the unpack produces": word w of a vector gives A pairs (k0,k4) (k1,k5) for one MMA and
// (k2,k6) (k3,k7) for the next, and the matching B pairs are one 16-byte read of x, which sits in shared memory
// already permuted to (0,4,1,5,2,6,3,7) inside every 8 k.  The legacy HMMA pipe of this part retires one m16n8k16
// per 8 cycles and sub-partition (measured; 1.6 us for K = 4096, N = 14336 in this form), the 13 instructions of the exact
// unpack take 24, so the instruction stream is what counts: 26 warp instructions per MMA
// are left, after taking everything out of the loop that does not depend on the
// codes -- no zero-filling of registers for columns past N or rows past M (they read a valid column or row and
// feed outputs that are never stored), scales widened to half2 when they are fetched, one base pointer per column.
// The grid is one wave (as many CTAs as are resident at once), the groups of 16 columns dealt evenly.
// A CTA is eight warps that split K eight ways over the same 16 columns and add their partial sums in shared
// memory in warp order.  A warp's work is a sequence of batches (a column pass x a round of up to four 128-k chunks
// of its K share); the loads of the next batch are in flight while the current one is unpacked and multiplied, in
// two register buffers, so the weight stream never waits for the tensor pipe nor the pipe for the stream.
//
// Two shapes of it: batches of four chunks and two CTAs per SM (127 registers), or of two chunks and three (80), for more
// column groups than two CTAs per SM take in one pass each, while x is small enough to leave the third CTA room and the L1
// cache its scales.
template <int CHUNKS>
struct MmaBatch {
  U4 wv[CHUNKS][2];       // [chunk][column n, column n + 8]: 32 codes each
  __half2 sc[CHUNKS][2];  // their scale, in both halves
};

template <int CHUNKS, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS)
w4a16_mma_kernel(W4Args a, int col_groups) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int pitch = a.k * 2 + 16;                          // bytes per x row: the pad puts the 8 rows on different banks
  unsigned char* xs = smem_raw;                            // [m rows][pitch], k permuted inside every 8
  float* red = reinterpret_cast<float*>(smem_raw + ((static_cast<size_t>(a.m) * pitch + 127) & ~static_cast<size_t>(127)));  // [2][8 warps][32 lanes][4]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = lane >> 2, q = lane & 3;
  const int row_bytes = a.k / 2;
  const int k_warp = a.k / kWarps;          // this warp's share of K, a multiple of 128
  const int chunks = k_warp / 128;          // 128 k per chunk: 32 per lane of a quad
  constexpr int kBatchChunks = CHUNKS;
  const int rounds = (chunks + kBatchChunks - 1) / kBatchChunks;
  const int k0 = warp * k_warp + q * 32;    // first k of this lane's vectors
  // the groups of 16 columns are dealt evenly to the CTAs of the grid (all resident at once: no second wave)
  const int group0 = static_cast<int>(static_cast<int64_t>(blockIdx.x) * col_groups / gridDim.x);
  const int my_passes = static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * col_groups / gridDim.x) - group0;  // >= 1
  const int cta_col0 = group0 * 16;

  const int scale_shift = 31 - __clz(a.group);  // group sizes are powers of two
  // Columns past N (the last pass of the last CTA when N % 16 != 0) read the last column instead and chunks past the
  // warp's share are not loaded at all: what they would feed is never stored, respectively never computed.
  auto fetch = [&](MmaBatch<CHUNKS>& b, int col_base, int chunk0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = min(col_base + h * 8 + n, a.n - 1), k = k0 + chunk0 * 128;
      const uint8_t* wp = a.packed + static_cast<size_t>(col) * row_bytes + k / 2;
      const __half* sp = a.scales + static_cast<size_t>(col) * a.groups;
#pragma unroll
      for (int c = 0; c < kBatchChunks; ++c)
        if (chunk0 + c < chunks) {
          b.wv[c][h] = ld_stream16(wp + c * 64);
          b.sc[c][h] = __half2half2(__ldg(sp + ((k + c * 128) >> scale_shift)));
        }
    }
  };
  MmaBatch<CHUNKS> buf0, buf1;
  pdl_launch_dependents();
  fetch(buf0, cta_col0, 0);  // the first batch's weights go out before x is staged
  pdl_wait();                // x may be the preceding kernel's output; the weights are not

  // x into shared memory: 16 bytes per thread and load, eight loads in flight, then four, two and one for the rest (K % 1024 == 0: the
  // same for all threads of a warp)
  const int units = a.k / 8, x_units = a.m * units;
  const uint32_t per_unit = 0xffffffffu / units + 1;  // i / units = the high word of i * per_unit, for i * units below 2^32
  int at = threadIdx.x;
  auto stage = [&](auto flight) {
    constexpr int F = decltype(flight)::value;
    U4 v[F];
#pragma unroll
    for (int j = 0; j < F; ++j) v[j] = ld_ordered16(a.x + static_cast<size_t>(at + j * kThreads) * 8);
#pragma unroll
    for (int j = 0; j < F; ++j) {
      const int i = at + j * kThreads, r = static_cast<int>(__umulhi(i, per_unit));
      U4 o;  // k 0..7 -> 0,4,1,5,2,6,3,7: the pairs the unpack produces
      o.x = __byte_perm(v[j].x, v[j].z, 0x5410);
      o.y = __byte_perm(v[j].x, v[j].z, 0x7632);
      o.z = __byte_perm(v[j].y, v[j].w, 0x5410);
      o.w = __byte_perm(v[j].y, v[j].w, 0x7632);
      *reinterpret_cast<U4*>(xs + (i + r) * 16) = o;  // 16 bytes of pad behind every row
    }
    at += F * kThreads;
  };
  while (at + 7 * kThreads < x_units) stage(std::integral_constant<int, 8>{});
  if (at + 3 * kThreads < x_units) stage(std::integral_constant<int, 4>{});
  if (at + kThreads < x_units) stage(std::integral_constant<int, 2>{});
  if (at < x_units) stage(std::integral_constant<int, 1>{});
  __syncthreads();
  // this lane's B fragments: row n of x; lanes past M read row 0 and feed output rows that are never stored
  const unsigned char* xrow = xs + static_cast<size_t>(n < a.m ? n : 0) * pitch;

  // two accumulator sets (the two MMAs of a word alternate, halving the dependent chain), summed at the end of a pass:
  // (column n, rows 2 q + {0, 1} of x), (column n + 8, the same rows)
  float acc0[4], acc1[4];
  int pass = 0, round = 0;  // of the batch being computed
  auto step = [&](MmaBatch<CHUNKS>& cur, MmaBatch<CHUNKS>& nxt) -> bool {
    int np = pass, nr = round + 1;
    if (nr == rounds) nr = 0, ++np;
    const bool has_next = np < my_passes;
    if (has_next) fetch(nxt, cta_col0 + np * 16, nr * kBatchChunks);
    if (round == 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc0[e] = acc1[e] = 0.0f;
    }
    const int chunk0 = round * kBatchChunks;
#pragma unroll
    for (int c = 0; c < kBatchChunks; ++c) {
      if (chunk0 + c < chunks) {
        const unsigned char* xk = xrow + (k0 + (chunk0 + c) * 128) * 2;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const U4 xv = *reinterpret_cast<const U4*>(xk + w * 16);
          const uint32_t w0 = w == 0 ? cur.wv[c][0].x : (w == 1 ? cur.wv[c][0].y : (w == 2 ? cur.wv[c][0].z : cur.wv[c][0].w));
          const uint32_t w1 = w == 0 ? cur.wv[c][1].x : (w == 1 ? cur.wv[c][1].y : (w == 2 ? cur.wv[c][1].z : cur.wv[c][1].w));
          __half2 h0[4], h1[4];
          dequant8(w0, cur.sc[c][0], h0);
          dequant8(w1, cur.sc[c][1], h1);
          mma16816(acc0, *reinterpret_cast<uint32_t*>(&h0[0]), *reinterpret_cast<uint32_t*>(&h1[0]), *reinterpret_cast<uint32_t*>(&h0[1]),
                   *reinterpret_cast<uint32_t*>(&h1[1]), xv.x, xv.y);
          mma16816(acc1, *reinterpret_cast<uint32_t*>(&h0[2]), *reinterpret_cast<uint32_t*>(&h1[2]), *reinterpret_cast<uint32_t*>(&h0[3]),
                   *reinterpret_cast<uint32_t*>(&h1[3]), xv.z, xv.w);
        }
      }
    }
    if (round == rounds - 1) {
      // the partial sums of the pass meet in shared memory; the buffer alternates between passes, so one barrier
      // per pass is enough (the warp that adds pass p has passed the barrier of pass p + 1 before anybody writes
      // the buffer of pass p + 2), and the adding warp rotates
      float* mine = red + (pass & 1) * (kWarps * 32 * 4);
      *reinterpret_cast<float4*>(mine + (warp * 32 + lane) * 4) =
          make_float4(__fadd_rn(acc0[0], acc1[0]), __fadd_rn(acc0[1], acc1[1]), __fadd_rn(acc0[2], acc1[2]), __fadd_rn(acc0[3], acc1[3]));
      __syncthreads();
      if (warp == (pass & (kWarps - 1))) {  // the eight partial sums in warp order, bias, store
        const int col_base = cta_col0 + pass * 16;
        float4 total = *reinterpret_cast<const float4*>(mine + lane * 4);
        for (int w = 1; w < kWarps; ++w) {
          const float4 part = *reinterpret_cast<const float4*>(mine + (w * 32 + lane) * 4);
          total.x = __fadd_rn(total.x, part.x), total.y = __fadd_rn(total.y, part.y);
          total.z = __fadd_rn(total.z, part.z), total.w = __fadd_rn(total.w, part.w);
        }
        const float out[4] = {total.x, total.y, total.z, total.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = col_base + (e >> 1) * 8 + n, row = q * 2 + (e & 1);
          if (row < a.m && col < a.n)
            a.y[static_cast<size_t>(row) * a.n + col] = __float2half_rn(out[e] + (a.bias ? __half2float(a.bias[col]) : 0.0f));
        }
      }
    }
    pass = np, round = nr;
    return has_next;
  };
  while (step(buf0, buf1) && step(buf1, buf0)) {
  }
}

template <int CHUNKS, int CTAS>
int launch_mma(W4Args a, bool dependent, cudaStream_t stream) {
  const size_t xbytes = (static_cast<size_t>(a.m) * (a.k * 2 + 16) + 127) & ~static_cast<size_t>(127);
  const size_t smem = xbytes + 2 * static_cast<size_t>(kWarps) * 32 * 4 * sizeof(float);
  cudaError_t err = cudaFuncSetAttribute(w4a16_mma_kernel<CHUNKS, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return note_launch(err);
  // one wave: as many CTAs as the device holds at once (two per SM unless x takes more than half the shared memory);
  // a grid of a few CTAs more than that ran as two waves and took twice the time
  int resident = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, w4a16_mma_kernel<CHUNKS, CTAS>, kThreads, smem);
  if (err != cudaSuccess) return note_launch(err);
  if (resident < 1) return XDK_ERR_LIMIT;
  const int groups = (a.n + 15) / 16;
  const int ctas = groups < resident * sm_count() ? groups : resident * sm_count();
  return launch_opts(w4a16_mma_kernel<CHUNKS, CTAS>, dim3(ctas), dim3(kThreads), smem, stream, 1u, dependent, a, groups);
}

// ------------------------------------------------------------------------------------------------
// Tensor-core path for K % 128 == 0 (every M, every group size): x stays in registers, W streams past it.
//
// An MMA (m16n8k16) takes 16 columns of W as its rows and 8 rows of x as its columns.  A warp owns one slice of 256 k
// and keeps x of that slice -- all rows -- in registers as ready B fragments (32 registers per 8 rows); it walks
// column groups of 16, one pass each.  So the loop touches shared memory only for the codes: TMA box copies
// ([16 columns][128 B], 128-byte swizzle) into a ring private to the warp, refilled by the warp itself.  Lane
// (i = lane / 4, q = lane % 4) unpacks 32 codes of two columns at a time; the slots of a fragment are simply "the half2
// pairs the exact unpack produces": word w of a vector gives A pairs (k0,k4) (k1,k5) for one MMA and (k2,k6) (k3,k7)
// for the next, and x is permuted to match when it is loaded.  MMA row i stands for column (i / 2) + 4 (i % 2) of the
// group: with the swizzle, the two rows a quarter-warp reads then lie on different halves of the banks.
//
// The warps of a column set (one per slice) park their partial sums in shared memory, pass by pass; the warp whose turn
// it is adds them in slice order one pass later, so nobody waits at a barrier.  K > 4096 is split over the CTAs of a
// cluster: a rank's sums go through distributed shared memory to the rank that owns the pass, and are added there, in
// rank order, once after the cluster's barrier.  K < 4096 leaves warps over, which form further column sets.
//
// What bounds it: the exact unpack.  HFMA2 and LOP3 take two issue slots each and do not overlap on this part, so the 13
// instructions of eight codes cost a sub-partition 24 cycles per 256 weights, an MMA 8 (measured); a pass runs at about
// half of that bound, the rest is the passes' hand-overs.  Against the tcgen05 kernel, which pays for K split over its lane
// quarters with four x ranges a step: M = 16, K = 14336, N = 4096 34.0 -> 22.6 us, K = 11008 30.5 -> 19.6; the dispatch at the
// end of the file has both sides of its rule.  The lanes sharing one scale load each through shuffles measured slower
// (M = 1, N = 28672 25.6 against 22.7).
constexpr int kRxWarps = 16;       // at most, per CTA (one CTA per SM: 128 registers a thread)
constexpr int kRxSliceK = 256;     // k per warp
constexpr int kRxStage = 16 * kRxSliceK / 2;  // bytes of codes of a pass
constexpr int kRxMaxDepth = 6;     // passes in flight per warp
constexpr int kRxParts = 3;        // buffers of partial sums per column set
constexpr int kRxMaxPasses = 64;   // of a cluster: bounds the sums it parks
constexpr int kRxSmem = 226 * 1024;

struct RxPlan {
  int slices;      // of K, all ranks
  int ranks;       // CTAs per cluster that share K
  int cta_slices;  // slices per CTA
  int sets;        // column sets per CTA
  int total_sets;  // of the launch
  int groups;      // column groups of 16
  int depth;       // ring slots per warp
  int parked;      // passes a rank owns (ranks > 1)
};

template <int MR>  // rows of x in eights
__global__ void __launch_bounds__(kRxWarps * 32, 1)
w4a16_rx_kernel(W4Args a, RxPlan plan, const __grid_constant__ CUtensorMap wmap) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const int warps = plan.cta_slices * plan.sets;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = lane >> 2, q = lane & 3;
  const int set = warp / plan.cta_slices, ws = warp - set * plan.cta_slices;
  const int rank = blockIdx.y;
  const int slice = rank * plan.cta_slices + ws;
  const int live_slices = min(plan.cta_slices, plan.slices - rank * plan.cta_slices);  // the last rank may hold fewer
  const int depth = plan.depth;
  unsigned char* ring = smem_raw + warp * depth * kRxStage;
  float4* part = reinterpret_cast<float4*>(smem_raw + warps * depth * kRxStage) + set * kRxParts * plan.cta_slices * MR * 32;
  float4* parked = reinterpret_cast<float4*>(smem_raw + warps * depth * kRxStage) + plan.sets * kRxParts * plan.cta_slices * MR * 32;
  uint64_t* bars = reinterpret_cast<uint64_t*>(parked + (plan.ranks > 1 ? plan.parked * plan.ranks * MR * 32 : 0));
  uint64_t* full = bars + warp * depth;                                  // this warp's slots
  uint64_t* part_full = bars + warps * depth + set * 2 * kRxParts;       // every warp of the set wrote its partial sums
  uint64_t* part_empty = part_full + kRxParts;                           // they have been added

  const int set_id = blockIdx.x * plan.sets + set;
  const int g0 = static_cast<int>(static_cast<int64_t>(set_id) * plan.groups / plan.total_sets);
  const int passes = ws < live_slices
      ? static_cast<int>(static_cast<int64_t>(set_id + 1) * plan.groups / plan.total_sets) - g0 : 0;

  auto issue = [&](int slot, int pass) {  // one lane
    mbar_expect_tx(full + slot, kRxStage);  // parts of a box past K or N are zero-filled and still counted
    tma_box_2d(ring + slot * kRxStage, &wmap, slice * (kRxSliceK / 8), (g0 + pass) * 16, full + slot);
  };
  if (lane == 0) {
    for (int s = 0; s < depth; ++s) mbar_init(full + s, 1);
    if (ws == 0)
      for (int b = 0; b < kRxParts; ++b) mbar_init(part_full + b, live_slices), mbar_init(part_empty + b, 1);
    mbar_fence_init();
    for (int p = 0; p < depth && p < passes; ++p) issue(p, p);  // the weights do not depend on the preceding kernel
    pdl_launch_dependents();
  }
  const int col_lo = (i >> 1) + ((i & 1) << 2);  // this lane's columns of a group: col_lo and col_lo + 8
  const int k0 = slice * kRxSliceK + q * 32;
  // this lane's scales of a pass, fetched a pass ahead: two columns h, its quarter of each 128-k chunk c
  const int scale_shift = 31 - __clz(a.group);
  int scale_idx[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) scale_idx[c] = min((k0 + c * 128) >> scale_shift, a.groups - 1);
  // A second chunk past K (the first one never is) has codes of zero, which stand for -8: its scale counts as zero, any above
  // 8188 would make infinities of them.
  const uint32_t second_live = k0 + 128 < a.k ? 0xffffffffu : 0u;
  __half scale_next[2][2];
  auto fetch_scales = [&](int pass) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // past N: any column, its sums are not stored
      const __half* at = a.scales + static_cast<size_t>(min((g0 + pass) * 16 + h * 8 + col_lo, a.n - 1)) * a.groups;
#pragma unroll
      for (int c = 0; c < 2; ++c) scale_next[c][h] = __ldg(at + scale_idx[c]);
    }
  };
  fetch_scales(0);
  __syncthreads();  // barriers of the sets
  if (plan.ranks > 1) cg::this_cluster().barrier_arrive();  // the other ranks' shared memory is there after the wait

  pdl_wait();  // x may be the preceding kernel's output; codes, scales and bias are not
  uint32_t xf[2][MR][4][4];  // [chunk of 128 k][row group][word][fragment pair]
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < MR; ++r) {
      // rows past M and k past K are zeros; they read a valid address, so that the loads go out without a branch
      const int row = r * 8 + i, k = k0 + c * 128;
      const bool live = row < a.m && k < a.k;
      const __half* src = a.x + static_cast<size_t>(min(row, a.m - 1)) * a.k + (k < a.k ? k : 0);
      U4 v[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) v[w] = ld_ordered16(src + w * 8);
#pragma unroll
      for (int w = 0; w < 4; ++w) {  // k 0..7 -> 0,4 1,5 2,6 3,7
        xf[c][r][w][0] = live ? __byte_perm(v[w].x, v[w].z, 0x5410) : 0u;
        xf[c][r][w][1] = live ? __byte_perm(v[w].x, v[w].z, 0x7632) : 0u;
        xf[c][r][w][2] = live ? __byte_perm(v[w].y, v[w].w, 0x5410) : 0u;
        xf[c][r][w][3] = live ? __byte_perm(v[w].y, v[w].w, 0x7632) : 0u;
      }
    }
  if (plan.ranks > 1) cg::this_cluster().barrier_wait();

  bool ok = true;
  const size_t out_at = static_cast<size_t>(q * 2) * a.n + g0 * 16 + col_lo;  // plain outputs only: strided ones go elsewhere
  auto store = [&](int pass, const float4 (&sum)[MR]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = (g0 + pass) * 16 + h * 8 + col_lo;
      if (col >= a.n) continue;
      const float bv = a.bias ? __half2float(a.bias[col]) : 0.0f;
      __half* dst = a.y + out_at + pass * 16 + h * 8;
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        if (r * 8 + q * 2 < a.m) dst[static_cast<size_t>(r) * 8 * a.n] = __float2half_rn((h ? sum[r].z : sum[r].x) + bv);
        if (r * 8 + q * 2 + 1 < a.m) dst[static_cast<size_t>(r * 8 + 1) * a.n] = __float2half_rn((h ? sum[r].w : sum[r].y) + bv);
      }
    }
  };
  auto reduce = [&](int pass) {  // one warp: the partial sums of a pass in slice order
    const int b = pass % kRxParts;
    if (ok) ok = mbar_wait(part_full + b, (pass / kRxParts) & 1);
    const float4* src = part + b * plan.cta_slices * MR * 32 + lane;
    float4 sum[MR];
#pragma unroll
    for (int r = 0; r < MR; ++r) sum[r] = src[r * 32];
#pragma unroll 4
    for (int s = 1; s < live_slices; ++s)
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        const float4 v = src[(s * MR + r) * 32];
        sum[r].x = __fadd_rn(sum[r].x, v.x), sum[r].y = __fadd_rn(sum[r].y, v.y);
        sum[r].z = __fadd_rn(sum[r].z, v.z), sum[r].w = __fadd_rn(sum[r].w, v.w);
      }
    __syncwarp();
    if (lane == 0) mbar_arrive_cta(part_empty + b);
    if (plan.ranks == 1) {
      if (ok) store(pass, sum);
    } else {
      const int owner = pass % plan.ranks;
      const uint32_t dst = cluster_map(parked + ((pass / plan.ranks) * plan.ranks + rank) * MR * 32 + lane, owner);
#pragma unroll
      for (int r = 0; r < MR; ++r) cluster_store_f4(dst + r * 32 * sizeof(float4), sum[r]);
    }
  };

  RingPos slot, pb;  // ring slot, partial-sum buffer
  int turn = 0;      // whose turn it is to add the previous pass (pass - 1) % live_slices
  for (int pass = 0; pass < passes; ++pass) {
    __half2 sc[2][2];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const __half2 both = __half2half2(scale_next[c][h]);
        const uint32_t bits = *reinterpret_cast<const uint32_t*>(&both) & (c ? second_live : 0xffffffffu);
        sc[c][h] = *reinterpret_cast<const __half2*>(&bits);
      }
    if (pass + 1 < passes) fetch_scales(pass + 1);
    if (ok) ok = mbar_wait(full + slot.slot, slot.parity);
    float acc[MR][4];
#pragma unroll
    for (int r = 0; r < MR; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[r][e] = 0.0f;
    const unsigned char* lo = ring + slot.slot * kRxStage + col_lo * 128;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int at = ((c * 4 + q) ^ col_lo) << 4;
      const U4 v0 = *reinterpret_cast<const U4*>(lo + at), v1 = *reinterpret_cast<const U4*>(lo + 8 * 128 + at);
      const uint32_t w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        __half2 h0[4], h1[4];
        dequant8(w0[w], sc[c][0], h0);
        dequant8(w1[w], sc[c][1], h1);
        const uint32_t* f0 = reinterpret_cast<const uint32_t*>(h0);
        const uint32_t* f1 = reinterpret_cast<const uint32_t*>(h1);
#pragma unroll
        for (int r = 0; r < MR; ++r) mma16816(acc[r], f0[0], f1[0], f0[1], f1[1], xf[c][r][w][0], xf[c][r][w][1]);
#pragma unroll
        for (int r = 0; r < MR; ++r) mma16816(acc[r], f0[2], f1[2], f0[3], f1[3], xf[c][r][w][2], xf[c][r][w][3]);
      }
    }
    __syncwarp();  // every lane has read the slot
    if (lane == 0 && ok && pass + depth < passes) issue(slot.slot, pass + depth);
    slot.advance(depth);
    if (ok) ok = mbar_wait(part_empty + pb.slot, pb.parity ^ 1u);  // a fresh barrier passes: nothing is parked yet
    float4* mine = part + (pb.slot * plan.cta_slices + ws) * MR * 32 + lane;
#pragma unroll
    for (int r = 0; r < MR; ++r) mine[r * 32] = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    __syncwarp();
    if (lane == 0) mbar_arrive_cta(part_full + pb.slot);
    pb.advance(kRxParts);
    if (pass > 0) {
      if (ws == turn) reduce(pass - 1);
      if (++turn == live_slices) turn = 0;
    }
  }
  if (passes > 0 && ws == turn) reduce(passes - 1);
  if (plan.ranks > 1) {
    __syncwarp();
    cg::this_cluster().barrier_arrive();  // release: the sums pushed to other ranks
    cg::this_cluster().barrier_wait();
    const int all = static_cast<int>(static_cast<int64_t>(set_id + 1) * plan.groups / plan.total_sets) - g0;
    for (int p = warp * plan.ranks + rank; p < all; p += warps * plan.ranks) {
      const float4* src = parked + (p / plan.ranks) * plan.ranks * MR * 32 + lane;
      float4 sum[MR];
#pragma unroll
      for (int r = 0; r < MR; ++r) sum[r] = src[r * 32];
      for (int s = 1; s < plan.ranks; ++s)
#pragma unroll
        for (int r = 0; r < MR; ++r) {
          const float4 v = src[(s * MR + r) * 32];
          sum[r].x = __fadd_rn(sum[r].x, v.x), sum[r].y = __fadd_rn(sum[r].y, v.y);
          sum[r].z = __fadd_rn(sum[r].z, v.z), sum[r].w = __fadd_rn(sum[r].w, v.w);
        }
      store(p, sum);
    }
  }
  if (!ok && lane == 0) atomicOr(&g_w4_fault, 2u);
}

// Clusters of `ranks` such CTAs (one per SM) that are resident at once on the current device.
int rx_resident_clusters(int ranks) {  // the same for every variant: one CTA per SM
  static std::atomic<int> known[64][9];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = known[dev][ranks].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaFuncSetAttribute(w4a16_rx_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRxSmem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sm_count() / ranks, ranks);
  cfg.blockDim = dim3(kRxWarps * 32);
  cfg.dynamicSmemBytes = kRxSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = static_cast<unsigned>(ranks), attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, w4a16_rx_kernel<2>, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    return 0;
  }
  known[dev][ranks].store(n, std::memory_order_relaxed);
  return n;
}

// XDK_ERR_LIMIT: K > 32768, or more columns than the resident clusters take in one wave when `one_wave` asks for it.
template <int MR>
int launch_rx(const W4Args& a, bool dependent, bool one_wave, cudaStream_t stream) {
  RxPlan p = {};
  cudaError_t err = cudaFuncSetAttribute(w4a16_rx_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRxSmem);
  if (err != cudaSuccess) return note_launch(err);
  const int sms = sm_count();
  p.slices = (a.k + kRxSliceK - 1) / kRxSliceK;
  p.groups = (a.n + 15) / 16;
  p.ranks = (p.slices + kRxWarps - 1) / kRxWarps;
  // few columns: more CTAs share K, down to four slices each, while they all fit
  while (p.ranks * 2 <= 8 && p.groups * p.ranks * 2 <= sms && p.slices >= p.ranks * 8) p.ranks *= 2;
  if (p.ranks > 8) return XDK_ERR_LIMIT;
  p.cta_slices = (p.slices + p.ranks - 1) / p.ranks;
  p.ranks = (p.slices + p.cta_slices - 1) / p.cta_slices;
  p.sets = 1;
  int passes;
  if (p.ranks == 1) {
    p.sets = min(kRxWarps / p.cta_slices, (p.groups + sms - 1) / sms);
    p.total_sets = min(sms, (p.groups + p.sets - 1) / p.sets) * p.sets;
  } else {
    int clusters = rx_resident_clusters(p.ranks);
    if (clusters < 1) return XDK_ERR_LIMIT;
    clusters = min(clusters, p.groups);
    p.total_sets = max(clusters, (p.groups + kRxMaxPasses - 1) / kRxMaxPasses);
    if (one_wave && p.total_sets > clusters) return XDK_ERR_LIMIT;
  }
  passes = (p.groups + p.total_sets - 1) / p.total_sets;
  p.parked = p.ranks > 1 ? (passes + p.ranks - 1) / p.ranks : 0;
  const int warps = p.cta_slices * p.sets;
  const int fixed = (kRxParts * warps + p.parked * (p.ranks > 1 ? p.ranks : 0)) * MR * 512 +
                    (warps * kRxMaxDepth + p.sets * 2 * kRxParts) * static_cast<int>(sizeof(uint64_t));
  p.depth = min(min(kRxMaxDepth, passes), (kRxSmem - fixed) / (warps * kRxStage));
  if (p.depth < 1) return XDK_ERR_LIMIT;
  const size_t smem = static_cast<size_t>(fixed) + static_cast<size_t>(warps) * p.depth * kRxStage;
  CUtensorMap wmap;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(a.k / 8), static_cast<cuuint64_t>(a.n)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(a.k / 2)};
  const cuuint32_t box[2] = {kRxSliceK / 8, 16};
  static_assert(kRxSliceK / 2 == 128, "the box of codes is one 128-byte swizzle span wide");
  if (!encode_tiled(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, a.packed, dims, strides, box, true)) return XDK_ERR_LAUNCH;
  return launch_opts(w4a16_rx_kernel<MR>, dim3(p.total_sets / p.sets, p.ranks), dim3(warps * 32), smem, stream,
                     static_cast<unsigned>(p.ranks), dependent, a, p, wmap);
}

template <int MT, int CW>
int launch_simt(W4Args a, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(MT) * a.k * sizeof(__half);
  auto kernel = w4a16_simt_kernel<MT, CW>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return note_launch(err);
  a.col_groups = (a.n + kWarps * CW - 1) / (kWarps * CW);
  const int max_ctas = 4 * sm_count();
  a.groups_per_cta = (a.col_groups + max_ctas - 1) / max_ctas;
  const int ctas = (a.col_groups + a.groups_per_cta - 1) / a.groups_per_cta;
  return launch(kernel, dim3(ctas), dim3(kThreads), smem, stream, 1u, a);
}

}  // namespace
}  // namespace xdk

namespace xdk {
unsigned w4a16_fault_word() {
  unsigned v = 0;
  if (cudaMemcpyFromSymbol(&v, g_w4_fault, sizeof(v)) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0x80000000u;
  }
  return v;
}
}  // namespace xdk

extern "C" int xdk_w4a16(const void* x, const uint8_t* packed, const void* scales, const void* bias, void* y,
                         int64_t m, int64_t k, int64_t n, int group_size, void* stream) {
  return xdk_w4a16_v2(x, packed, scales, bias, y, m, k, n, group_size, 0u, stream);
}

extern "C" int xdk_w4a16_v2(const void* x, const uint8_t* packed, const void* scales, const void* bias, void* y,
                            int64_t m, int64_t k, int64_t n, int group_size, unsigned flags, void* stream) {
  if (!y || n < 1) return XDK_ERR_ARG;
  xdk_peer_out one = {};
  one.ptr[0] = y, one.world = 1, one.ld = n, one.col0 = 0;
  return xdk_w4a16_peer(x, packed, scales, bias, &one, m, k, n, group_size, flags, stream);
}

extern "C" int xdk_w4a16_peer(const void* x, const uint8_t* packed, const void* scales, const void* bias,
                              const xdk_peer_out* y_out, int64_t m, int64_t k, int64_t n, int group_size, unsigned flags,
                              void* stream) {
  using namespace xdk;
  if (flags & ~XDK_DEPENDENT_LAUNCH) return XDK_ERR_ARG;
  PeerOut out;
  if (int st = make_out(y_out, nullptr, n, &out)) return st;
  void* y = out.ptr[0];
  const bool plain = out.world == 1 && out.ld == n && out.col0 == 0;  // the kernels of this file write y[m][n] only
  if (!x || !packed || !scales || !y) return XDK_ERR_ARG;
  if (m < 1 || m > 16 || k < 1 || n < 1) return XDK_ERR_ARG;
  if (!(group_size == 32 || group_size == 64 || group_size == 128 || group_size == 256)) return XDK_ERR_ARG;
  if (k >= (1LL << 31) || n >= (1LL << 31) || m * n >= (1LL << 31) || n * ((k + 1) / 2) >= (1LL << 31))
    return XDK_ERR_LIMIT;
  if (int st = require_sm100()) return st;
  W4Args a;
  a.x = static_cast<const __half*>(x);
  a.packed = packed;
  a.scales = static_cast<const __half*>(scales);
  a.bias = static_cast<const __half*>(bias);
  a.y = static_cast<__half*>(y);
  a.m = static_cast<int>(m), a.k = static_cast<int>(k), a.n = static_cast<int>(n);
  a.group = group_size;
  a.groups = static_cast<int>((k + group_size - 1) / group_size);
  a.col_groups = a.groups_per_cta = 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool dependent = (flags & XDK_DEPENDENT_LAUNCH) != 0;
  a.out = out;
  const bool vec_ok = k % 32 == 0 && aligned16(packed) && aligned16(x);  // 16-byte vectors of 32 codes
  // Who takes what, by measurement (us; K = 4096 unless said):
  //  * M <= 2, K a multiple of 1024, and M <= 8 while x leaves room for two CTAs per SM: the direct-load mma.sync kernel
  //    (N = 4096 6.0 / 6.5 / 7.3 at M = 1 / 4 / 8, N = 14336 14.7 / 15.7 / 16.4; the kernel that keeps x in registers 7.6 /
  //    7.9 / 8.5 and 16.4 / 17.2 / 17.7; the SIMT kernel 16.3 at M = 1, N = 14336).
  //    A larger x too where every SM has one group of columns at most anyway and most have one (M = 8, K = 7168, N = 2048
  //    8.6 / 9.3, N = 2368 8.7 / 9.5, but N = 1024 8.1 / 7.4; K = 9216, N = 2048 10.6 / 10.2).
  //  * M >= 9, figures for 16, the tcgen05 kernel / the one that keeps x in registers, by the 32-column units of the former's
  //    busiest CTA.  K up to 4096: the former where its CTAs walk whole strips of three or four units, or two (N = 14336 17.6 / 20.8,
  //    N = 18944 17.9 / 22.0, N = 8192 13.9 / 14.5; but one unit, K split over the lane quarters, N = 2048 10.7 / 7.7, a strip and a
  //    narrow rest N = 23680 24.5 / 23.8, N = 33152 30.4 / 29.5; from K = 2048 to 4096 the former there too, K = 3072, N = 33112 24.0 / 24.8 at M = 9).
  //    K up to 12288: the former from two units on (K = 5120, N = 9472 15.6 / 18.7, N = 23680 28.3 / 32.5; K = 10240, N = 9472 24.7 / 29.2,
  //    N = 33112 64 / 77; K = 12288, N = 18904 41.1 / 49.5; K = 8192, where the latter's warps are all busy, either way: N = 9472 22.1 / 23.4,
  //    N = 23680 44 / 40, N = 37888 56 / 58), and for a wide single one (N = 4696, K = 5120 12.4 / 13.0, 10240 18.8 / 20.8, but 8192 17.0 / 16.2;
  //    N = 3584, K = 5120 12.3 / 12.3, 10240 18.4 / 17.0, N = 2400 18.1 / 14.8).
  //    Longer K: the latter (K = 14336, N = 4096 34.0 / 22.6, N = 14208 66 / 49, N = 33152 133 / 103; K = 20480, N = 9432 75 / 44), as long as the
  //    resident clusters take all columns in one wave (K = 14336, N = 37888 150 / 205).
  //    Shapes the tcgen05 kernel declines: the latter (K = 2304, N = 8192 15.5 / 11.8 with the stream kernel, K = 896, N = 23640 11.9 / 11.6),
  //    but for a short K on a middling width (K = 384, N = 9432 4.5 / 5.0, K = 896 6.4 / 7.6, N = 4096 4.7 / 5.2).
  //    Every strided or multi-rank output: the tcgen05 kernel.
  //  * 3 <= M <= 8 otherwise: the kernel that keeps x in registers.  M = 8: x too large for two CTAs (K = 14336, N = 4096 18.9, tcgen05
  //    27.9, K = 7168, N = 20480 29.6 / 39.9), K = 2304, N = 8192 9.8 / 14.1.  But the tcgen05 kernel for strips of four units of a K between 8192
  //    and 12288 (M = 8, K = 10240, N = 18904 34.1 / 40.4), and the direct-load one, x permitting, for more columns than one wave takes (M = 3,
  //    K = 20480, N = 28672 135 / 166).
  // XDK_W4A16_MMA=0 and XDK_W4A16_UMMA=0 / 1 take the first kernel out, and the second out or in wherever it can run
  // (comparison runs).
  static const bool mma_env = !(getenv("XDK_W4A16_MMA") && getenv("XDK_W4A16_MMA")[0] == '0');
  static const int umma_env = getenv("XDK_W4A16_UMMA") ? (getenv("XDK_W4A16_UMMA")[0] == '1' ? 1 : 0) : -1;
  const size_t x_bytes = static_cast<size_t>(m) * (static_cast<size_t>(k) * 2 + 16);
  const int64_t groups = (n + 15) / 16, sms = sm_count();
  const bool one_each = groups <= sms && (groups * 8 > sms * 7 || (groups * 4 > sms * 3 && k <= 8192));  // group of 16 columns on most SMs
  if (mma_env && plain && vec_ok && k % 1024 == 0 &&
      (m <= 2 || (m <= 8 && one_each) ? x_bytes <= 160 * 1024 : m <= 8 && x_bytes <= 104 * 1024)) {
    // Three CTAs per SM where that saves a pass over the column groups, or K is short (us with two / three, M = 1: K = 4096,
    // N = 6144 9.3 / 7.7, N = 20480 17.6 / 16.0, N = 28672 23.3 / 22.8, N = 8192 -- two passes either way -- 9.7 / 10.6; K = 2048,
    // N = 8192 6.6 / 6.3, N = 28672 16.1 / 13.8; M = 4 alike).  A larger x leaves the L1 cache too little for the scales.
    const int64_t two = 2 * sms, three = 3 * sms;
    if (x_bytes <= 40 * 1024 && k <= 4096 && groups > two && (k <= 2048 || (groups + three - 1) / three < (groups + two - 1) / two))
      return launch_mma<2, 3>(a, dependent, s);
    return launch_mma<4, 2>(a, dependent, s);
  }
  const bool umma_ok = vec_ok && k % 256 == 0 && group_size >= 64 && a.groups <= 256 && a.groups % 8 == 0 && aligned16(scales);
  const int64_t units = ((n + 31) / 32 + sms - 1) / sms;  // 32-column units of the tcgen05 kernel's busiest CTA
  const bool whole = k <= 4096    ? units % 4 == 0 || units == 2 || units == 3 || (units > 4 && k >= 2048 && k < 4096)
                     : k <= 12288 ? units >= 2 || (k != 8192 && n >= (k > 10240 ? 4097 : 4096))
                                  : false;
  const bool umma_first = !plain || umma_env == 1 || (umma_env != 0 && (m > 8 ? whole : units % 4 == 0 && k > 8192 && k <= 12288));
  const bool stream_first = m > 8 && k < 1024 && n >= (k <= 128 ? 1 : (k <= 384 ? 2048 : 3072)) && n <= 4 * 32 * sms;
  if (plain && vec_ok && k % 128 == 0 && m >= 3 && !(umma_ok && umma_first) && !stream_first) {
    const bool umma_next = umma_ok && umma_env != 0;
    const int st = m > 8 ? launch_rx<2>(a, dependent, umma_next, s) : launch_rx<1>(a, dependent, umma_next, s);
    if (st != XDK_ERR_LIMIT) return st;  // the kernels below
    if (mma_env && m <= 8 && k % 1024 == 0 && x_bytes <= 160 * 1024) return launch_mma<4, 2>(a, dependent, s);
  }
  if (umma_ok && (!plain || (umma_env != 0 && (m >= 3 || (m == 2 && k * n >= (32LL << 20)))))) {
    const int st = launch_umma(a, dependent, s);
    if (st != XDK_ERR_LIMIT || !plain) return st;
  }
  if (!plain) return XDK_ERR_LIMIT;  // a strided or multi-rank destination needs the tcgen05 kernel's shape
  if (vec_ok && k % 128 == 0 && m >= 3) return m > 8 ? launch_stream<16>(a, s) : launch_stream<8>(a, s);
  // the SIMT kernel keeps all rows of x (padded to a power of two) in shared memory
  const int mt = m == 1 ? 1 : (m == 2 ? 2 : (m <= 4 ? 4 : (m <= 8 ? 8 : 16)));
  if (vec_ok && static_cast<int64_t>(mt) * k * 2 <= 200 * 1024) {
    if (mt == 1) return launch_simt<1, 2>(a, s);
    if (mt == 2) return launch_simt<2, 2>(a, s);
    if (mt == 4) return launch_simt<4, 2>(a, s);
    if (mt == 8) return launch_simt<8, 1>(a, s);
    return launch_simt<16, 1>(a, s);
  }
  return launch(w4a16_generic_kernel, dim3(static_cast<unsigned>((n + kWarps - 1) / kWarps)), dim3(kThreads), 0, s, 1u,
                a);
}
