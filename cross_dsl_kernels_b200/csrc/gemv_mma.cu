// FP32 projection of more than 16 rows and a long K on mma.sync (tf32), with the accuracy of FP32 FMAs.
//
// y[M, N] = x[M, K] . W + bias.  Both operands are split into two TF32 numbers, v = hi + lo (hi = v rounded to
// TF32's 11 significant bits, lo = v - hi, exact and of either sign), and the product is hi.hi + hi.lo + lo.hi.  The tensor
// core truncates as it accumulates, so an accumulator only takes the six MMAs of 16 k, the small products first, before it
// is added to an FP32 sum with rounding.  What the products lose (the last bit of an operand, lo.lo, the truncation) is about
// 1e-7 at any K, the sum's own error grows with K as that of FMAs does: so the kernel only takes shapes where it is no less
// accurate than the FP32-FMA kernels that had them.  Relative L2 error against 64 bits, e-7, here / FMAs, normal operands:
//   [K, N]  K = 128 1.17 / 0.93, 1024 1.29 / 1.25, 2048 1.40 / 1.31, 4096 1.57 / 1.65, 8192 1.87 / 2.18, 14336 2.25 / 2.80
//   [N, K]  N <= 2368, where FMAs split K four ways or eight: 4096 1.58 / 1.27, 14336 2.26 / 2.04
//           wider, two ways: 1024 1.29 / 1.00, 2048 1.39 / 1.22, 4096 1.57 / 1.59, 8192 1.87 / 2.14, 14336 2.25 / 2.77
// (With hi cut off instead of rounded 5.7 at K = 4096, in another order of the products 1.9.)  Operands of one sign: 0.87 at
// K = 4096, 1.01 at 14336; FMAs 0.45 .. 0.6.
// An infinity does not split (lo = inf - inf): a pass with a sum that is not finite is done once more, with a split that carries
// infinities and NaNs in its leading product alone (us for M = 64, K = N = 4096 and a NaN in every row of x, [K, N] / [N, K]: 224 / 221;
// with a thread that went through K for each such output 1669 / 4004).
//
// Times, us, against the kernels that had the shapes before (K = 4096 unless said): M = 64, N = 4096 57 .. 60 against 89 .. 94
// (FP32 FMAs of a 16 x 4 register tile, W walked once per 16 rows), M = 64, N = 14336 200 / 266 .. 281, M = 64, K = 14336,
// N = 4096 174 .. 187 / 267 .. 290; M = 592 426 / 765, M = 1200 1137 / 1541, M = 5000 3903 / 6396 (N = 4096, [K, N]; [N, K] alike).  Narrow [K, N]:
// N = 768, M = 17 16 / 17, M = 64 21 / 31, M = 1200 283 / 524, but N = 512, M = 17 .. 48 17 .. 22 / 14 .. 17, N = 256, M = 64 18 / 12: a
// block of rows has too few column groups there.  What bounds it: with one CTA of eight warps an SM,
// latency -- the tensor pipe would need 22 us for M = 64, N = 4096.
//
// The loop is built round the stream of W.  A CTA (one per SM) owns up to 16 rows and 16 G columns over all of its K; its
// eight warps take the 16-k steps in turn and keep the sums of all the CTA's columns in registers, so nothing is exchanged
// until the end.  A warp copies its own steps into a ring of its own with cp.async -- no barrier in the loop -- and an x
// fragment, read from global memory a step ahead and split once, serves all column groups of the step.  16 columns of W are
// the 16 rows of an MMA, 8 rows of x its columns; a step is two MMAs deep, and which k a fragment slot stands for is free as
// long as both operands agree:
//   W as [N, K]: a lane's four k of a column are 16 consecutive bytes, slots (4 q, 4 q + 1) and (4 q + 2, 4 q + 3)
//   W as [K, N]: a lane's two columns are neighbours in a k row, slots (q, q + 4) and (q + 8, q + 12)
// The warps' sums meet in shared memory in warp order.  A narrow matrix splits K over the CTAs of a cluster, whose sums
// are added in rank order through distributed shared memory.  Deterministic.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace xdk {
namespace {

constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kStepK = 16;

struct MmaArgs {
  const float* x;
  const float* w;
  const float* bias;
  PeerOut out;
  int m, k, n;
  int groups;  // of 16 columns
  int k_rank;  // k per CTA of a cluster (a multiple of kStepK)
  int block0;  // first block of 16 rows of this launch
};

struct Split {
  uint32_t hi, lo, lead;  // lead: the factor of the leading product, hi but for what does not split
};
__device__ __forceinline__ Split split_tf32(float v) {
  const uint32_t hi = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
  return Split{hi, __float_as_uint(__fsub_rn(v, __uint_as_float(hi))), hi};
}
// The same parts of what splits.  An infinity or a NaN is in the leading product only, whose outcome is then that of the plain
// product; a value that would round up to infinity is cut off instead, and one that would round to zero is kept apart from it.
__device__ __forceinline__ Split split_any(float v) {
  const uint32_t bits = __float_as_uint(v), size = bits & 0x7fffffffu;
  if (size >= 0x7f800000u) return Split{0u, 0u, size > 0x7f800000u ? 0x7fffffffu : bits};
  uint32_t hi = (bits + 0x1000u) & 0xffffe000u;
  if ((hi & 0x7fffffffu) == 0x7f800000u) hi = bits & 0xffffe000u;
  if ((hi & 0x7fffffffu) == 0u && size != 0u) hi |= 0x2000u;
  return Split{hi, __float_as_uint(__fsub_rn(v, __uint_as_float(hi))), hi};
}
template <bool ANY>
__device__ __forceinline__ Split split(float v) {
  return ANY ? split_any(v) : split_tf32(v);
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool NK, int G>
struct Ring {  // G: column groups a pass can hold
  static constexpr int kPitch = NK ? kStepK : G * 16 + 8;                        // floats per staged row: a column's 16 k, or a k row
  static constexpr int kStage = (NK ? G * 16 : kStepK) * kPitch;                 // floats
  static constexpr int kDepth = G <= 2 ? 8 : (G <= 4 ? 5 : 3);
  static constexpr int kSumPitch = G * 16;
  static constexpr size_t sum_bytes(int mr) { return static_cast<size_t>(kWarps) * 8 * mr * kSumPitch * 4; }
  static constexpr size_t bytes(int mr) {
    const size_t ring = static_cast<size_t>(kWarps) * kDepth * kStage * 4;
    return ring > sum_bytes(mr) ? ring : sum_bytes(mr);
  }
};

template <bool NK, int MR, int G>
__global__ void __launch_bounds__(kThreads, 1)
gemv_mma_kernel(MmaArgs a) {
  using R = Ring<NK, G>;
  constexpr int D = R::kDepth;
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = lane >> 2, q = lane & 3;
  const int ranks = gridDim.y, rank = blockIdx.y;
  const int row0 = (a.block0 + blockIdx.z) * 16, rows = min(16, a.m - row0);  // blocks of rows: W comes from L2 for all but one
  const int k_begin = rank * a.k_rank, k_end = min(a.k, k_begin + a.k_rank);
  const int all_steps = k_begin < k_end ? (k_end - k_begin + kStepK - 1) / kStepK : 0;
  const int steps = all_steps > warp ? (all_steps - warp + kWarps - 1) / kWarps : 0;  // of this warp: warp, warp + 8, ...
  const int first = static_cast<int>(static_cast<int64_t>(blockIdx.x) * a.groups / gridDim.x);
  const int count = static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * a.groups / gridDim.x) - first;
  float* ring = smem + warp * D * R::kStage;

  pdl_launch_dependents();
  pdl_wait();
  // every CTA of a cluster runs the same passes: the deal of the groups does not depend on the rank
  const int passes = (count + G - 1) / G;
  for (int pass = 0; pass < passes; ++pass) {
    const int g0 = first + static_cast<int>(static_cast<int64_t>(pass) * count / passes);
    const int ng = first + static_cast<int>(static_cast<int64_t>(pass + 1) * count / passes) - g0;
    const int col0 = g0 * 16;

    auto fetch = [&](int s) {  // this warp's step s; columns past N and k past the end become zeros
      if (s < steps) {
        float* dst = ring + (s % D) * R::kStage;
        const int k0 = k_begin + (s * kWarps + warp) * kStepK;
        if (NK) {
          const int c = lane >> 2, kk = (lane & 3) * 4;
          const float* src = a.w + static_cast<size_t>(col0 + c) * a.k + k0 + kk;
#pragma unroll
          for (int j = 0; j < 2 * G; ++j) {  // eight columns at a time
            if (j >= 2 * ng) break;
            const bool live = col0 + j * 8 + c < a.n && k0 + kk < k_end;
            cp_async16_or_zero(dst + (j * 8 + c) * R::kPitch + kk, live ? src + static_cast<size_t>(j) * 8 * a.k : a.w, live);
          }
        } else {
          constexpr int kRows = G <= 2 ? 4 : (G <= 4 ? 2 : 1);  // k rows at a time
          const int r = lane / (32 / kRows), c = (lane % (32 / kRows)) * 4;
          const bool col_live = c < ng * 16 && col0 + c < a.n;
          const float* src = a.w + static_cast<size_t>(k0 + r) * a.n + col0 + c;
          if (c < ng * 16) {
#pragma unroll
            for (int j = 0; j < kStepK / kRows; ++j) {
              const bool live = col_live && k0 + j * kRows + r < k_end;
              cp_async16_or_zero(dst + (j * kRows + r) * R::kPitch + c, live ? src + static_cast<size_t>(j) * kRows * a.n : a.w, live);
            }
          }
        }
      }
      cp_async_commit();
    };
    // x of a step: rows i and i + 8, this lane's four k in slot order; rows past M and k past the end are zeros
    auto fetch_x = [&](int s, float (&v)[MR][4]) {
      const int k0 = k_begin + (s * kWarps + warp) * kStepK;
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        const bool row_live = s < steps && r * 8 + i < rows;
        const float* src = a.x + static_cast<size_t>(row_live ? row0 + r * 8 + i : 0) * a.k;
        if (NK) {
          float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (row_live && k0 + q * 4 < k_end) t = *reinterpret_cast<const float4*>(src + k0 + q * 4);
          v[r][0] = t.x, v[r][1] = t.y, v[r][2] = t.z, v[r][3] = t.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) v[r][e] = row_live && k0 + q + e * 4 < k_end ? src[k0 + q + e * 4] : 0.0f;
        }
      }
    };

    float sum[G][MR][4];
    auto multiply = [&](auto any) {  // any: operands that do not split
      constexpr bool ANY = decltype(any)::value;
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int r = 0; r < MR; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) sum[g][r][e] = 0.0f;
      float xn[MR][4];
      for (int s = 0; s < D - 1; ++s) fetch(s);
      fetch_x(0, xn);
      for (int s = 0; s < steps; ++s) {
        Split xs[MR][4];
#pragma unroll
        for (int r = 0; r < MR; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) xs[r][e] = split<ANY>(xn[r][e]);
        cp_async_wait<D - 2>();
        __syncwarp();  // the step has landed for every lane, and every lane has read the slot that is refilled now
        fetch(s + D - 1);
        fetch_x(s + 1, xn);
        const float* tile = ring + (s % D) * R::kStage;
#pragma unroll
        for (int g = 0; g < G; g += 2) {  // two groups at a time: twice the independent MMA chains
          if (g >= ng) break;             // (an odd last group is paired with columns whose sums are not stored)
          float w[2][2][4];               // [group][column i, column i + 8 of the MMA][slot]
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (NK) {
              const float4 t0 = *reinterpret_cast<const float4*>(tile + ((g + h) * 16 + i) * R::kPitch + q * 4);
              const float4 t1 = *reinterpret_cast<const float4*>(tile + ((g + h) * 16 + i + 8) * R::kPitch + q * 4);
              w[h][0][0] = t0.x, w[h][0][1] = t0.y, w[h][0][2] = t0.z, w[h][0][3] = t0.w;
              w[h][1][0] = t1.x, w[h][1][1] = t1.y, w[h][1][2] = t1.z, w[h][1][3] = t1.w;
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 t = *reinterpret_cast<const float2*>(tile + (q + e * 4) * R::kPitch + (g + h) * 16 + i * 2);
                w[h][0][e] = t.x, w[h][1][e] = t.y;
              }
            }
          }
          float acc[2][MR][4];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int r = 0; r < MR; ++r)
#pragma unroll
              for (int e = 0; e < 4; ++e) acc[h][r][e] = 0.0f;
          uint32_t hi[2][2][4], lo[2][2][4], lead[2][2][4];  // [MMA j: slots 2 j and 2 j + 1][group][fragment register]
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const Split v = split<ANY>(w[h][e & 1][2 * j + (e >> 1)]);
                hi[j][h][e] = v.hi, lo[j][h][e] = v.lo, lead[j][h][e] = v.lead;
              }
          // the small products first: what the tensor core truncates off an accumulator then only counts for the last two
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int r = 0; r < MR; ++r)
#pragma unroll
              for (int h = 0; h < 2; ++h) mma_tf32(acc[h][r], lo[j][h], xs[r][2 * j].hi, xs[r][2 * j + 1].hi);
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int r = 0; r < MR; ++r)
#pragma unroll
              for (int h = 0; h < 2; ++h) mma_tf32(acc[h][r], hi[j][h], xs[r][2 * j].lo, xs[r][2 * j + 1].lo);
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int r = 0; r < MR; ++r)
#pragma unroll
              for (int h = 0; h < 2; ++h) mma_tf32(acc[h][r], lead[j][h], xs[r][2 * j].lead, xs[r][2 * j + 1].lead);
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int r = 0; r < MR; ++r)
#pragma unroll
              for (int e = 0; e < 4; ++e) sum[g + h][r][e] = __fadd_rn(sum[g + h][r][e], acc[h][r][e]);
        }
      }
    };
    const int cols = ng * 16, outs = rows * cols;
    for (bool again = false;;) {  // once more if a sum is not finite
      if (again) multiply(std::true_type{});
      else multiply(std::false_type{});
      cp_async_wait<0>();
      __syncthreads();  // the rings are done with: their memory takes the sums, [warp][row][column of the pass]
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g >= ng) break;
#pragma unroll
        for (int r = 0; r < MR; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // rows 2 q + (e & 1) of x, column i (e < 2) or i + 8 of the MMA
            const int row = r * 8 + q * 2 + (e & 1);
            const int col = g * 16 + (NK ? i + (e >> 1) * 8 : i * 2 + (e >> 1));
            smem[(warp * 8 * MR + row) * R::kSumPitch + col] = sum[g][r][e];
          }
      }
      __syncthreads();
      bool bad = false;
      for (int o = threadIdx.x; o < outs; o += kThreads) {
        const int row = o / cols, at = row * R::kSumPitch + (o - row * cols);
        float v = smem[at];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) v = __fadd_rn(v, smem[w * 8 * MR * R::kSumPitch + at]);
        smem[at] = v;
        bad |= !isfinite(v);
      }
      if (!__syncthreads_or(bad) || again) break;
      again = true;
    }
    if (ranks > 1) cg::this_cluster().sync();  // every rank's sums stand in its shared memory
    for (int o = threadIdx.x + rank * kThreads; o < outs; o += kThreads * ranks) {
      const int row = o / cols, c = o - row * cols;
      if (col0 + c >= a.n) continue;
      float* at = smem + row * R::kSumPitch + c;
      float v = ranks > 1 ? *cg::this_cluster().map_shared_rank(at, 0) : *at;
      for (int p = 1; p < ranks; ++p) v = __fadd_rn(v, *cg::this_cluster().map_shared_rank(at, p));  // rank order
      if (a.bias) v = __fadd_rn(v, a.bias[col0 + c]);
      peer_store(a.out, row0 + row, col0 + c, v);
    }
    if (ranks > 1) cg::this_cluster().sync();  // nobody leaves, or refills, what another rank still reads
    else __syncthreads();
  }
}

template <bool NK, int MR, int G>
int launch_mma(const MmaArgs& a, int ctas, int ranks, int blocks, cudaStream_t stream) {
  constexpr size_t smem = Ring<NK, G>::bytes(MR);
  static_assert(smem <= 227 * 1024, "one CTA per SM");
  auto kernel = gemv_mma_kernel<NK, MR, G>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return note_launch(err);
  return launch_opts(kernel, dim3(ctas, ranks, blocks), dim3(kThreads), smem, stream, static_cast<unsigned>(ranks),
                     (call_flags() & XDK_DEPENDENT_LAUNCH) != 0, a);
}
template <bool NK, int MR>
int launch_mma(const MmaArgs& a, int ctas, int ranks, int blocks, cudaStream_t stream) {
  const int per = (a.groups + ctas - 1) / ctas;  // column groups of the busiest CTA
  if (per <= 2) return launch_mma<NK, MR, 2>(a, ctas, ranks, blocks, stream);
  if (per <= 4) return launch_mma<NK, MR, 4>(a, ctas, ranks, blocks, stream);
  return launch_mma<NK, MR, 8>(a, ctas, ranks, blocks, stream);
}

}  // namespace

bool gemv_mma_eligible(const float* x, const float* w, int64_t m, int64_t k, int64_t n, bool nk) {
  // the least K, and for [N, K] the least N, at which the error is no larger than that of FMAs, and for [K, N] the least N at
  // which it is no slower at any M (figures above)
  if (k < 4096 || n <= (nk ? 2368 : 764)) return false;
  return m >= 1 && m <= 16 * 65535LL && k % 4 == 0 && (nk || n % 4 == 0) && aligned16(x) && aligned16(w) && k < (1 << 30) && n < (1 << 30);
}

int launch_gemv_mma(const float* x, const float* w, const float* bias, const PeerOut& y, int m, int k, int n, bool nk,
                    cudaStream_t stream) {
  MmaArgs a;
  a.x = x, a.w = w, a.bias = bias, a.out = y, a.m = m, a.k = k, a.n = n;
  a.groups = (n + 15) / 16;
  const int sms = sm_count();
  // Few column groups: two CTAs of a cluster share K.  By N alone: the order of the sums, and with it the bits of a row, do not
  // depend on how many rows there are.
  const int ranks = a.groups * 2 <= sms ? 2 : 1;
  a.k_rank = ((k + ranks - 1) / ranks + kStepK - 1) / kStepK * kStepK;
  // A block of 16 rows gets an equal share of the SMs, in whole CTAs.  Many rows go in several launches of blocks that have at
  // least four CTAs each: the fewer there are, the more SMs the rounding leaves idle (1200 rows in one launch had 75 CTAs).
  const int blocks = (m + 15) / 16, most = sms > 4 ? sms / 4 : 1;
  const int launches = (blocks + most - 1) / most;
  for (int i = 0; i < launches; ++i) {
    a.block0 = static_cast<int>(static_cast<int64_t>(i) * blocks / launches);
    const int count = static_cast<int>(static_cast<int64_t>(i + 1) * blocks / launches) - a.block0;
    const int share = sms / (count * ranks), ctas = a.groups < share ? a.groups : (share > 1 ? share : 1);
    const int st = nk ? launch_mma<true, 2>(a, ctas, ranks, count, stream) : launch_mma<false, 2>(a, ctas, ranks, count, stream);
    if (st != XDK_OK) return st;
  }
  return XDK_OK;
}

}  // namespace xdk
