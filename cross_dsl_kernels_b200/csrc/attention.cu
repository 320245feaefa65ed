// Paged decode attention: one query token per sequence against the K/V cache the append kernel writes.
//
//   out[t][h] = sum_j softmax_j( scale * q[t][h] . K[seq(t)][j][h / G] ) * V[seq(t)][j][h / G],   j = 0 .. positions[t]
//
// (the token's own K/V are in the cache already: the append runs first), G = q_heads / kv_heads query heads
// sharing one KV head.  Pages are found through page_table exactly as the append kernel finds them, in the NHD
// ([page][offset][head][dim]) or HND ([page][head][offset][dim]) cache layout.  Not part of upstream, which stops
// at the append; it is the op that reads what this library's append writes.
//
// HBM-bound: every K and V row of the context is read once (2 * dim * sizeof(T) bytes per position and KV head)
// and used for all G heads of its group.  Work is cut as (context split, KV head, token): a CTA of four warps walks
// its slice of the context in tiles of 32 positions per warp.
//   scores : the warp copies the tile's 32 K rows into shared memory with cp.async, two rows per instruction (a lane
//            reading its own row straight from global memory touches 32 lines per instruction and caps the kernel at
//            a third of the HBM rate); then a lane owns one position: it reads that row from shared memory (row pitch
//            padded by 16 bytes: conflict-free) and accumulates the G dot products against q (FP32 in shared
//            memory, broadcast reads); no shuffles.
//   softmax: per warp and head, running maximum and sum (online softmax) -- one warp max per tile and head.
//   values : lanes turn to own dim/32 dims each; the tile's probabilities and row addresses go through shared
//            memory (one broadcast read per position); the V rows were staged together with the K rows (head sizes
//            whose tiles would leave too few CTAs per SM read them straight from global memory instead).
// 16-bit caches take the tensor-core variant further down: same staging and merges, both contractions as mma tiles.
// The four warps' partial (max, sum, accumulator) are merged in shared memory.  Who computes what: without scratch, or for
// short contexts, the slices of one (token, KV head) form a thread-block cluster and are merged in rank order through
// distributed shared memory; with scratch the tiles of the whole batch are dealt evenly to the CTAs (below) and a second
// launch merges what several of them hold of an item.  Either way the result is deterministic.
#include <cooperative_groups.h>
#include <math.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace xdk {
namespace {

constexpr int kAttnWarps = 4;
constexpr int kAttnThreads = kAttnWarps * 32;
constexpr int kMaxSplits = 8;  // portable cluster size
__device__ __forceinline__ int warp_of(unsigned tid) { return static_cast<int>(tid >> 5); }

struct AttnArgs {
  const int64_t* positions;
  const int64_t* page_table;
  const int64_t* sequence_ids;
  int64_t max_pages, page_size;
  int q_heads, kv_heads;
  int hnd;
  int narrow;      // every position a page table row can hold fits 31 bits: 32-bit divisions
  float scale;
  int tokens;
  float* scratch;  // even split of the batch's tiles over the grid, partial results here; nullptr: grid = (splits, heads, tokens)
};

// 16 bytes of a row, or zeros and no access for a dead position (row < 0).  (Dead positions used to read row 0 of the cache: with
// contexts of every length that was megabytes from one line, and its L2 slice set the time -- 64 contexts of 1 .. 2048 took
// longer than 64 of 2048.)
template <typename T>
__device__ __forceinline__ void cp_async16_row(void* dst_smem, const T* cache, int64_t row, int at) {
  cp_async16_or_zero(dst_smem, reinterpret_cast<const unsigned char*>(cache + (row < 0 ? 0 : row)) + at, row >= 0);
}

// Merges partial (m, l, acc) `b` into `a` (online softmax): both cover disjoint position sets.
__device__ __forceinline__ void merge_stats(float& m_a, float& l_a, float& scale_a, float& scale_b, float m_b, float l_b) {
  const float m = fmaxf(m_a, m_b);
  scale_a = m_a == -INFINITY ? 0.0f : __expf(m_a - m);
  scale_b = m_b == -INFINITY ? 0.0f : __expf(m_b - m);
  l_a = l_a * scale_a + l_b * scale_b;
  m_a = m;
}

// ---- even split of a batch ---------------------------------------------------------------------------------------
// Contexts differ from token to token, and only the device knows them.  The tiles of all (token, KV head) items stand
// one behind the other, token-major, and CTA b of B takes tiles [b W / B, (b + 1) W / B) of the W there are (B: the CTAs of the
// grid, or W, if there are fewer tiles than CTAs: the CTAs past W have no part in it).  An item
// that lies inside one CTA is finished there; the others leave one partial result (max, sum, accumulator per head) per
// CTA in scratch -- slot 2 b + 1 for the item that CTA b begins and does not end, slot 2 b for one begun before it --
// and paged_decode_attention_merge_kernel adds them in CTA order.
constexpr int kMergeThreads = 256;
constexpr int kMaxTokensSplit = 16384;  // every CTA adds up the tiles of all tokens: longer batches have items enough
// Shorter contexts stay on the grid of splits: finding the share and the second launch cost 1 .. 4 us, which the even split
// only earns back on uneven or long ones.  (A caller that names no bound gets that of the page table's rows: one token, 2 heads x 64,
// 8.6 us on the grid of splits and 9.6 on the even one for a table of 1024; 16 tokens x 8 heads x 128, 9.8 / 11.2 for one of 256.)
// Short contexts under a long bound cost no more: one token, 8 heads x 128, 512 positions, bound 8192 8.8 / 10.9, 16 tokens 11.9 / 12.5 (one
// token of 2 heads x 64, 1024 positions 20.3 while CTAs without a share left zeros for the merge, which then had them all to add).
// us, contexts of every length up to the bound / all at the bound, even against
// splits: 16 tokens x 8 heads x 128, bound 512 13.8 / 13.3 against 12.3 / 14.9, 1024 15.9 / 19.4 against 15.9 / 18.1, 2048
// 20.0 / 33.2 against 24.1 / 32.9; one token, 8192 13.9 / 16.8 against 14.9 / 24.8; FP32, 64 tokens x 4 heads, 2048 63 / 102 against 123 / 131.
// Against the kernel before the even split, whose dead positions were read: 16 tokens, 8192 56 / 95 from 82 / 98; 64 tokens,
// 2048 58 / 96 from 103 / 122.
constexpr int kMinEvenContext = 1536;
// A larger bound on the contexts says no more than this one: it is far beyond any cache, and keeps tokens * heads * tiles, and the
// roundings up, inside 64 bits.
constexpr int64_t kMaxContextHint = 1LL << 38;

// 32-bit words of scratch per CTA: two accumulators, twice two statistics, a header
constexpr size_t partial_words(size_t g, size_t d) { return 2 * g * d + 2 * (2 * g) + 4; }
template <int G, int D>
struct Partials {  // scratch of a grid of `ctas`
  static constexpr size_t kAcc = 2 * G * D, kStat = 2 * G, kHeader = 4;  // words per CTA
  static_assert(kAcc + 2 * kStat + kHeader == partial_words(G, D), "what the size function asks for is what is laid out here");
  float* acc;      // [2 ctas][G * D]
  float* m;        // [2 ctas][G]
  float* l;        // [2 ctas][G]
  int* header;     // [ctas][kHeader]: token, KV head, CTA that ends the item that CTA b begins; token < 0: none
  __device__ Partials(float* base, int ctas) {
    acc = base;
    m = acc + kAcc * ctas;
    l = m + kStat * ctas;
    header = reinterpret_cast<int*>(l + kStat * ctas);
  }
};

// Context length and sequence of the batch's first tokens, in shared memory: a step to the next item would otherwise cost two
// dependent trips to memory.
constexpr int kCachedTokens = 128;
struct TokenCache {
  int64_t ctx[kCachedTokens], seq[kCachedTokens];
};

struct ItemCursor {  // a tile of an item
  int token, kvh, tile, tiles;
  int64_t ctx;
  const int64_t* table;
  template <int U>  // positions per tile
  __device__ __forceinline__ void load(const AttnArgs& a, const TokenCache* cache) {
    const bool hit = cache != nullptr && token < kCachedTokens;
    ctx = hit ? cache->ctx[token] : a.positions[token] + 1;
    tiles = ctx > U ? static_cast<int>((ctx + U - 1) / U) : 1;  // an empty context is one dead tile
    table = a.page_table + (hit ? cache->seq[token] : a.sequence_ids[token]) * a.max_pages;
  }
  template <int U>
  __device__ __forceinline__ void advance(const AttnArgs& a, const TokenCache* cache) {  // not past the batch's last tile
    if (++tile < tiles) return;
    tile = 0;
    if (++kvh < a.kv_heads) return;
    kvh = 0, ++token;
    load<U>(a, cache);
  }
};

// CTAs that have a share of `total` tiles; each of them has at least one.
__device__ __forceinline__ int64_t share_ctas(int64_t total) { return total < gridDim.x ? total : gridDim.x; }

// Sets `at` to this CTA's first tile and returns how many tiles it has, 0 for a CTA without a share; `batch_tiles` (in shared memory): tiles of the batch.
// All threads call it.
template <int U>
__device__ __forceinline__ int64_t seek_share(const AttnArgs& a, ItemCursor& at, int64_t& batch_tiles, TokenCache& cache) {
  __shared__ int64_t warp_sums[kAttnWarps];
  __shared__ int64_t found[2];
  const int lane = threadIdx.x & 31, warp = warp_of(threadIdx.x);
  auto tiles_of = [&](int t) -> int64_t {
    if (t >= a.tokens) return 0;
    const int64_t ctx = a.positions[t] + 1;
    return (ctx > U ? (ctx + U - 1) / U : 1) * a.kv_heads;
  };
  static_assert(kCachedTokens == kAttnThreads, "one token per thread");
  if (static_cast<int>(threadIdx.x) < a.tokens) {
    cache.ctx[threadIdx.x] = a.positions[threadIdx.x] + 1;
    cache.seq[threadIdx.x] = a.sequence_ids[threadIdx.x];
  }
  const int64_t first = tiles_of(threadIdx.x);
  int64_t sum = first;
  for (int t = threadIdx.x + kAttnThreads; t < a.tokens; t += kAttnThreads) sum += tiles_of(t);
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
  if (lane == 0) warp_sums[warp] = sum;
  __syncthreads();
  int64_t total = 0;
#pragma unroll
  for (int w = 0; w < kAttnWarps; ++w) total += warp_sums[w];
  if (threadIdx.x == 0) batch_tiles = total;
  const int64_t ctas = share_ctas(total);
  if (blockIdx.x >= ctas) return 0;
  const int64_t w0 = total * blockIdx.x / ctas, w1 = total * (blockIdx.x + 1) / ctas;
  int64_t before = 0;  // tiles of the tokens in front of the chunk
  for (int t0 = 0;; t0 += kAttnThreads) {
    const int64_t mine = t0 == 0 ? first : tiles_of(t0 + threadIdx.x);
    int64_t upto = mine;
#pragma unroll
    for (int sh = 1; sh < 32; sh <<= 1) {
      const int64_t v = __shfl_up_sync(0xffffffffu, upto, sh);
      if (lane >= sh) upto += v;
    }
    __syncthreads();
    if (lane == 31) warp_sums[warp] = upto;
    __syncthreads();
    int64_t chunk = 0;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      if (w < warp) upto += warp_sums[w];
      chunk += warp_sums[w];
    }
    if (before + upto - mine <= w0 && w0 < before + upto) found[0] = t0 + threadIdx.x, found[1] = w0 - (before + upto - mine);
    before += chunk;
    if (w0 < before) break;  // same for all threads
  }
  __syncthreads();
  at.token = static_cast<int>(found[0]);
  at.load<U>(a, &cache);
  at.kvh = static_cast<int>(found[1] / at.tiles);
  at.tile = static_cast<int>(found[1] - static_cast<int64_t>(at.kvh) * at.tiles);
  return w1 - w0;
}

// The four warps' partial results of a segment (in part_m, part_l and at acc_of(warp)) -> the output, when the CTA has the
// whole item, or this CTA's slot.  Two block barriers: afterwards the warps' accumulators may be overwritten.
template <typename T, int G, int D, typename AccOf>
__device__ __forceinline__ void finish_segment(const AttnArgs& a, const PeerOut& out, int token, int kvh, int tiles_left, bool begins,
                                               int64_t total, const float (&part_m)[kAttnWarps][G], const float (&part_l)[kAttnWarps][G],
                                               AccOf acc_of) {
  __syncthreads();
  const Partials<G, D> p(a.scratch, gridDim.x);
  const int slot = 2 * blockIdx.x + (begins ? 1 : 0);
  const bool ends = tiles_left == 0;  // of the item, behind this segment
  if (begins && !ends && threadIdx.x == 0) {
    // the CTA that holds the item's last tile: the tile's number in the batch is this CTA's last one + what is left
    const int64_t ctas = share_ctas(total), last = total * (blockIdx.x + 1) / ctas + tiles_left - 1;
    int* h = p.header + 4 * blockIdx.x;
    h[0] = token, h[1] = kvh, h[2] = static_cast<int>(((last + 1) * ctas - 1) / total);
  }
  for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
    const int g = i / D, d = i - g * D;
    float mm = part_m[0][g], ll = part_l[0][g], aa = acc_of(0)[i];
    for (int w = 1; w < kAttnWarps; ++w) {
      float sa, sb;
      merge_stats(mm, ll, sa, sb, part_m[w][g], part_l[w][g]);
      aa = aa * sa + acc_of(w)[i] * sb;
    }
    if (begins && ends) {
      peer_store(out, token, (kvh * G + g) * D + d, Elem<T>::from_f32(aa / ll));
    } else {
      p.acc[static_cast<size_t>(slot) * G * D + i] = aa;
      if (d == 0) p.m[slot * G + g] = mm, p.l[slot * G + g] = ll;
    }
  }
  __syncthreads();
}

// Block b adds the partial results of the item that CTA b began and others went on with.  A thread owns four head dims and
// every NG-th partial result; the NG sums of a dim meet in shared memory.
template <typename T, int G, int D>
__global__ void __launch_bounds__(kMergeThreads)
paged_decode_attention_merge_kernel(const __grid_constant__ PeerOut out, float* scratch) {
  constexpr int kAll = G * D / 4, L = kAll < kMergeThreads ? kAll : kMergeThreads, NG = kMergeThreads / L;
  __shared__ float4 accs[NG][L];
  __shared__ float ms[NG][L], ls[NG][L];
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x;
  const Partials<G, D> p(scratch, gridDim.x);
  const int4 h = __ldcg(reinterpret_cast<const int4*>(p.header + 4 * b));
  if (h.x < 0) return;
  const int group = threadIdx.x / L, lane = threadIdx.x - group * L;
  const int count = h.z - b + 1;
#pragma unroll
  for (int part = 0; part < kAll / L; ++part) {
    const int l4 = part * L + lane, g = l4 * 4 / D;
    float m = -INFINITY, l = 0.0f;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto add = [&](const float4& v, float mv, float lv) {
      float sa, sb;
      merge_stats(m, l, sa, sb, mv, lv);
      acc.x = acc.x * sa + v.x * sb, acc.y = acc.y * sa + v.y * sb;
      acc.z = acc.z * sa + v.z * sb, acc.w = acc.w * sa + v.w * sb;
    };
#pragma unroll 4
    for (int i = group; i < count; i += NG) {
      const int slot = i == 0 ? 2 * b + 1 : 2 * (b + i);
      add(__ldcg(reinterpret_cast<const float4*>(p.acc) + static_cast<size_t>(slot) * kAll + l4), __ldcg(p.m + slot * G + g), __ldcg(p.l + slot * G + g));
    }
    if constexpr (NG > 1) {
      accs[group][lane] = acc, ms[group][lane] = m, ls[group][lane] = l;
      __syncthreads();
      if (group != 0) continue;
      for (int i = 1; i < NG; ++i) add(accs[i][lane], ms[i][lane], ls[i][lane]);
    }
    const int col = h.y * G * D + l4 * 4;
    peer_store(out, h.x, col, Elem<T>::from_f32(acc.x / l));
    peer_store(out, h.x, col + 1, Elem<T>::from_f32(acc.y / l));
    peer_store(out, h.x, col + 2, Elem<T>::from_f32(acc.z / l));
    peer_store(out, h.x, col + 3, Elem<T>::from_f32(acc.w / l));
  }
}

// Element offset of position j of the cursor's sequence and head, -1 for a dead position (its probability is 0).  The page is
// looked up here, the address is made from it when it is used.
struct RowAt {
  int64_t page;
  int off;
  __device__ __forceinline__ void find(const AttnArgs& a, const ItemCursor& c, int64_t j) {
    page = -1, off = 0;
    if (j >= c.ctx) return;
    int64_t logical;
    if (a.narrow) logical = static_cast<uint32_t>(j) / static_cast<uint32_t>(a.page_size);
    else logical = j / a.page_size;
    off = static_cast<int>(j - logical * a.page_size);
    page = c.table[logical];
  }
  __device__ __forceinline__ int64_t offset(const AttnArgs& a, int kvh, int dim) const {
    if (page < 0) return -1;
    return (a.hnd ? (page * a.kv_heads + kvh) * a.page_size + off : (page * a.page_size + off) * a.kv_heads + kvh) * dim;
  }
};

template <typename T, int D>
struct StageV {  // whether a warp's V rows are staged in shared memory beside its K rows
  static constexpr bool value = static_cast<size_t>(kAttnWarps) * 32 * (2 * D * sizeof(T) + 16) <= 72 * 1024;
};

template <typename T, int G, int D>
__global__ void __launch_bounds__(kAttnThreads, D <= 128 ? 3 : 1)  // what its shared memory leaves room for
paged_decode_attention_kernel(const T* q, const T* k_cache, const T* v_cache,
                              const __grid_constant__ PeerOut out, const __grid_constant__ AttnArgs a, int splits) {
  constexpr int E = 16 / sizeof(T);   // elements per 16-byte piece
  constexpr int PIECES = D / E;       // pieces per row
  constexpr int DPL = D / 32;         // dims per lane in the value phase
  static_assert(D % 32 == 0 && D % E == 0, "head_dim must be a multiple of 32");
  constexpr int kRowPitch = D * static_cast<int>(sizeof(T)) + 16;  // bytes; the pad spreads the lanes' rows over the banks
  extern __shared__ __align__(16) unsigned char attn_smem[];
  constexpr int kVPitch = D * static_cast<int>(sizeof(T));         // V rows are read along the row: no pad needed
  // V is staged beside K while that leaves room for three CTAs per SM; longer rows read V straight from global memory
  constexpr bool kStageV = StageV<T, D>::value;
  constexpr int kWarpTile = 32 * (kRowPitch + (kStageV ? kVPitch : 0));
  // [warp][32 K rows of kRowPitch | 32 V rows]; reused after the loop for the warps' accumulators [warp][G][D] floats
  unsigned char* ktile = attn_smem + warp_of(threadIdx.x) * kWarpTile;
  unsigned char* vtile = ktile + 32 * kRowPitch;
  float (*part_acc)[G][D] = reinterpret_cast<float (*)[G][D]>(attn_smem);
  __shared__ __align__(16) float qs[G][D];                 // q of the group, pre-multiplied by scale
  __shared__ __align__(16) float probs[kAttnWarps][32][G];  // the tile's probabilities, [position][head]
  __shared__ int64_t rows[kAttnWarps][32];                  // the tile's row offsets (elements)
  __shared__ float part_m[kAttnWarps][G], part_l[kAttnWarps][G];
  __shared__ float cta_m[G], cta_l[G];                      // the CTA's merged (max, sum)
  __shared__ int64_t batch_tiles;
  __shared__ TokenCache cache;

  pdl_launch_dependents();
  pdl_wait();  // q and the caches are the preceding kernels' output
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool even = a.scratch != nullptr;
  const int split = even ? 0 : blockIdx.x;
  ItemCursor cur;
  int64_t left_tiles = 0;
  if (even) {
    if (threadIdx.x == 0) Partials<G, D>(a.scratch, gridDim.x).header[4 * blockIdx.x] = -1;
    left_tiles = seek_share<kAttnThreads>(a, cur, batch_tiles, cache);
    if (left_tiles == 0) return;
  } else {
    cur.kvh = blockIdx.y, cur.token = blockIdx.z, cur.load<kAttnThreads>(a, nullptr);
  }
  do {  // segments: the tiles this CTA has of an item
  const int kvh = cur.kvh, token = cur.token;
  const int64_t ctx = cur.ctx;
  // a split's slice of the context: whole tiles of 128 positions, dealt evenly
  const int64_t tiles = cur.tiles;
  const int64_t t0 = even ? cur.tile : tiles * split / splits;
  const int64_t t1 = even ? (tiles - t0 < left_tiles ? tiles : t0 + left_tiles) : tiles * (split + 1) / splits;

  for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
    const int g = i / D, d = i - g * D;
    qs[g][d] = Elem<T>::to_f32(q[(static_cast<int64_t>(token) * a.q_heads + kvh * G + g) * D + d]) * a.scale;
  }
  __syncthreads();

  float m[G], l[G], acc[G][DPL];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY, l[g] = 0.0f;
#pragma unroll
    for (int e = 0; e < DPL; ++e) acc[g][e] = 0.0f;
  }

  for (int64_t tile = t0; tile < t1; ++tile) {
    // ---- scores: this lane's position
    const int64_t j = tile * kAttnThreads + warp * 32 + lane;
    const bool live = j < ctx;
    RowAt at;
    at.find(a, cur, j);
    rows[warp][lane] = at.offset(a, kvh, D);
    __syncwarp();
    // the tile's K and V rows into shared memory: chunk c = 16-byte piece (c % PIECES) of row (c / PIECES).  Both
    // go out together, so a tile costs one trip to HBM (V read row by row after the scores cost eight more)
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
      const int c = i * 32 + lane, r = c / PIECES, p = c - r * PIECES;
      cp_async16_row(ktile + r * kRowPitch + p * 16, k_cache, rows[warp][r], p * 16);
    }
    if constexpr (kStageV) {
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const int c = i * 32 + lane, r = c / PIECES, p = c - r * PIECES;
        cp_async16_row(vtile + r * kVPitch + p * 16, v_cache, rows[warp][r], p * 16);
      }
    }
    cp_async_wait_all();
    __syncwarp();
    float s[G];
#pragma unroll
    for (int g = 0; g < G; ++g) s[g] = 0.0f;
    {
      const unsigned char* mine = ktile + lane * kRowPitch;
#pragma unroll 8
      for (int p = 0; p < PIECES; ++p) {
        const U4 raw = *reinterpret_cast<const U4*>(mine + p * 16);
        const T* kv = reinterpret_cast<const T*>(&raw);
        float kf[E];
#pragma unroll
        for (int e = 0; e < E; ++e) kf[e] = Elem<T>::to_f32(kv[e]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
          for (int e = 0; e < E; e += 4) {
            const float4 qv = *reinterpret_cast<const float4*>(&qs[g][p * E + e]);
            s[g] = fmaf(kf[e], qv.x, s[g]);
            s[g] = fmaf(kf[e + 1], qv.y, s[g]);
            s[g] = fmaf(kf[e + 2], qv.z, s[g]);
            s[g] = fmaf(kf[e + 3], qv.w, s[g]);
          }
        }
      }
    }
    // ---- softmax bookkeeping of the tile (per warp)
    float corr[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float mx = live ? s[g] : -INFINITY;
#pragma unroll
      for (int sh = 16; sh > 0; sh >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sh));
      const float m_new = fmaxf(m[g], mx);
      corr[g] = m[g] == -INFINITY ? 0.0f : __expf(m[g] - m_new);
      const float p = live ? __expf(s[g] - m_new) : 0.0f;
      l[g] = l[g] * corr[g] + p;  // per-lane share of the sum; lanes are added at the end
      m[g] = m_new;
      probs[warp][lane][g] = p;
    }
    __syncwarp();
    // ---- values: lanes own DPL dims each
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int e = 0; e < DPL; ++e) acc[g][e] *= corr[g];
    const int64_t left = ctx - (tile * kAttnThreads + warp * 32);
    const int n_live = left >= 32 ? 32 : (left > 0 ? static_cast<int>(left) : 0);
    if constexpr (kStageV) {
    for (int j0 = 0; j0 < n_live; ++j0) {
      float vf[DPL];
      const T* vp = reinterpret_cast<const T*>(vtile + j0 * kVPitch) + lane * DPL;
      if constexpr (DPL * sizeof(T) == 8) {
        const uint2 raw = *reinterpret_cast<const uint2*>(vp);
        const T* ve = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int e = 0; e < DPL; ++e) vf[e] = Elem<T>::to_f32(ve[e]);
      } else if constexpr (DPL * sizeof(T) == 16) {
        const U4 raw = *reinterpret_cast<const U4*>(vp);
        const T* ve = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int e = 0; e < DPL; ++e) vf[e] = Elem<T>::to_f32(ve[e]);
      } else {
#pragma unroll
        for (int e = 0; e < DPL; ++e) vf[e] = Elem<T>::to_f32(vp[e]);
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float p = probs[warp][j0][g];
#pragma unroll
        for (int e = 0; e < DPL; ++e) acc[g][e] = fmaf(p, vf[e], acc[g][e]);
      }
    }
    } else {
    // four positions per pass, their V loads issued together (past the live ones: the last one again, with probability 0)
    for (int j0 = 0; j0 < n_live; j0 += 4) {
      float vf[4][DPL];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const T* vp = v_cache + rows[warp][min(j0 + u, n_live - 1)] + lane * DPL;
        if constexpr (DPL * sizeof(T) == 8) {
          const uint2 raw = *reinterpret_cast<const uint2*>(vp);
          const T* ve = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int e = 0; e < DPL; ++e) vf[u][e] = Elem<T>::to_f32(ve[e]);
        } else if constexpr (DPL * sizeof(T) == 16) {
          const U4 raw = ld_ordered_stream16(vp);
          const T* ve = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int e = 0; e < DPL; ++e) vf[u][e] = Elem<T>::to_f32(ve[e]);
        } else {
#pragma unroll
          for (int e = 0; e < DPL; ++e) vf[u][e] = Elem<T>::to_f32(vp[e]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float p = probs[warp][j0 + u][g];
#pragma unroll
          for (int e = 0; e < DPL; ++e) acc[g][e] = fmaf(p, vf[u][e], acc[g][e]);
        }
    }
    }
    __syncwarp();  // the tile's shared entries are free for the next tile
  }

  // ---- warp totals, then the four warps of the CTA (fixed order)
  __syncthreads();  // every warp is done with its K tile: the buffer now holds the accumulators
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float sum = l[g];  // every lane scaled its share by the same corrections, so shares can simply be added
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
    if (lane == 0) part_m[warp][g] = m[g], part_l[warp][g] = sum;
#pragma unroll
    for (int e = 0; e < DPL; ++e) part_acc[warp][g][lane * DPL + e] = acc[g][e];
  }
  if (even) {
    cur.tile = static_cast<int>(t1 - 1);
    finish_segment<T, G, D>(a, out, token, kvh, static_cast<int>(tiles - t1), t0 == 0, batch_tiles, part_m, part_l, [&](int w) { return &part_acc[w][0][0]; });
    left_tiles -= t1 - t0;
    if (left_tiles > 0) cur.advance<kAttnThreads>(a, &cache);
    continue;
  }
  __syncthreads();
  // thread (g, d) pairs merge the warps; results land in slot 0
  for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
    const int g = i / D, d = i - g * D;
    float mm = part_m[0][g], ll = part_l[0][g], aa = part_acc[0][g][d];
    for (int w = 1; w < kAttnWarps; ++w) {
      float sa, sb;
      merge_stats(mm, ll, sa, sb, part_m[w][g], part_l[w][g]);
      aa = aa * sa + part_acc[w][g][d] * sb;
    }
    part_acc[0][g][d] = aa;
    if (d == 0) cta_m[g] = mm, cta_l[g] = ll;
  }
  __syncthreads();

  if (splits > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();  // every slice's partial is in its CTA's shared memory
    if (split == 0) {
      for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
        const int g = i / D, d = i - g * D;
        float mm = cta_m[g], ll = cta_l[g], aa = part_acc[0][g][d];
        for (int r = 1; r < splits; ++r) {  // rank order
          const float mr = *cluster.map_shared_rank(&cta_m[g], r), lr = *cluster.map_shared_rank(&cta_l[g], r);
          const float ar = *cluster.map_shared_rank(&part_acc[0][g][d], r);
          float sa, sb;
          merge_stats(mm, ll, sa, sb, mr, lr);
          aa = aa * sa + ar * sb;
        }
        peer_store(out, token, (kvh * G + g) * D + d, Elem<T>::from_f32(aa / ll));
      }
    }
    cluster.sync();  // nobody leaves while rank 0 may still read its shared memory
  } else {
    for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
      const int g = i / D, d = i - g * D;
      peer_store(out, token, (kvh * G + g) * D + d, Elem<T>::from_f32(part_acc[0][g][d] / cta_l[g]));
    }
  }
  } while (left_tiles > 0);
}

// ---- the same kernel with both contractions on the tensor cores (16-bit caches) --------------------------------
// The lane-per-position kernel above spends ~1700 warp instructions per tile of 32 positions (two FMAs per cache
// element and G heads) and is issue-bound.  Here positions (for the scores) and head dims (for the values) are the 16 rows
// of mma.m16n8k16 tiles and the G query heads of the group its (zero-padded) eight columns: S^T = K q^T with K straight from
// the staged tile (ldmatrix), O^T = V^T P^T with V through ldmatrix.trans and P, rounded to the cache type, turned from
// result to operand layout by movmatrix.  32 MMAs per tile, every accumulator register in use.  (With the heads as the 16
// rows it was 64, and the half of each accumulator that padding wasted had to be rebuilt with moves: 1050 warp instructions
// per tile, and a tile took 6 us of latency however idle the memory was.)  Staging, online softmax and merges are as above.
template <typename T> struct Mma16816;
template <> struct Mma16816<__half> {
  __device__ static __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  __device__ static __forceinline__ uint32_t pack(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
};
template <> struct Mma16816<__nv_bfloat16> {
  __device__ static __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  __device__ static __forceinline__ uint32_t pack(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
};
// An 8 x 8 matrix of 16-bit elements spread over the warp as a fragment, transposed.
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem_row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(smem_row)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem_row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(smem_row)));
}

// A warp has one tile of 32 positions in shared memory, K and V rows together; twelve warps of an SM take turns loading and
// computing.  (Two stages of 16 positions, the next one's copies in flight, measured slower: 688 warp instructions per 16
// positions.)
template <int D>
struct TcTile {
  static constexpr int kPositions = 32;                         // per warp
  static constexpr int kPitch = D * 2 + 16;                     // bytes; the pad keeps the eight rows of an ldmatrix on eight bank groups
  static constexpr int kStage = 2 * kPositions * kPitch;        // K rows, then V rows
  static constexpr int kUnit = kAttnWarps * kPositions;         // positions of a CTA's tile
  static constexpr int kBytes = kAttnWarps * kStage;
};

template <typename T, int G, int D>
__global__ void __launch_bounds__(kAttnThreads, D <= 128 ? 3 : 1)
paged_decode_attention_tc_kernel(const T* q, const T* k_cache, const T* v_cache,
                                 const __grid_constant__ PeerOut out, const __grid_constant__ AttnArgs a, int splits) {
  static_assert(sizeof(T) == 2 && G <= 8 && D % 32 == 0, "16-bit caches, at most eight heads per group");
  using Tile = TcTile<D>;
  constexpr int PIECES = D / 8;                 // 16-byte pieces per row
  constexpr int kPitch = Tile::kPitch, TP = Tile::kPositions, PB = TP / 16;  // blocks of 16 positions
  static_assert(G * D * 4 <= Tile::kStage, "a warp's accumulators fit the tile that it is done with");
  extern __shared__ __align__(16) unsigned char attn_smem[];
  unsigned char* ktile = attn_smem + warp_of(threadIdx.x) * Tile::kStage;
  unsigned char* vtile = ktile + TP * kPitch;
  __shared__ uintptr_t rows[kAttnWarps][TP];  // addresses of the tile's K rows
  __shared__ float part_m[kAttnWarps][G], part_l[kAttnWarps][G];
  __shared__ float cta_m[G], cta_l[G];
  __shared__ int64_t batch_tiles;
  __shared__ TokenCache cache;

  pdl_launch_dependents();
  pdl_wait();  // q and the caches are the preceding kernels' output
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grow = lane >> 2, quad = lane & 3;  // fragment row, position inside the quad
  const bool head_live = grow < G;              // as a column of B: this lane's head
  const bool even = a.scratch != nullptr;
  const int split = even ? 0 : blockIdx.x;
  ItemCursor cur;  // the tile whose rows are fetched next
  int n_tiles;
  if (even) {
    if (threadIdx.x == 0) Partials<G, D>(a.scratch, gridDim.x).header[4 * blockIdx.x] = -1;
    n_tiles = static_cast<int>(seek_share<Tile::kUnit>(a, cur, batch_tiles, cache));
    if (n_tiles == 0) return;
  } else {
    cur.kvh = blockIdx.y, cur.token = blockIdx.z, cur.load<Tile::kUnit>(a, nullptr);
    cur.tile = static_cast<int>(static_cast<int64_t>(cur.tiles) * split / splits);
    n_tiles = static_cast<int>(static_cast<int64_t>(cur.tiles) * (split + 1) / splits) - cur.tile;
  }

  // V rows lie where the K rows lie, this many bytes on
  const int64_t v_from_k = static_cast<int64_t>(reinterpret_cast<uintptr_t>(v_cache) - reinterpret_cast<uintptr_t>(k_cache));
  RowAt at;  // this lane's row of the tile
  auto look_up = [&]() { at.find(a, cur, static_cast<int64_t>(cur.tile) * Tile::kUnit + warp * TP + lane); };
  if (n_tiles > 0) look_up();

  // q^T as B fragments: b0 = (dims 16 ks + 2 quad + {0,1}, head grow), b1 = the same + 8 dims; heads >= G are zero
  uint32_t qb0[D / 16], qb1[D / 16];
  float m_run[2], l_run[2];  // of heads 2 quad + {0, 1}; l_run is this thread's share of the sum
  float o[D / 16][4];        // O^T: dims 16 dt + grow (+ 8 in the upper two registers), heads 2 quad + {0, 1}
  bool fresh = true;   // the tile begins a segment
  bool begins = false; // the segment begins at its item's first tile
  auto write_partials = [&](float* acc) {  // of this warp
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int sh = 4; sh < 32; sh <<= 1) l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], sh);
      const int head = quad * 2 + e;
      if (head < G) {
        if (grow == 0) part_m[warp][head] = m_run[e], part_l[warp][head] = l_run[e];
#pragma unroll
        for (int dt = 0; dt < D / 16; ++dt) {
          acc[head * D + dt * 16 + grow] = o[dt][e];
          acc[head * D + dt * 16 + grow + 8] = o[dt][e + 2];
        }
      }
    }
  };
  auto begin_segment = [&](int token, int kvh) {
#pragma unroll
    for (int e = 0; e < 2; ++e) m_run[e] = -INFINITY, l_run[e] = 0.0f;
#pragma unroll
    for (int dt = 0; dt < D / 16; ++dt)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[dt][e] = 0.0f;
    const T* qrow = q + (static_cast<int64_t>(token) * a.q_heads + kvh * G + (head_live ? grow : 0)) * D;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      qb0[ks] = head_live ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + quad * 2) : 0u;
      qb1[ks] = head_live ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + quad * 2 + 8) : 0u;
    }
  };
  if (n_tiles == 0) begin_segment(cur.token, cur.kvh);  // a split without tiles (more splits than tiles) contributes nothing

  for (int u = 0; u < n_tiles; ++u) {
    rows[warp][lane] = reinterpret_cast<uintptr_t>(k_cache) + (at.page < 0 ? 0 : at.offset(a, cur.kvh, D) * static_cast<int64_t>(sizeof(T)));
    __syncwarp();
    const int64_t rest = cur.ctx - static_cast<int64_t>(cur.tile) * Tile::kUnit - warp * TP;
    const int live_end = rest < TP ? static_cast<int>(rest > 0 ? rest : 0) : TP;  // of this warp's positions
    // K and V rows of the tile, 16 bytes per lane and instruction: one trip to HBM.  Dead positions, the last ones of the
    // tile, are zero-filled and not read.
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
      const int c = i * 32 + lane, r = c / PIECES, p = c - r * PIECES;
      const unsigned char* src = reinterpret_cast<const unsigned char*>(rows[warp][r]) + p * 16;
      const bool live = r < live_end;
      cp_async16_or_zero(ktile + r * kPitch + p * 16, src, live);
      cp_async16_or_zero(vtile + r * kPitch + p * 16, src + v_from_k, live);
    }
    const int token = cur.token, kvh = cur.kvh, tiles_left = cur.tiles - 1 - cur.tile;
    if (fresh) {
      begin_segment(token, kvh);
      begins = cur.tile == 0;
    }
    if (u + 1 < n_tiles) {  // the page of the next tile's row is on its way while this tile lands and is computed
      if (even) cur.advance<Tile::kUnit>(a, &cache);
      else ++cur.tile;
      look_up();
    }
    cp_async_wait_all();
    __syncwarp();

    // ---- S^T = K q^T: lane supplies the address of row lane % 16 of a block, dims half lane / 16
    float sc[PB][4];  // positions 16 pb + grow (+ 8 in the upper two), heads 2 quad + {0, 1}
#pragma unroll
    for (int pb = 0; pb < PB; ++pb)
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[pb][e] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
      for (int pb = 0; pb < PB; ++pb) {
        uint32_t k[4];
        ldmatrix_x4(k, ktile + (pb * 16 + (lane & 15)) * kPitch + (lane >> 4) * 16 + ks * 32);
        Mma16816<T>::run(sc[pb], k, qb0[ks], qb1[ks]);
      }
    // ---- online softmax of the two heads
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int pb = 0; pb < PB; ++pb)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool live = pb * 16 + grow + (e >> 1) * 8 < live_end;
        sc[pb][e] = live ? sc[pb][e] * a.scale : -INFINITY;
        mx[e & 1] = fmaxf(mx[e & 1], sc[pb][e]);
      }
    float corr[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int sh = 4; sh < 32; sh <<= 1) mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], sh));
      const float m_new = fmaxf(m_run[e], mx[e]);
      corr[e] = m_run[e] == -INFINITY ? 0.0f : __expf(m_run[e] - m_new);
      m_run[e] = m_new;
      l_run[e] *= corr[e];
    }
    uint32_t pb0[PB], pb1[PB];  // P^T as B fragments: positions 16 pb + 2 quad + {0,1} (+ 8 in pb1), head grow
#pragma unroll
    for (int pb = 0; pb < PB; ++pb) {
      float p[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        p[e] = sc[pb][e] == -INFINITY ? 0.0f : __expf(sc[pb][e] - m_run[e & 1]);
        l_run[e & 1] += p[e];
      }
      pb0[pb] = transpose8x8(Mma16816<T>::pack(p[0], p[1]));
      pb1[pb] = transpose8x8(Mma16816<T>::pack(p[2], p[3]));
    }
#pragma unroll
    for (int dt = 0; dt < D / 16; ++dt)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[dt][e] *= corr[e & 1];
    // ---- O^T += V^T P^T: matrix lane / 8 of a load = (position half, dim half)
#pragma unroll
    for (int pb = 0; pb < PB; ++pb)
#pragma unroll
      for (int dt = 0; dt < D / 16; ++dt) {
        uint32_t v[4];
        ldmatrix_x4_trans(v, vtile + (pb * 16 + (lane >> 4) * 8 + (lane & 7)) * kPitch + (lane >> 3 & 1) * 16 + dt * 32);
        Mma16816<T>::run(o[dt], v, pb0[pb], pb1[pb]);
      }
    __syncwarp();  // every lane has read the tile

    fresh = even && (tiles_left == 0 || u + 1 == n_tiles);
    if (fresh) {
      write_partials(reinterpret_cast<float*>(ktile));
      finish_segment<T, G, D>(a, out, token, kvh, tiles_left, begins, batch_tiles, part_m, part_l,
                              [&](int w) { return reinterpret_cast<const float*>(attn_smem + w * Tile::kStage); });
    }
  }
  if (even) return;

  // ---- grid of splits: warp totals, then the four warps of the CTA (fixed order), then the cluster
  const int token = cur.token, kvh = cur.kvh;
  auto acc_of = [&](int w) { return reinterpret_cast<float*>(attn_smem + w * Tile::kStage); };
  write_partials(acc_of(warp));
  float* cta_acc = acc_of(0);
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
    const int g = i / D, d = i - g * D;
    float mm = part_m[0][g], ll = part_l[0][g], aa = cta_acc[i];
    for (int w = 1; w < kAttnWarps; ++w) {
      float sa, sb;
      merge_stats(mm, ll, sa, sb, part_m[w][g], part_l[w][g]);
      aa = aa * sa + acc_of(w)[i] * sb;
    }
    cta_acc[i] = aa;
    if (d == 0) cta_m[g] = mm, cta_l[g] = ll;
  }
  __syncthreads();

  if (splits > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();  // every slice's partial is in its CTA's shared memory
    if (split == 0) {
      for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
        const int g = i / D, d = i - g * D;
        float mm = cta_m[g], ll = cta_l[g], aa = cta_acc[i];
        for (int r = 1; r < splits; ++r) {  // rank order
          const float mr = *cluster.map_shared_rank(&cta_m[g], r), lr = *cluster.map_shared_rank(&cta_l[g], r);
          const float ar = *cluster.map_shared_rank(&cta_acc[i], r);
          float sa, sb;
          merge_stats(mm, ll, sa, sb, mr, lr);
          aa = aa * sa + ar * sb;
        }
        peer_store(out, token, (kvh * G + g) * D + d, Elem<T>::from_f32(aa / ll));
      }
    }
    cluster.sync();  // nobody leaves while rank 0 may still read its shared memory
  } else {
    for (int i = threadIdx.x; i < G * D; i += kAttnThreads) {
      const int g = i / D, d = i - g * D;
      peer_store(out, token, (kvh * G + g) * D + d, Elem<T>::from_f32(cta_acc[i] / cta_l[g]));
    }
  }
}

// CTAs of a launch that splits the batch evenly (0: the batch stays on the grid of splits): what the SMs hold at once, and
// no more than leaves every CTA as many tiles as the busiest would have anyway, by the bound on the contexts.
inline int even_grid(int64_t tokens, int64_t kv_heads, int64_t dim, int64_t hint, int elem, int g) {
  if (tokens > kMaxTokensSplit || kv_heads > 65535 || (hint > 0 && hint < kMinEvenContext)) return 0;
  if (hint > kMaxContextHint) hint = kMaxContextHint;
  const bool stage_v = kAttnWarps * 32 * (2 * dim * elem + 16) <= 72 * 1024;  // StageV of the FP32 kernel
  int64_t smem = elem == 4 ? kAttnWarps * 32 * ((stage_v ? 2 : 1) * dim * elem + 16) : kAttnWarps * 64 * (dim * 2 + 16);
  smem += elem == 4 ? g * dim * 4 + kAttnWarps * 32 * (g * 4 + 8) + 3840 : 4608;  // static and reserved
  const int64_t regs_allow = dim > 128 ? 1 : 3;
  int64_t per_sm = (227 * 1024) / smem;
  per_sm = per_sm < 1 ? 1 : (per_sm > regs_allow ? regs_allow : per_sm);
  int64_t ctas = per_sm * sm_count();
  if (hint > 0) {
    const int64_t most = tokens * kv_heads * ((hint + kAttnThreads - 1) / kAttnThreads);  // tiles
    if (most < ctas) ctas = most;
    const int64_t each = (most + ctas - 1) / ctas;
    ctas = (most + each - 1) / each;
  }
  return static_cast<int>(ctas);
}

// launch_opts puts the cluster along y; this kernel's cluster runs along x (the context splits)
template <typename T, int G, int D>
int launch_attention_cluster(const void* q, const void* kc, const void* vc, const PeerOut& out, const AttnArgs& a, int64_t tokens,
                             int splits, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = a.scratch ? dim3(static_cast<unsigned>(splits))
                          : dim3(static_cast<unsigned>(splits), static_cast<unsigned>(a.kv_heads), static_cast<unsigned>(tokens));
  cfg.blockDim = dim3(kAttnThreads);
  constexpr bool kTensorCores = sizeof(T) == 2;  // 16-bit caches: both contractions as mma.sync tiles
  constexpr size_t acc_bytes = static_cast<size_t>(kAttnWarps) * G * D * sizeof(float);
  size_t smem;
  void (*kernel)(const T*, const T*, const T*, const PeerOut, AttnArgs, int);
  if constexpr (kTensorCores) {
    kernel = paged_decode_attention_tc_kernel<T, G, D>;
    smem = TcTile<D>::kBytes;
  } else {
    kernel = paged_decode_attention_kernel<T, G, D>;
    smem = static_cast<size_t>(kAttnWarps) * 32 * ((StageV<T, D>::value ? 2 : 1) * D * sizeof(T) + 16);
    if (smem < acc_bytes) smem = acc_bytes;
  }
  if (smem > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return note_launch(err);
  }
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (splits > 1 && !a.scratch) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = static_cast<unsigned>(splits);
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (call_flags() & XDK_DEPENDENT_LAUNCH) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  const int st = note_launch(cudaLaunchKernelEx(&cfg, kernel, static_cast<const T*>(q), static_cast<const T*>(kc),
                                                static_cast<const T*>(vc), out, a, splits));
  if (st != XDK_OK || !a.scratch) return st;
  return launch_opts(paged_decode_attention_merge_kernel<T, G, D>, dim3(static_cast<unsigned>(splits)), dim3(kMergeThreads), 0, s, 1u,
                     true, out, a.scratch);
}

template <typename T, int G>
int dispatch_dim(int64_t d, const void* q, const void* kc, const void* vc, const PeerOut& out, const AttnArgs& a, int64_t tokens, int splits,
                 cudaStream_t s) {
  switch (d) {
    case 64: return launch_attention_cluster<T, G, 64>(q, kc, vc, out, a, tokens, splits, s);
    case 128: return launch_attention_cluster<T, G, 128>(q, kc, vc, out, a, tokens, splits, s);
    case 256: return launch_attention_cluster<T, G, 256>(q, kc, vc, out, a, tokens, splits, s);
    default: return XDK_ERR_LIMIT;
  }
}

template <typename T>
int dispatch_group(int g, int64_t d, const void* q, const void* kc, const void* vc, const PeerOut& out, const AttnArgs& a, int64_t tokens,
                   int splits, cudaStream_t s) {
  switch (g) {
    case 1: return dispatch_dim<T, 1>(d, q, kc, vc, out, a, tokens, splits, s);
    case 2: return dispatch_dim<T, 2>(d, q, kc, vc, out, a, tokens, splits, s);
    case 4: return dispatch_dim<T, 4>(d, q, kc, vc, out, a, tokens, splits, s);
    case 8: return dispatch_dim<T, 8>(d, q, kc, vc, out, a, tokens, splits, s);
    default: return XDK_ERR_LIMIT;
  }
}

}  // namespace
}  // namespace xdk

extern "C" int xdk_paged_decode_attention(const void* q, const void* k_cache, const void* v_cache, const int64_t* positions,
                                          const int64_t* page_table, const int64_t* sequence_ids, void* out, int64_t tokens,
                                          int64_t q_heads, int64_t kv_heads, int64_t head_dim, int64_t max_pages_per_seq,
                                          int64_t page_size, int cache_is_hnd, float scale, int64_t context_hint, int dtype,
                                          unsigned flags, void* stream) {
  if (!out) return XDK_ERR_ARG;
  xdk_peer_out one = {};
  one.ptr[0] = out, one.world = 1, one.ld = q_heads * head_dim, one.col0 = 0;
  return xdk_paged_decode_attention_peer(q, k_cache, v_cache, positions, page_table, sequence_ids, &one, tokens, q_heads, kv_heads,
                                         head_dim, max_pages_per_seq, page_size, cache_is_hnd, scale, context_hint, dtype, flags,
                                         stream);
}

extern "C" int xdk_paged_decode_attention_peer(const void* q, const void* k_cache, const void* v_cache, const int64_t* positions,
                                               const int64_t* page_table, const int64_t* sequence_ids, const xdk_peer_out* out_dst,
                                               int64_t tokens, int64_t q_heads, int64_t kv_heads, int64_t head_dim,
                                               int64_t max_pages_per_seq, int64_t page_size, int cache_is_hnd, float scale,
                                               int64_t context_hint, int dtype, unsigned flags, void* stream) {
  return xdk_paged_decode_attention_ws(q, k_cache, v_cache, positions, page_table, sequence_ids, out_dst, tokens, q_heads, kv_heads,
                                       head_dim, max_pages_per_seq, page_size, cache_is_hnd, scale, context_hint, dtype, nullptr, 0,
                                       flags, stream);
}

extern "C" size_t xdk_paged_decode_attention_scratch_bytes(int64_t tokens, int64_t q_heads, int64_t kv_heads, int64_t head_dim,
                                                           int64_t context_hint, int dtype) {
  using namespace xdk;
  if (tokens < 1 || q_heads < 1 || kv_heads < 1 || q_heads % kv_heads != 0 || q_heads / kv_heads > 8) return 0;
  if (head_dim != 64 && head_dim != 128 && head_dim != 256) return 0;
  const int g = static_cast<int>(q_heads / kv_heads);
  const int ctas = even_grid(tokens, kv_heads, head_dim, context_hint, dtype == XDK_F32 ? 4 : 2, g);
  return ctas * partial_words(g, head_dim) * 4;
}

extern "C" int xdk_paged_decode_attention_ws(const void* q, const void* k_cache, const void* v_cache, const int64_t* positions,
                                             const int64_t* page_table, const int64_t* sequence_ids, const xdk_peer_out* out_dst,
                                             int64_t tokens, int64_t q_heads, int64_t kv_heads, int64_t head_dim,
                                             int64_t max_pages_per_seq, int64_t page_size, int cache_is_hnd, float scale,
                                             int64_t context_hint, int dtype, void* scratch, size_t scratch_bytes, unsigned flags,
                                             void* stream) {
  using namespace xdk;
  PeerOut out;
  if (int st = make_out(out_dst, nullptr, 1, &out)) return st;
  if (q_heads > 0 && head_dim > 0 && out.ld < out.col0 + q_heads * head_dim) return XDK_ERR_ARG;
  if (flags & ~XDK_DEPENDENT_LAUNCH) return XDK_ERR_ARG;
  CallFlagsScope scope(flags);
  if (!q || !k_cache || !v_cache || !positions || !page_table || !sequence_ids) return XDK_ERR_ARG;
  if (tokens < 1 || q_heads < 1 || kv_heads < 1 || head_dim < 1 || max_pages_per_seq < 1 || page_size < 1) return XDK_ERR_ARG;
  if (q_heads % kv_heads != 0 || !(scale == scale)) return XDK_ERR_ARG;
  if (tokens > 65535 || kv_heads > 65535) return XDK_ERR_LIMIT;
  // no bound from the caller: a row of the page table has one
  if (context_hint <= 0 && max_pages_per_seq <= kMaxContextHint / page_size) context_hint = max_pages_per_seq * page_size;
  if (context_hint > kMaxContextHint) context_hint = kMaxContextHint;
  if (!aligned16(q) || !aligned16(k_cache) || !aligned16(v_cache)) return XDK_ERR_ARG;
  if (int st = require_sm100()) return st;
  AttnArgs a;
  a.positions = positions, a.page_table = page_table, a.sequence_ids = sequence_ids;
  a.max_pages = max_pages_per_seq, a.page_size = page_size;
  a.q_heads = static_cast<int>(q_heads), a.kv_heads = static_cast<int>(kv_heads);
  a.hnd = cache_is_hnd ? 1 : 0;
  a.narrow = page_size < (1LL << 31) && max_pages_per_seq < (1LL << 31) && page_size * max_pages_per_seq < (1LL << 31) ? 1 : 0;
  a.scale = scale;
  a.tokens = static_cast<int>(tokens);
  a.scratch = nullptr;
  const int g = static_cast<int>(q_heads / kv_heads);
  int splits = 0;
  if (scratch && g <= 8 && aligned16(scratch)) {
    const size_t need = xdk_paged_decode_attention_scratch_bytes(tokens, q_heads, kv_heads, head_dim, context_hint, dtype);
    if (need > 0 && scratch_bytes >= need) {
      a.scratch = static_cast<float*>(scratch);
      splits = even_grid(tokens, kv_heads, head_dim, context_hint, dtype == XDK_F32 ? 4 : 2, g);
    }
  }
  if (!a.scratch) {
  // Context splits: as many CTAs as the SMs hold at once, at most one split per 128-position tile of the longest
  // context the caller expects (context_hint; <= 0: assume long contexts), at most the portable cluster size.
  // CTAs an SM holds at once, by the shared memory of the kernel that will run (registers allow four)
  const int64_t elem = dtype == XDK_F32 ? 4 : 2;
  const bool staged = kAttnWarps * 32 * (2 * head_dim * elem + 16) <= 72 * 1024;  // StageV of the FP32 kernel
  const int64_t tile_smem = dtype == XDK_F32 ? kAttnWarps * 32 * ((staged ? 2 : 1) * head_dim * elem + 16)
                                            : kAttnWarps * 2 * 32 * (head_dim * elem + 16);
  int64_t resident = (220 * 1024) / (tile_smem > 0 ? tile_smem : 1);
  resident = resident < 1 ? 1 : (resident > 4 ? 4 : resident);
  splits = static_cast<int>(resident * sm_count() / (tokens * kv_heads));      // one wave, never a partial second one
  if (context_hint > 0) {
    const int64_t tiles = (context_hint + kAttnThreads - 1) / kAttnThreads;
    if (splits > tiles) splits = static_cast<int>(tiles);
  }
  if (splits > kMaxSplits) splits = kMaxSplits;
  if (splits < 1) splits = 1;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case XDK_F32: return dispatch_group<float>(g, head_dim, q, k_cache, v_cache, out, a, tokens, splits, s);
    case XDK_BF16: return dispatch_group<__nv_bfloat16>(g, head_dim, q, k_cache, v_cache, out, a, tokens, splits, s);
    case XDK_F16: return dispatch_group<__half>(g, head_dim, q, k_cache, v_cache, out, a, tokens, splits, s);
    default: return XDK_ERR_ARG;
  }
}
