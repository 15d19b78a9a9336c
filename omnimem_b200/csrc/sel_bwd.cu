// Selection attention backward, general geometry (bf16 / fp16, D in {64,128}):
//   * inverted (block -> query groups) CSR index: histogram, per-(b,h) scan, scatter, sort;
//   * dQ: the forward's two forms, a ring of K/V tiles per warp (sel_rows.cuh) or packed tiles per group
//     (sel_packed.cuh); computes delta = sum(O*dO) in its prologue and stores it for the dK/dV kernel;
//   * dK/dV kernel: one thread block OWNS a tile of at most 32 or 64 tokens of one (b, h, block) and walks the
//     block's bucket of query groups in ascending group order - no atomics, results are
//     bit-reproducible from run to run.  (Blocks of at most 32 tokens take sel_bwd_dkv_rows_tc.cu where tensor maps
//     describe the query rows.)
#include "sel_packed.cuh"
#include "sel_rows.cuh"

#include <type_traits>

namespace nsa {
namespace {

__host__ __device__ __forceinline__ int64_t min64(int64_t a, int64_t b) { return a < b ? a : b; }
constexpr int kIdxThreads = 256;

struct IdxParams {
  const int32_t* ids;
  int64_t i_sb, i_sg, i_sh, i_st;
  int B, MG, H, T;
  int64_t NS;
  int block_size, chunk_size, causal, G;
  int32_t* slots;          // optional second output (same layout as groups): the entry's position in its group's id list
};

// With a slot output the entries travel as (group << 8 | slot) through scatter and sort (T <= 256,
// MG < 2^23), so that equal groups stay ordered by slot, and are taken apart at the end.
constexpr int kSlotBits = 8;
__device__ __forceinline__ int32_t inv_entry(const IdxParams& p, int g, int t) {
  return p.slots != nullptr ? ((g << kSlotBits) | t) : g;
}

__device__ __forceinline__ bool pair_bucket(const IdxParams& p, int b, int g, int h, int t,
                                            int& bucket) {
  const int32_t bid = p.ids[b * p.i_sb + g * p.i_sg + h * p.i_sh + t * p.i_st];
  if (bid < 0 || bid >= p.NS) return false;
  if (p.causal) {
    // chunk of the block's first token <= chunk of the group's first token; one division, in 32 bits where it fits
    const int64_t q0 = static_cast<int64_t>(g) * p.G;
    const int64_t in_chunk = q0 <= 0xffffffffll ? static_cast<uint32_t>(q0) % static_cast<uint32_t>(p.chunk_size) : q0 % p.chunk_size;
    if (static_cast<int64_t>(bid) * p.block_size >= q0 - in_chunk + p.chunk_size) return false;
  }
  bucket = bid;
  return true;
}

template <bool SCATTER>
__global__ void inv_pass_kernel(const IdxParams p, int32_t* __restrict__ counts,
                                int32_t* __restrict__ groups) {
  const uint32_t pair = blockIdx.x * blockDim.x + threadIdx.x;        // (the host keeps them below 2^31)
  if (pair >= static_cast<uint32_t>(p.MG) * static_cast<uint32_t>(p.T)) return;
  const int h = blockIdx.y, b = blockIdx.z;
  const int g = static_cast<int>(pair / static_cast<uint32_t>(p.T)), t = static_cast<int>(pair - static_cast<uint32_t>(g) * p.T);
  int bucket;
  if (!pair_bucket(p, b, g, h, t, bucket)) return;
  const int64_t row = static_cast<int64_t>(b) * p.H + h;
  const int pos = atomicAdd(&counts[row * p.NS + bucket], 1);
  if (SCATTER) groups[row * p.MG * p.T + pos] = inv_entry(p, g, t);
}

// One thread block per (b, h) row: exclusive scan of the NS counts -> offsets[NS+1]; the
// counts are replaced by the offsets so the scatter pass can use them as cursors.
__global__ void inv_scan_kernel(int32_t* __restrict__ counts, int32_t* __restrict__ offsets,
                                int64_t NS) {
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  const int64_t row = blockIdx.x;
  int32_t* c = counts + row * NS;
  int32_t* o = offsets + row * (NS + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < NS; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int v = i < NS ? c[i] : 0;
    int x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += y;
      }
      warp_sums[lane] = w;   // inclusive sums of the warps
    }
    __syncthreads();
    const int carry = carry_s;
    const int excl = carry + (warp ? warp_sums[warp - 1] : 0) + x - v;
    if (i < NS) { o[i] = excl; c[i] = excl; }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry_s = carry + warp_sums[nw - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) o[NS] = carry_s;
}

// A warp sorts a bucket of n <= 32 HELD entries in registers (bitonic network, entry e = 32 x + lane in v[x]) and writes
// it in order; in place is fine.
constexpr int kHeld = 8;
template <int HELD>
__device__ __forceinline__ void sort_held(const int32_t* in, int32_t* out, int32_t* out_slots, int n) {
  const int lane = threadIdx.x & 31;
  int32_t v[HELD];
#pragma unroll
  for (int x = 0; x < HELD; ++x) v[x] = x * 32 + lane < n ? in[x * 32 + lane] : 0x7fffffff;
#pragma unroll
  for (int k = 2; k <= 32 * HELD; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int x = 0; x < HELD; ++x) {
        if (j >= 32) {
          const int y = x ^ (j / 32);
          if (y > x) {
            const int32_t lo = min(v[x], v[y]), hi = max(v[x], v[y]);
            const bool up = ((x * 32) & k) == 0;
            v[x] = up ? lo : hi;
            v[y] = up ? hi : lo;
          }
        } else {
          const int32_t o = __shfl_xor_sync(0xffffffffu, v[x], j);
          const bool up = ((x * 32 + lane) & k) == 0, lower = (lane & j) == 0;
          v[x] = up == lower ? min(v[x], o) : max(v[x], o);
        }
      }
#pragma unroll
  for (int x = 0; x < HELD; ++x)
    if (x * 32 + lane < n) {
      out[x * 32 + lane] = out_slots != nullptr ? v[x] >> kSlotBits : v[x];
      if (out_slots != nullptr) out_slots[x * 32 + lane] = v[x] & ((1 << kSlotBits) - 1);
    }
}
__device__ __forceinline__ void warp_sort(const int32_t* in, int32_t* out, int32_t* out_slots, int n) {
  if (n <= 32) sort_held<1>(in, out, out_slots, n);
  else if (n <= 64) sort_held<2>(in, out, out_slots, n);
  else if (n <= 128) sort_held<4>(in, out, out_slots, n);
  else sort_held<kHeld>(in, out, out_slots, n);
}

// Puts buckets [i0, i1) of row (b, h) in order, by a block of 32 warps: a warp sorts a bucket of `shortest` to 32 kHeld
// entries, a longer one is written again by the whole block walking over the row's pairs.  Bucket i is
// [begin(i), begin(i + 1)) of `in`, `out` and `slots`.
template <typename Begin>
__device__ __forceinline__ void inv_order(const IdxParams& p, int b, int h, const int32_t* in, int32_t* out, int32_t* slots,
                                          int i0, int i1, int shortest, Begin&& begin) {
  constexpr int longest = 32 * kHeld;
  __shared__ int found[2][32];
  __shared__ int any_long;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) any_long = 0;
  __syncthreads();
  for (int i = i0 + warp; i < i1; i += 32) {
    const int beg = begin(i), n = begin(i + 1) - beg;
    if (n > longest) {
      if (lane == 0) any_long = 1;
    } else if (n >= shortest) {
      warp_sort(in + beg, out + beg, slots != nullptr ? slots + beg : nullptr, n);
    }
  }
  __syncthreads();
  if (any_long == 0) return;
  const int pairs = p.MG * p.T;
  for (int i = i0; i < i1; ++i) {
    int at = begin(i);
    if (begin(i + 1) - at <= longest) continue;
    __syncthreads();                                 // the counters of the bucket before
    for (int p0 = 0, turn = 0; p0 < pairs; p0 += 1024, turn ^= 1) {
      const int pr = p0 + threadIdx.x, g = pr / p.T;
      int bucket = -1;
      const bool mine = pr < pairs && pair_bucket(p, b, g, h, pr - g * p.T, bucket) && bucket == i;
      const uint32_t m = __ballot_sync(0xffffffffu, mine);
      if (lane == 0) found[turn][warp] = __popc(m);
      __syncthreads();
      int upto = found[turn][lane];                  // inclusive prefix sum over the warps
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += y;
      }
      const int before = __shfl_sync(0xffffffffu, upto, warp > 0 ? warp - 1 : 0);
      const int to = at + (warp > 0 ? before : 0) + __popc(m & ((1u << lane) - 1));
      if (mine) {
        out[to] = g;
        if (slots != nullptr) slots[to] = pr - g * p.T;
      }
      at += __shfl_sync(0xffffffffu, upto, 31);
    }
  }
}

// After the scatter pass: a thread block puts `per` buckets of a row in order, where they lie.
__global__ void __launch_bounds__(1024) inv_sort_kernel(const IdxParams p, const int32_t* __restrict__ offsets, int32_t* groups, int per) {
  const int h = blockIdx.y, b = blockIdx.z;
  const int64_t row = static_cast<int64_t>(b) * p.H + h, pairs = static_cast<int64_t>(p.MG) * p.T;
  const int32_t* o = offsets + row * (p.NS + 1);
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * per, i1 = min64(i0 + per, p.NS);
  inv_order(p, b, h, groups + row * pairs, groups + row * pairs, p.slots != nullptr ? p.slots + row * pairs : nullptr,
            static_cast<int>(i0), static_cast<int>(i1), 1, [&](int i) { return o[i]; });
}

// The whole index of one (b, h) row in a single thread block: histogram, cursors and buckets in shared memory, scatter,
// then one thread per bucket sorts it (a warp where it is long) and the bucket array is written out once, coalesced.
constexpr int kThreadSort = 48;
__global__ void __launch_bounds__(1024) inv_fused_kernel(const IdxParams p, int32_t* __restrict__ groups, int32_t* __restrict__ offsets) {
  extern __shared__ int s_cnt[];                   // [NS], then [pairs]
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H;
  const int64_t row = blockIdx.x;
  const int NS = static_cast<int>(p.NS);
  const int pairs = p.MG * p.T;
  int32_t* o = offsets + row * (p.NS + 1);
  int32_t* gr_out = groups + row * static_cast<int64_t>(pairs);
  int32_t* gr = s_cnt + NS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = threadIdx.x; i < NS; i += blockDim.x) s_cnt[i] = 0;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int pr = threadIdx.x; pr < pairs; pr += blockDim.x) {
    int bucket;
    if (pair_bucket(p, b, pr / p.T, h, pr % p.T, bucket)) atomicAdd(&s_cnt[bucket], 1);
  }
  __syncthreads();
  for (int base = 0; base < NS; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < NS ? s_cnt[i] : 0;
    int x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w += y;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    const int carry = carry_s;
    const int excl = carry + (warp ? warp_sums[warp - 1] : 0) + x - v;
    if (i < NS) { o[i] = excl; s_cnt[i] = excl; }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry_s = carry + warp_sums[nw - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) o[NS] = carry_s;
  for (int pr = threadIdx.x; pr < pairs; pr += blockDim.x) {
    int bucket;
    const int g = pr / p.T;
    if (pair_bucket(p, b, g, h, pr % p.T, bucket)) gr[atomicAdd(&s_cnt[bucket], 1)] = inv_entry(p, g, pr % p.T);
  }
  __syncthreads();                                   // cursors now point one past their bucket
  bool any = false;
  const auto begin = [&](int i) { return i > 0 ? s_cnt[i - 1] : 0; };
  for (int sidx = threadIdx.x; sidx < NS; sidx += blockDim.x) {
    const int end = s_cnt[sidx], beg = begin(sidx);
    if (end - beg > kThreadSort) { any = true; continue; }
    for (int a = beg + 1; a < end; ++a) {
      const int32_t v = gr[a];
      int c = a - 1;
      while (c >= beg && gr[c] > v) { gr[c + 1] = gr[c]; --c; }
      gr[c + 1] = v;
    }
  }
  any = __syncthreads_or(any);
  const int total = carry_s;                         // pairs that landed in a bucket
  int32_t* sl_out = p.slots != nullptr ? p.slots + row * static_cast<int64_t>(pairs) : nullptr;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int32_t v = gr[i];
    if (sl_out != nullptr) {
      gr_out[i] = v >> kSlotBits;
      sl_out[i] = v & ((1 << kSlotBits) - 1);
    } else {
      gr_out[i] = v;
    }
  }
  if (any) inv_order(p, b, h, gr, gr_out, sl_out, 0, NS, kThreadSort + 1, begin);        // (its first barrier: after the copies)
}

// ------------------------------------------------------------------------------------ dQ
struct BwdParams {
  const char* q; int64_t q_sb, q_sm, q_sh;
  const char* o; int64_t o_sb, o_sm, o_sh;
  const char* dO; int64_t do_sb, do_sm, do_sh;
  char* dq; int64_t dq_sb, dq_sm, dq_sh;
  char* dk; char* dv;                    // contiguous [B,N,H,D]
  const float* lse;                      // [B,H,M]
  float* delta;                          // [B,H,M]
  const int32_t* ids; int64_t i_sb, i_sg, i_sh, i_st;
  const int32_t* groups;                 // [B,H,MG*T]
  const int32_t* offsets;                // [B,H,NS+1]
  KVSrc kv;
  int B, H, T, block_size, chunk_size, causal, G, MG;
  int parts;                             // dQ: thread blocks that share a group's rows
  int64_t M, NS;
  float scale, scale_log2;
  // dK/dV kernel only, pointer mode (selection_bwd.cu:1409-1527, bwd_common.cuh:64-121): K/V blocks
  // and the fp32 gradient scratch of a block are found through [H, MAXB] tables of byte addresses
  // (block-level, or chunk-level plus an in-chunk offset); a zero or out-of-range entry skips the block.
  struct Tables {
    int on;
    const int64_t *base_k, *base_v, *base_dk, *base_dv;
    int64_t base_sh, base_sb;
    int max_base;
    const int32_t* n_blocks_per_head;
    int64_t batch_kv_bytes, batch_dkv_bytes, in_chunk_kv_bytes, in_chunk_dkv_bytes;
    int blocks_per_chunk;
    int64_t s_bn, s_dbn;        // elements between tokens: K/V blocks, fp32 scratch
  } tab;
};

// W warps of 16 query rows share one ring of K/V tiles; p.parts such thread blocks take a group and walk the list each for
// itself; with W = 1 the list may be dealt out to KS warps.  Bounds as in the forward, with 9 warps per SM (registers: Q and dO fragments and the
// accumulator).  32760 queries x 12 heads, 15-query groups, 16 blocks of 30: 623 us (10142 us with packed tiles).
// 3120 queries x 12 heads, 16 blocks of 64, D = 128, groups of 32 / 64 / 128: 130 / 131 / 173 us; 151 / 152 / 184 us with two warps per
// ring, 417 / 294 / 294 us with four, 506 / 259 / 203 us with eight.
template <typename T, int D, int W, int KS, bool TMA>
__global__ void __launch_bounds__(32 * W * KS, 1) sel_bwd_dq_rows_kernel(
    const __grid_constant__ RingMaps maps, const BwdParams p, const int stages, int32_t* status) {
  static_assert(W == 1 || KS == 1, "only single-warp groups are split");
  constexpr int ESZ = sizeof(T), ROWS = 32;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t4 = lane & 3;
  const int g = p.parts == 1 ? blockIdx.x : blockIdx.x / p.parts, first_row = (blockIdx.x - g * p.parts) * (16 * W);
  const int h = blockIdx.y, b = blockIdx.z;
  const int64_t g0 = static_cast<int64_t>(g) * p.G;
  const int row_warp = W > 1 ? warp : 0, part = KS > 1 ? warp : 0;
  const int block_rows = static_cast<int>(p.M - g0 < p.G ? p.M - g0 : p.G) - first_row;
  if (block_rows <= 0) return;                                     // (a short last group)
  const int n_q = block_rows - row_warp * 16;                      // rows of this warp (may be <= 0)
  const int64_t m0 = g0 + first_row + row_warp * 16;

  const uint32_t ring_bytes = static_cast<uint32_t>(stages) * 2 * kRingTile<D, ROWS>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + KS * ring_bytes);
  int* words = reinterpret_cast<int*>(bars + KS * kRingBars);                          // abort, tile count
  RingSlot* list = reinterpret_cast<RingSlot*>(words + 4);
  if (warp == 0) {
    const int count = ring_list<ESZ, TMA>(list, p.kv, p.ids, b * p.i_sb + g * p.i_sg + h * p.i_sh, p.i_st, p.T, b, h, D,
                                     p.block_size, p.chunk_size, p.causal != 0, static_cast<int>(g0 / p.chunk_size));
    if (lane == 0) { words[0] = 0; words[1] = count; }
  }
  Ring<D, ROWS, TMA> ring{smem_u32(smem) + part * ring_bytes, bars + part * kRingBars, words,
                          0, stages, row_warp, W};
  ring.init();
  __syncthreads();
  ring.count = KS > 1 ? (words[1] - part + KS - 1) / KS : words[1];
  const RingSource src = kv_ring_source<ESZ>(p.kv, maps, p.B, b, h, D, p.block_size);
  const int per_block = (p.block_size + ROWS - 1) / ROWS;
  const auto tile_of = [&](int i) { return ring_tile<TMA>(list, part + i * KS, per_block, src); };
  ring.start(src, tile_of);

  // delta = sum_d O * dO of this thread's rows (lo, hi), from the fragments of both
  uint32_t q[D / 16][4], dO[D / 16][4];
  float delta[2] = {0.f, 0.f}, lse2[2];
  load_a_frag<D>(dO, p.dO + (b * p.do_sb + m0 * p.do_sm + h * p.do_sh) * ESZ, p.do_sm * ESZ, n_q);
  load_a_frag<D>(q, p.o + (b * p.o_sb + m0 * p.o_sm + h * p.o_sh) * ESZ, p.o_sm * ESZ, n_q);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack2<T>(q[kk][e]), y = unpack2<T>(dO[kk][e]);
      delta[e & 1] += x.x * y.x + x.y * y.y;
    }
  load_a_frag<D>(q, p.q + (b * p.q_sb + m0 * p.q_sm + h * p.q_sh) * ESZ, p.q_sm * ESZ, n_q);
  const int64_t bhm = (static_cast<int64_t>(b) * p.H + h) * p.M + m0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    delta[r] += __shfl_xor_sync(0xffffffffu, delta[r], 1);
    delta[r] += __shfl_xor_sync(0xffffffffu, delta[r], 2);
    const int row = gid + 8 * r;
    lse2[r] = row < n_q ? p.lse[bhm + row] * kLog2e : INFINITY;
    if (t4 == 0 && row < n_q && part == 0) p.delta[bhm + row] = delta[r];
  }

  float dq[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) dq[n][0] = dq[n][1] = dq[n][2] = dq[n][3] = 0.f;
  bool ok = true;
  for (int i = 0; i < ring.count && ok; ++i) {
    const RingTile now = tile_of(i);
    const int n = now.n, brought = now.clear;
    const int n16 = (n + 15) >> 4;
    float s[ROWS / 8][4], dp[ROWS / 8][4];
#pragma unroll
    for (int j = 0; j < ROWS / 8; ++j) {
      s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
      dp[j][0] = dp[j][1] = dp[j][2] = dp[j][3] = 0.f;
    }
    if (!ring.template wait<0>()) { ok = false; break; }
    mma_rows_t<T, D, ROWS>(s, q, ring.tile(0), n16);
    if (!ring.template wait<1>()) { ok = false; break; }
    mma_rows_t<T, D, ROWS>(dp, dO, ring.tile(1), n16);
    // V can go; K is still wanted for dQ (a ring with several readers lets go of both at the end)
    if (W == 1) ok = ring.template release<1>(i, src, tile_of);
    uint32_t ds[ROWS / 16][4];
#pragma unroll
    for (int j = 0; j < ROWS / 8; ++j) {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float pe = fast_exp2(s[j][e] * p.scale_log2 - lse2[e >> 1]);
        x[e] = 8 * j + 2 * t4 + (e & 1) < n ? pe * (dp[j][e] - delta[e >> 1]) * p.scale : 0.f;
      }
      ds[j >> 1][(j & 1) * 2] = pack2<T>(x[0], x[1]);
      ds[j >> 1][(j & 1) * 2 + 1] = pack2<T>(x[2], x[3]);
    }
    if (TMA && n < brought) ring_clear_rows<D, ROWS>(ring.tile(0), n, brought);
    mma_rows<T, D, ROWS>(dq, ds, ring.tile(0), n16);
    if (TMA && n < brought) fence_async_shared();        // the cleared rows before the next copy into this tile
    ok = (W == 1 ? ring.template release<0>(i, src, tile_of) : ring.template release<1>(i, src, tile_of)) && ok;
    ring.step();
  }
  if (!ok) atomicExch(status, NSA_ERR_CUDA);

  __syncthreads();                                        // the rings are done with: their memory stages what follows
  if constexpr (KS > 1) {
    float4* part_mem = reinterpret_cast<float4*>(smem) + (warp - 1) * (D / 8 * 32);
    if (warp > 0) {
#pragma unroll
      for (int n = 0; n < D / 8; ++n) part_mem[n * 32 + lane] = make_float4(dq[n][0], dq[n][1], dq[n][2], dq[n][3]);
    }
    __syncthreads();
    if (warp > 0) return;
    for (int k = 0; k < KS - 1; ++k)
#pragma unroll
      for (int n = 0; n < D / 8; ++n) {
        const float4 x = reinterpret_cast<const float4*>(smem)[(k * (D / 8) + n) * 32 + lane];
        dq[n][0] += x.x; dq[n][1] += x.y; dq[n][2] += x.z; dq[n][3] += x.w;
      }
    __syncwarp();
  }
  if (n_q > 0)
    store_rows<T, D>(dq, 1.f, 1.f, smem_u32(smem) + row_warp * 16 * (D * 2 + 16),
                     p.dq + (b * p.dq_sb + m0 * p.dq_sm + h * p.dq_sh) * ESZ, p.dq_sm * ESZ, n_q);
}

// ------------------------------------------------------------------------- dQ, packed tiles
template <typename T, int D>
__global__ void __launch_bounds__(256) sel_bwd_dq_packed_kernel(const BwdParams p) {
  constexpr int PITCH = D + 8;
  constexpr int ESZ = sizeof(T);
  constexpr int KK = D / 16;
  constexpr int DN = D / 8;
  extern __shared__ __align__(1024) uint8_t smem[];

  const int g = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t4 = lane & 3;
  const int rows_pad = (blockDim.x >> 5) * 16;
  const int64_t m0 = static_cast<int64_t>(g) * p.G;
  const int n_q = static_cast<int>(p.M - m0 < p.G ? p.M - m0 : p.G);
  const int q_chunk = static_cast<int>(m0 / p.chunk_size);

  T* tiles = reinterpret_cast<T*>(smem);                         // [2][2][64][PITCH]
  T* sQ = tiles + 4 * kPackedRows * PITCH;                          // [rows_pad][PITCH]
  T* sdO = sQ + rows_pad * PITCH;
  float* s_lse = reinterpret_cast<float*>(sdO + rows_pad * PITCH);
  float* s_delta = s_lse + rows_pad;
  const SlotTable st = carve_slot_table(reinterpret_cast<char*>(s_delta + rows_pad), p.T);
  auto stageK = [&](int s) { return tiles + (s * 2) * kPackedRows * PITCH; };
  auto stageV = [&](int s) { return tiles + (s * 2 + 1) * kPackedRows * PITCH; };

  const int total = build_slot_table<ESZ>(st, p.kv, p.ids, b * p.i_sb + g * p.i_sg + h * p.i_sh, p.i_st,
                                          p.T, b, h, D, p.block_size, p.chunk_size, p.causal != 0, q_chunk);

  const char* q_base = p.q + (b * p.q_sb + m0 * p.q_sm + h * p.q_sh) * ESZ;
  const char* o_base = p.o + (b * p.o_sb + m0 * p.o_sm + h * p.o_sh) * ESZ;
  const char* do_base = p.dO + (b * p.do_sb + m0 * p.do_sm + h * p.do_sh) * ESZ;
  char* dq_base = p.dq + (b * p.dq_sb + m0 * p.dq_sm + h * p.dq_sh) * ESZ;
  const int64_t bhm = (static_cast<int64_t>(b) * p.H + h) * p.M + m0;

  // delta = sum_d O * dO (one warp per row), kept in shared memory and stored for dK/dV
  for (int r = warp; r < rows_pad; r += (blockDim.x >> 5)) {
    float acc = 0.f;
    if (r < n_q) {
      const T* orow = reinterpret_cast<const T*>(o_base + r * p.o_sm * ESZ);
      const T* drow = reinterpret_cast<const T*>(do_base + r * p.do_sm * ESZ);
      for (int d = lane * 2; d < D; d += 64) {
        const float2 a = unpack2<T>(*reinterpret_cast<const uint32_t*>(orow + d));
        const float2 c = unpack2<T>(*reinterpret_cast<const uint32_t*>(drow + d));
        acc += a.x * c.x + a.y * c.y;
      }
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (lane == 0) {
      s_delta[r] = acc;
      s_lse[r] = r < n_q ? p.lse[bhm + r] * kLog2e : INFINITY;
      if (r < n_q) p.delta[bhm + r] = acc;
    }
  }

  if (total == 0) {
    for (int i = threadIdx.x; i < n_q * (D / 8); i += blockDim.x) {
      const int r = i / (D / 8), c = i % (D / 8);
      *reinterpret_cast<uint4*>(dq_base + r * p.dq_sm * ESZ + c * 16) = make_uint4(0, 0, 0, 0);
    }
    return;
  }

  const int64_t k_row_bytes = kv_row_bytes(p.kv, false, D, ESZ);
  const int64_t v_row_bytes = kv_row_bytes(p.kv, true, D, ESZ);
  const int ntiles = (total + kPackedRows - 1) / kPackedRows;

  issue_rows<T, D, PITCH>(sQ, q_base, p.q_sm * ESZ, n_q, rows_pad);
  issue_rows<T, D, PITCH>(sdO, do_base, p.do_sm * ESZ, n_q, rows_pad);
  issue_kv_tile<T, D, PITCH>(stageK(0), stageV(0), st, p.T, 0, total, k_row_bytes, v_row_bytes, p.q);
  cp_async_commit();

  float dq[DN][4];
#pragma unroll
  for (int n = 0; n < DN; ++n) { dq[n][0] = dq[n][1] = dq[n][2] = dq[n][3] = 0.f; }
  const bool warp_active = warp * 16 < n_q;
  const T* qa = sQ + (warp * 16 + (lane & 15)) * PITCH + (lane >> 4) * 8;
  const T* da = sdO + (warp * 16 + (lane & 15)) * PITCH + (lane >> 4) * 8;

  for (int i = 0; i < ntiles; ++i) {
    if (i + 1 < ntiles) {
      issue_kv_tile<T, D, PITCH>(stageK((i + 1) & 1), stageV((i + 1) & 1), st, p.T,
                                 (i + 1) * kPackedRows, total, k_row_bytes, v_row_bytes, p.q);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (warp_active) {
      const T* sK = stageK(i & 1);
      const T* sV = stageV(i & 1);
      const int nvalid = min(kPackedRows, total - i * kPackedRows);
      const int nb_off = ((lane & 7) + ((lane >> 4) << 3)) * PITCH + ((lane >> 3) & 1) * 8;
      float s[8][4], dp[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
        dp[n][0] = dp[n][1] = dp[n][2] = dp[n][3] = 0.f;
      }
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        uint32_t aq[4], ad[4];
        ldmatrix_x4(aq, qa + kk * 16);
        ldmatrix_x4(ad, da + kk * 16);
#pragma unroll
        for (int n16 = 0; n16 < 4; ++n16) {
          if (n16 * 16 < nvalid) {
            uint32_t bf[4];
            ldmatrix_x4(bf, sK + nb_off + n16 * 16 * PITCH + kk * 16);
            mma16816<T>(s[2 * n16], aq, bf[0], bf[1]);
            mma16816<T>(s[2 * n16 + 1], aq, bf[2], bf[3]);
            ldmatrix_x4(bf, sV + nb_off + n16 * 16 * PITCH + kk * 16);
            mma16816<T>(dp[2 * n16], ad, bf[0], bf[1]);
            mma16816<T>(dp[2 * n16 + 1], ad, bf[2], bf[3]);
          }
        }
      }
      const float lse0 = s_lse[warp * 16 + gid], lse1 = s_lse[warp * 16 + gid + 8];
      const float dl0 = s_delta[warp * 16 + gid], dl1 = s_delta[warp * 16 + gid + 8];
      uint32_t dsa[4][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        float ds[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = n * 8 + 2 * t4 + (e & 1);
          const float l = (e >> 1) ? lse1 : lse0;
          const float dl = (e >> 1) ? dl1 : dl0;
          const float pe = (col < nvalid) ? fast_exp2(s[n][e] * p.scale_log2 - l) : 0.f;
          ds[e] = pe * (dp[n][e] - dl) * p.scale;
        }
        dsa[n >> 1][(n & 1) * 2] = pack2<T>(ds[0], ds[1]);
        dsa[n >> 1][(n & 1) * 2 + 1] = pack2<T>(ds[2], ds[3]);
      }
      const T* kb = sK + ((lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + (lane >> 4) * 8;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j * 16 < nvalid) {
#pragma unroll
          for (int d16 = 0; d16 < D / 16; ++d16) {
            uint32_t bf[4];
            ldmatrix_x4_trans(bf, kb + j * 16 * PITCH + d16 * 16);
            mma16816<T>(dq[2 * d16], dsa[j], bf[0], bf[1]);
            mma16816<T>(dq[2 * d16 + 1], dsa[j], bf[2], bf[3]);
          }
        }
      }
    }
    __syncthreads();
  }

  if (warp_active) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = warp * 16 + gid + 8 * r;
      if (row < n_q) {
        char* drow = dq_base + row * p.dq_sm * ESZ;
#pragma unroll
        for (int n = 0; n < DN; ++n)
          *reinterpret_cast<uint32_t*>(drow + (n * 8 + 2 * t4) * ESZ) =
              pack2<T>(dq[n][2 * r], dq[n][2 * r + 1]);
      }
    }
  }
}

// --------------------------------------------------------------------------------- dK / dV
// A thread block of TW warps owns at most 16 TW tokens of one (batch, head, block) tile, 16 per warp, keeps their K and
// V rows in shared memory as A operands and streams the Q and dO rows (and LSE and delta) of the block's bucket, in
// ascending group order, through the ring, QR query rows at a time: S^T = K Q^T and dP^T = V dO^T, then dV += P^T dO
// and dK += dS^T Q.  No atomics: results are bit-reproducible.  What bounds it is the length of a step (products,
// exponentials, and the issue of the next copies: 3.5 k cycles at 16 rows, of them 1.8 k products) times the 12 warps
// per SM that two accumulators of 16 x 128 allow; with more rows a step there are 8 warps (12 at D = 64) but the K and V
// operands, the barriers and the exponentials' latency serve them all.
// 3120 queries x 12 heads, 16 of 98 blocks of 64, groups of 64, D = 128, 16 / 32 / 64 rows: 224 / 187 / 177 us; groups of
// 32: 213 / 178 / 234 us; of 80: 223 / 205 / 218 us; of 16: 207 / 270 / 359 us.  D = 64, groups of 64: 126 / 121 / 95 us; of
// 80, blocks of 64 and 128: 133 / 142 / 125 and 225 / 240 / 230 us.
template <typename T, int D, int TW, int QR, bool TMA>
__global__ void __launch_bounds__(32 * TW, (D == 128 ? (QR == 16 ? 12 : 8) : (QR == 64 ? 12 : 16)) / TW)
sel_bwd_dkv_rows_kernel(const __grid_constant__ RingMaps maps, const BwdParams p, const int tiles_per_block, const int stages,
                        int32_t* status) {
  constexpr int ESZ = sizeof(T), TROWS = 16 * TW, kList = 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t4 = lane & 3;
  const int blk = blockIdx.x / tiles_per_block, kt = blockIdx.x - blk * tiles_per_block;
  const int h = blockIdx.y, b = blockIdx.z;

  const int64_t t0 = static_cast<int64_t>(blk) * p.block_size;
  const int n_blk = p.tab.on ? p.block_size : static_cast<int>(min64(p.block_size, p.kv.n_tokens - t0));  // tokens that exist
  const int row_lo = kt * TROWS;                                  // first block row of this tile
  const int n_rows = min(TROWS, n_blk - row_lo);                  // rows this tile owns
  if (n_rows <= 0) return;
  const int64_t tok0 = t0 + row_lo;
  const int64_t out_row_bytes = static_cast<int64_t>(p.H) * D * ESZ;
  char* dk_base = p.dk + (static_cast<int64_t>(b) * p.kv.n_tokens + tok0) * out_row_bytes + h * D * ESZ;
  char* dv_base = p.dv + (static_cast<int64_t>(b) * p.kv.n_tokens + tok0) * out_row_bytes + h * D * ESZ;

  const int64_t bh = static_cast<int64_t>(b) * p.H + h;
  const int32_t* offs = p.offsets + bh * (p.NS + 1);
  const int beg = offs[blk], n_ent = offs[blk + 1] - beg;
  const int32_t* bucket = p.groups + bh * p.MG * p.T + beg;

  BlockRef br{nullptr, nullptr, 0};
  float* fdk = nullptr;
  float* fdv = nullptr;
  if (p.tab.on) {
    const auto& tb = p.tab;
    if (tb.n_blocks_per_head == nullptr || blk < tb.n_blocks_per_head[h]) {
      int64_t idx = blk, off_kv = 0, off_dkv = 0;
      if (tb.blocks_per_chunk > 0) {
        idx = blk / tb.blocks_per_chunk;
        const int64_t in_chunk = blk - idx * tb.blocks_per_chunk;
        off_kv = in_chunk * tb.in_chunk_kv_bytes;
        off_dkv = in_chunk * tb.in_chunk_dkv_bytes;
      }
      if (idx < tb.max_base) {
        const int64_t o = static_cast<int64_t>(h) * tb.base_sh + idx * tb.base_sb;
        const int64_t bk = tb.base_k[o], bv = tb.base_v[o], bdk = tb.base_dk[o], bdv = tb.base_dv[o];
        if (bk != 0 && bv != 0 && bdk != 0 && bdv != 0) {     // all four or nothing
          const int64_t okv = static_cast<int64_t>(b) * tb.batch_kv_bytes + off_kv;
          const int64_t odkv = static_cast<int64_t>(b) * tb.batch_dkv_bytes + off_dkv;
          br.k = reinterpret_cast<const char*>(static_cast<uintptr_t>(bk + okv));
          br.v = reinterpret_cast<const char*>(static_cast<uintptr_t>(bv + okv));
          br.n_vis = p.block_size;
          fdk = reinterpret_cast<float*>(static_cast<uintptr_t>(bdk + odkv)) + static_cast<int64_t>(row_lo) * tb.s_dbn;
          fdv = reinterpret_cast<float*>(static_cast<uintptr_t>(bdv + odkv)) + static_cast<int64_t>(row_lo) * tb.s_dbn;
        }
      }
    }
    if (n_ent == 0 || br.k == nullptr) return;      // the scratch of an untouched block is left as it is
  } else {
    br = resolve_block<ESZ>(p.kv, b, h, blk, D, p.block_size, 1, false, 0);
  }
  if (n_ent == 0 || br.k == nullptr) {
    for (int i = threadIdx.x; i < n_rows * (D / 8); i += 32 * TW) {
      const int r = i / (D / 8), c = i % (D / 8);
      *reinterpret_cast<uint4*>(dk_base + r * out_row_bytes + c * 16) = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(dv_base + r * out_row_bytes + c * 16) = make_uint4(0, 0, 0, 0);
    }
    return;
  }

  const uint32_t k_tile = smem_u32(smem), v_tile = k_tile + kRingTile<D, TROWS>;
  const uint32_t ring_mem = v_tile + kRingTile<D, TROWS>;
  const uint32_t ring_bytes = static_cast<uint32_t>(stages) * 2 * kRingTile<D, QR>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * kRingTile<D, TROWS> + ring_bytes);
  int* words = reinterpret_cast<int*>(bars + kRingBars);
  const float* rows32 = reinterpret_cast<const float*>(words + 4);         // [stage][LSE, delta][QR]
  int4* list = reinterpret_cast<int4*>(words + 4 + stages * 2 * QR);       // [2 kList] tiles: group, first row, rows, visible tokens

  const int subs = (p.G + QR - 1) / QR;                     // ring tiles per group
  Ring<D, QR, TMA, true> ring{ring_mem, bars, words, n_ent * subs, stages, warp, TW, p.lse, p.delta, smem_u32(rows32)};
  if (threadIdx.x == 0) words[0] = 0;
  ring.init();
  // tiles [from, from + kList) of the bucket
  const auto list_tiles = [&](int from) {
    for (int i = from + threadIdx.x; i < from + kList && i < ring.count; i += 32 * TW) {
      const int e = i / subs, r0 = (i - e * subs) * QR, g = bucket[e];
      const int64_t g0 = static_cast<int64_t>(g) * p.G;
      // rows of the tile (a short last group may leave one empty); rows of this block that the group may see
      const int n = max(0, min(QR, static_cast<int>(min64(p.G, p.M - g0)) - r0));
      int vis = n_rows;
      if (p.causal) vis = static_cast<int>(min64(vis, (g0 / p.chunk_size + 1) * p.chunk_size - tok0));
      list[i % (2 * kList)] = make_int4(g, r0, n, n > 0 ? vis : 0);
    }
  };
  list_tiles(0);
  __syncthreads();
  const RingSource src{&maps, p.q_sm * ESZ, p.do_sm * ESZ, h, b, p.G, static_cast<int>(p.M / p.G), p.B == 1};
  const int64_t bhm = bh * p.M;
  const auto tile_of = [&](int i) {
    const int4 w = list[i % (2 * kList)];
    RingTile t;
    t.unit = w.x;
    t.r0 = w.y;
    t.n = t.clear = w.z;
    const int64_t m = w.z > 0 ? static_cast<int64_t>(w.x) * p.G + w.y : 0;
    t.aux = bhm + m;
    if (!TMA) {
      t.a = reinterpret_cast<uint64_t>(p.q + (b * p.q_sb + m * p.q_sm + h * p.q_sh) * ESZ);
      t.b = reinterpret_cast<uint64_t>(p.dO + (b * p.do_sb + m * p.do_sm + h * p.do_sh) * ESZ);
    }
    return t;
  };
  ring.start(src, tile_of);

  // this block's K and V rows
  {
    const int64_t k_row = p.tab.on ? p.tab.s_bn * ESZ : kv_row_bytes(p.kv, false, D, ESZ);
    const int64_t v_row = p.tab.on ? p.tab.s_bn * ESZ : kv_row_bytes(p.kv, true, D, ESZ);
    const char* k_src = br.k + row_lo * k_row;
    const char* v_src = br.v + row_lo * v_row;
#pragma unroll 4
    for (int i = threadIdx.x; i < TROWS * (D / 8); i += 32 * TW) {
      const int r = i / (D / 8), c = i % (D / 8), bytes = r < n_rows ? 16 : 0;
      const int64_t at = r < n_rows ? r : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(k_tile + ring_at<TROWS>(r, c)), "l"(k_src + at * k_row + c * 16), "r"(bytes) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(v_tile + ring_at<TROWS>(r, c)), "l"(v_src + at * v_row + c * 16), "r"(bytes) : "memory");
    }
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncthreads();

  float dk[D / 8][4], dv[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    dk[n][0] = dk[n][1] = dk[n][2] = dk[n][3] = 0.f;
    dv[n][0] = dv[n][1] = dv[n][2] = dv[n][3] = 0.f;
  }
  bool ok = true;
  for (int i = 0; i < ring.count; ++i) {
    if (i % kList == 0 && i + kList < ring.count) {           // the copies run at most `stages` tiles ahead
      __syncthreads();
      list_tiles(i + kList);
      __syncthreads();
    }
    const int4 w = list[i % (2 * kList)];
    const int n = w.z, vis = w.w - warp * 16;                 // query rows; visible rows among this warp's
    ok = ok && ring.template wait<0>();
    if (ok && vis > 0) {
      const uint32_t qt = ring.tile(0), dt = ring.tile(1);
      constexpr int C = QR / 8;
      const int n16 = (n + 15) >> 4;
      float st[C][4], dp[C][4];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        st[j][0] = st[j][1] = st[j][2] = st[j][3] = 0.f;
        dp[j][0] = dp[j][1] = dp[j][2] = dp[j][3] = 0.f;
      }
      mma_rows_t2<T, D, TROWS, QR>(st, k_tile, qt, dp, v_tile, dt, warp * 16, n16);
      const float2* lse = reinterpret_cast<const float2*>(rows32 + ring.stage * 2 * QR) + t4;
      uint32_t pa[QR / 16][4], ds[QR / 16][4];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        const int q0 = 8 * j + 2 * t4;                         // this thread's columns: query rows q0, q0 + 1
        const float2 l = lse[j * 4], dl = lse[QR / 2 + j * 4];
        const float dls[2] = {dl.x, dl.y};
        // rows past the group's end: exp2(-inf) = 0
        const float l2[2] = {q0 < n ? l.x * kLog2e : INFINITY, q0 + 1 < n ? l.y * kLog2e : INFINITY};
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          st[j][y] = fast_exp2(st[j][y] * p.scale_log2 - l2[y & 1]);
          if (gid + 8 * (y >> 1) >= vis) st[j][y] = 0.f;
        }
        const int at = (j & 1) * 2;
        pa[j >> 1][at] = pack2<T>(st[j][0], st[j][1]);
        pa[j >> 1][at + 1] = pack2<T>(st[j][2], st[j][3]);
        ds[j >> 1][at] = pack2<T>(st[j][0] * (dp[j][0] - dls[0]) * p.scale, st[j][1] * (dp[j][1] - dls[1]) * p.scale);
        ds[j >> 1][at + 1] = pack2<T>(st[j][2] * (dp[j][2] - dls[0]) * p.scale, st[j][3] * (dp[j][3] - dls[1]) * p.scale);
      }
      mma_rows<T, D, QR>(dv, pa, dt, n16);
      mma_rows<T, D, QR>(dk, ds, qt, n16);
    }
    ok = ok && ring.template release<1>(i, src, tile_of);
    ring.step();
  }
  if (!ok) atomicExch(status, NSA_ERR_CUDA);

  __syncthreads();                                           // K and V tiles are done with: they stage the rows
  const int mine_rows = n_rows - warp * 16;
  if (mine_rows <= 0) return;
  if (p.tab.on) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = gid + 8 * r;
      if (row < mine_rows) {
        float* kr = fdk + static_cast<int64_t>(warp * 16 + row) * p.tab.s_dbn;
        float* vr = fdv + static_cast<int64_t>(warp * 16 + row) * p.tab.s_dbn;
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {
          *reinterpret_cast<float2*>(kr + n * 8 + 2 * t4) = make_float2(dk[n][2 * r], dk[n][2 * r + 1]);
          *reinterpret_cast<float2*>(vr + n * 8 + 2 * t4) = make_float2(dv[n][2 * r], dv[n][2 * r + 1]);
        }
      }
    }
    return;
  }
  const uint32_t stage = k_tile + warp * 16 * (D * 2 + 16);
  store_rows<T, D>(dk, 1.f, 1.f, stage, dk_base + warp * 16 * out_row_bytes, out_row_bytes, mine_rows);
  __syncwarp();
  store_rows<T, D>(dv, 1.f, 1.f, stage, dv_base + warp * 16 * out_row_bytes, out_row_bytes, mine_rows);
}

template <typename T, int D, int W, int KS, bool TMA>
int launch_dq_rows(const RingMaps& maps, BwdParams p, int32_t* status, cudaStream_t stream) {
  constexpr int stages = W <= 2 ? 1 : 3;                    // as in the forward
  static_assert(W * 16 * (D * 2 + 16) <= stages * 2 * kRingTile<D, 32>, "the epilogue stages its rows in the ring");
  static_assert((KS - 1) * (D / 8 * 512) <= KS * 2 * kRingTile<D, 32>, "the partial results are summed in the ring");
  const size_t smem = static_cast<size_t>(KS) * stages * 2 * kRingTile<D, 32> + KS * kRingBars * 8 + 16 +
                      ring_list_bytes(p.T);
  NSA_REQUIRE(smem <= 226 * 1024, NSA_ERR_UNSUPPORTED, "sel_bwd: T=%d needs too much shared memory", p.T);
  auto kernel = sel_bwd_dq_rows_kernel<T, D, W, KS, TMA>;
  NSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  p.parts = cdiv(p.G, 16 * W);
  kernel<<<dim3(static_cast<unsigned>(p.MG) * p.parts, p.H, p.B), 32 * W * KS, smem, stream>>>(maps, p, stages, status);
  NSA_LAUNCH_OK("sel_bwd_dq_rows_kernel");
  return NSA_OK;
}

template <typename T, int D, bool TMA>
int launch_dq_loader(const RingMaps& maps, const BwdParams& p, int32_t* st, cudaStream_t s) {
  // four warps share a ring where they fill it and a thread block of one has no better use for its registers: 4680 queries x
  // 12 heads, 16 blocks of 64, D = 64, groups of 64: 116 us, 121 us with a warp per ring; 3120 of D = 128: 294 and 131 us
  if constexpr (TMA && D == 64)
    if (p.G > 48 && p.G <= 64) return launch_dq_rows<T, D, 4, 1, TMA>(maps, p, st, s);
  if constexpr (!TMA)                       // (a warp's own cp.async loads: two share them)
    if (p.G > 16 && p.G <= 32) return launch_dq_rows<T, D, 2, 1, TMA>(maps, p, st, s);
  // a warp per 16 rows, and as many warps per list as still fit the chip at once (see the forward; two of them need more
  // registers each and pay only for the smallest groups: 624 units at D = 128, 16 blocks of 64, one / two warps: 62 / 83 us)
  const bool short_list = ring_list_bytes(p.T) <= 64 * 1024;                   // (each warp's ring needs its room)
  const int64_t units = static_cast<int64_t>(p.MG) * cdiv(p.G, 16) * p.H * p.B, room = 148 * (D == 128 ? 10 : 16);
  if (units * 4 <= room && short_list) return launch_dq_rows<T, D, 1, 4, TMA>(maps, p, st, s);
  if (units * 2 <= room && short_list && p.G <= 16) return launch_dq_rows<T, D, 1, 2, TMA>(maps, p, st, s);
  return launch_dq_rows<T, D, 1, 1, TMA>(maps, p, st, s);
}

size_t packed_dq_smem(int G, int D, int T) {
  const int rows = cdiv(G, 16) * 16;
  return static_cast<size_t>(4 * kPackedRows + 2 * rows) * (D + 8) * 2 + 2 * rows * 4 + slot_table_bytes(T);
}
template <typename T, int D>
int launch_dq_packed(const BwdParams& p, cudaStream_t stream) {
  const size_t smem = packed_dq_smem(p.G, D, p.T);
  NSA_CUDA_OK(cudaFuncSetAttribute(sel_bwd_dq_packed_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem)));
  sel_bwd_dq_packed_kernel<T, D><<<dim3(p.MG, p.H, p.B), cdiv(p.G, 16) * 32, smem, stream>>>(p);
  NSA_LAUNCH_OK("sel_bwd_dq_packed_kernel");
  return NSA_OK;
}
// Where the packed tiles are the faster ones.  3120 queries x 12 heads, 16 blocks each, packed / row kernel: D = 128, blocks
// of 1, groups of 17 / 64: 101 / 99, 37 / 56 us; of 8, groups of 48 / 65: 84 / 59, 54 / 75 us; D = 64, blocks of 8, groups of 32 / 64: 37 / 43,
// 35 / 43 us.  With cp.async loads, D = 128, blocks of 16, groups of 65 / 128: 84 / 110, 70 / 78 us; D = 64, blocks of 64, groups of
// 64 / 128: 134 / 122, 106 / 122 us.
bool packed_dq_is_better(bool tma, int G, int block_size, int D) {
  if (block_size < 4) return G > 16 || D == 64;
  if (block_size < 16) return G > (D == 64 ? 16 : tma ? 48 : 32);
  if (block_size < 24) return !tma && D == 128 && G > 64;
  if (!tma) return D == 64 && block_size >= 48 && G > 112;
  return D == 64 && G > 48 && G <= 64 && block_size > 32 && block_size <= 36;    // (whose second tile is hardly filled: 97 / 110 us)
}

template <typename T, int D>
int launch_dq(const nsa_kv_source* kv, const BwdParams& p, int32_t* st, cudaStream_t s) {
  RingMaps maps{};
  const bool tma = make_ring_maps(kv, p.B, p.H, D, p.block_size, 32, &maps);
  if (packed_dq_is_better(tma, p.G, p.block_size, D) && packed_dq_smem(p.G, D, p.T) <= 220 * 1024) return launch_dq_packed<T, D>(p, s);
  return tma ? launch_dq_loader<T, D, true>(maps, p, st, s) : launch_dq_loader<T, D, false>(maps, p, st, s);
}

template <typename T, int D, int TW, int QR, bool TMA>
int launch_dkv_rows(const RingMaps& maps, const BwdParams& p, int32_t* status, cudaStream_t stream) {
  const int tpb = cdiv(p.block_size, 16 * TW);
  constexpr int stages = TW == 2 && D == 128 ? 1 : 2;   // where registers leave the room
  constexpr size_t smem = 2 * kRingTile<D, 16 * TW> + static_cast<size_t>(stages) * (2 * kRingTile<D, QR> + 8 * QR) + kRingBars * 8 + 16 + 2 * 64 * 16;
  static_assert(TW * 16 * (D * 2 + 16) <= 2 * kRingTile<D, 16 * TW>, "the epilogue stages its rows in the K and V tiles");
  const int64_t nblk = p.NS * tpb;
  NSA_REQUIRE(nblk <= 0x7fffffff, NSA_ERR_INVALID, "sel_bwd: too many K/V tiles");
  if (nblk == 0) return NSA_OK;
  auto kernel = sel_bwd_dkv_rows_kernel<T, D, TW, QR, TMA>;
  NSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  kernel<<<dim3(static_cast<unsigned>(nblk), p.H, p.B), 32 * TW, smem, stream>>>(maps, p, tpb, stages, status);
  NSA_LAUNCH_OK("sel_bwd_dkv_rows_kernel");
  return NSA_OK;
}

template <typename T, int D, int TW, int QR>
int launch_dkv_loader(const BwdParams& p, const int64_t* qs, const int64_t* ds, int32_t* st, cudaStream_t s) {
  RingMaps maps{};
  const bool tma = make_unit_maps(&maps.a, &maps.a_tail, p.q, qs, p.B, p.M, p.H, D, p.G, QR) &&
                   make_unit_maps(&maps.b, &maps.b_tail, p.dO, ds, p.B, p.M, p.H, D, p.G, QR);
  return tma ? launch_dkv_rows<T, D, TW, QR, true>(maps, p, st, s) : launch_dkv_rows<T, D, TW, QR, false>(maps, p, st, s);
}

template <typename T, int D>
int launch_dkv(const BwdParams& p, int32_t* st, cudaStream_t s) {
  const int64_t qs[3] = {p.q_sb, p.q_sm, p.q_sh}, ds[3] = {p.do_sb, p.do_sm, p.do_sh};
  if (!p.tab.on) {
    const DkvRowsArgs a{p.q, p.dO, p.dk, p.dv, p.lse, p.delta, p.groups, p.offsets, p.kv, p.B, p.H, p.T, p.block_size, p.chunk_size,
                        p.causal, p.G, p.MG, 0, p.M, p.NS, p.scale, p.scale_log2};
    bool launched = false;
    const int rc = try_launch_sel_bwd_dkv_rows_tc(a, qs, ds, D, std::is_same<T, __half>::value ? NSA_F16 : NSA_BF16, st, s, &launched);
    if (rc || launched) return rc;
  }
  if (p.block_size <= 32) return launch_dkv_loader<T, D, 2, 16>(p, qs, ds, st, s);
  // a block of more than 32 tokens is one tile of four warps: its bucket's rows are fetched once, not per 32 tokens.  The
  // rows per step are those that fill their tiles (the figures are at the kernel).
  if (p.G <= 16) return launch_dkv_loader<T, D, 4, 16>(p, qs, ds, st, s);
  if (p.G <= 32) return launch_dkv_loader<T, D, 4, 32>(p, qs, ds, st, s);
  if (p.G <= 64 || p.G > 96) return launch_dkv_loader<T, D, 4, 64>(p, qs, ds, st, s);
  return launch_dkv_loader<T, D, 4, D == 128 ? 32 : 16>(p, qs, ds, st, s);
}

// kv: the source of the dQ kernel's K/V; nullptr: dK / dV
int dispatch_bwd(const nsa_kv_source* kv, const BwdParams& p, int dtype, int D, cudaStream_t s) {
  int32_t* st = nullptr;
  const int rc = device_status_address(&st);
  if (rc) return rc;
  if (dtype == NSA_BF16) {
    if (D == 128) return kv ? launch_dq<__nv_bfloat16, 128>(kv, p, st, s) : launch_dkv<__nv_bfloat16, 128>(p, st, s);
    return kv ? launch_dq<__nv_bfloat16, 64>(kv, p, st, s) : launch_dkv<__nv_bfloat16, 64>(p, st, s);
  }
  if (D == 128) return kv ? launch_dq<__half, 128>(kv, p, st, s) : launch_dkv<__half, 128>(p, st, s);
  return kv ? launch_dq<__half, 64>(kv, p, st, s) : launch_dkv<__half, 64>(p, st, s);
}

int run_inverted_index(const IdxParams& ip, int32_t* groups, int32_t* offsets, int32_t* counts,
                       cudaStream_t stream) {
  const int64_t rows = static_cast<int64_t>(ip.B) * ip.H;
  if (rows == 0) return NSA_OK;
  if (ip.NS == 0) {
    NSA_CUDA_OK(cudaMemsetAsync(offsets, 0, rows * sizeof(int32_t), stream));
    return NSA_OK;
  }
  const int64_t pairs = static_cast<int64_t>(ip.MG) * ip.T;
  NSA_REQUIRE(pairs <= 0x7fffffff && ip.NS <= 0x7fffffff, NSA_ERR_INVALID, "inverted_index: too many pairs or blocks");
  // One thread block per row while its pairs and their sort are little work (12 rows of 14208 pairs over 512 buckets:
  // 7.7 us); else every pass is spread over the chip (12 rows of 34944 pairs over 1092 buckets, causal: 121 us in one, 34 us
  // spread; 32 rows of 16640 pairs over 130 buckets: 139 and 39 us).
  const size_t smem = static_cast<size_t>(ip.NS + pairs) * 4;
  if (pairs <= 16384 && pairs <= kThreadSort * ip.NS && smem <= 200 * 1024 && rows <= 0x7fffffff) {
    NSA_CUDA_OK(cudaFuncSetAttribute(inv_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    inv_fused_kernel<<<static_cast<unsigned>(rows), 1024, smem, stream>>>(ip, groups, offsets);
    NSA_LAUNCH_OK("inv_fused_kernel");
    return NSA_OK;
  }
  NSA_CUDA_OK(cudaMemsetAsync(counts, 0, rows * ip.NS * sizeof(int32_t), stream));
  const dim3 grid(static_cast<unsigned>(cdiv64(pairs, kIdxThreads)), ip.H, ip.B);
  if (pairs > 0) {
    inv_pass_kernel<false><<<grid, kIdxThreads, 0, stream>>>(ip, counts, groups);
    NSA_LAUNCH_OK("inv_pass_kernel<count>");
  }
  inv_scan_kernel<<<static_cast<unsigned>(rows), 1024, 0, stream>>>(counts, offsets, ip.NS);
  NSA_LAUNCH_OK("inv_scan_kernel");
  if (pairs > 0) {
    inv_pass_kernel<true><<<grid, kIdxThreads, 0, stream>>>(ip, counts, groups);
    NSA_LAUNCH_OK("inv_pass_kernel<scatter>");
    // a bucket that a warp cannot hold takes its thread block a walk over the row: one such bucket per block, side by side
    const int per = pairs > ip.NS * (24 * kHeld) ? 1 : 32;
    inv_sort_kernel<<<dim3(static_cast<unsigned>(cdiv64(ip.NS, per)), ip.H, ip.B), 1024, 0, stream>>>(ip, offsets, groups, per);
    NSA_LAUNCH_OK("inv_sort_kernel");
  }
  return NSA_OK;
}

}  // namespace

int check_strides16(const char* what, const void* ptr, const int64_t* stride, int n, int esz);
int try_launch_sel_bwd_dq_tc(const void* q, const int64_t* q_stride, const nsa_kv_source* kv, const int32_t* ids,
                             const int64_t* idx_stride, const void* out, const int64_t* out_stride, const float* lse,
                             const void* d_out, const int64_t* do_stride, void* dq, const int64_t* dq_stride,
                             float* delta, int B, int64_t M, int H, int D, int T, int block_size, int chunk_size,
                             int causal, int G, float scale, int dtype, cudaStream_t stream, bool* launched,
                             void* pds);
int try_launch_sel_bwd_dkv_pds_tc(const void* q, const int64_t* q_stride, const nsa_kv_source* kv, const int32_t* groups,
                                  const int32_t* slots, const int32_t* offsets, const void* pds, const void* d_out,
                                  const int64_t* do_stride, void* dk, void* dv, int B, int64_t M, int H, int D, int T,
                                  int block_size, int G, int dtype, int32_t* counter, cudaStream_t stream,
                                  bool* launched);
int try_launch_sel_bwd_dkv_tc(const void* q, const int64_t* q_stride, const nsa_kv_source* kv, const int32_t* groups,
                              const int32_t* offsets, const float* lse, const float* delta, const void* d_out,
                              const int64_t* do_stride, void* dk, void* dv, int B, int64_t M, int H, int D, int T,
                              int block_size, int chunk_size, int causal, int G, float scale, int dtype,
                              int32_t* counter, cudaStream_t stream, bool* launched);

}  // namespace nsa

using namespace nsa;

extern "C" size_t nsa_inverted_index_workspace_bytes(int32_t B, int32_t H, int64_t NS) {
  return align_up(static_cast<size_t>(B) * H * NS * sizeof(int32_t), 256);
}

extern "C" int nsa_inverted_index_slots(const int32_t* block_indices, const int64_t idx_stride[4],
                                        int32_t B, int32_t MG, int32_t H, int32_t T, int64_t NS,
                                        int32_t block_size, int32_t chunk_size, int32_t causal,
                                        int32_t group_size, int32_t* groups, int32_t* offsets, int32_t* slots,
                                        void* workspace, size_t workspace_bytes, void* stream) {
  NSA_REQUIRE(B >= 0 && MG >= 0 && H >= 0 && T >= 0 && NS >= 0, NSA_ERR_INVALID, "inverted_index: negative size");
  NSA_REQUIRE(block_size > 0 && chunk_size > 0 && group_size > 0, NSA_ERR_INVALID, "inverted_index: sizes must be > 0");
  NSA_REQUIRE(H <= 65535 && B <= 65535, NSA_ERR_INVALID, "inverted_index: B and H must be <= 65535");
  NSA_REQUIRE(workspace_bytes >= nsa_inverted_index_workspace_bytes(B, H, NS), NSA_ERR_WORKSPACE,
              "inverted_index: workspace too small");
  if (B == 0 || H == 0) return NSA_OK;
  NSA_REQUIRE(block_indices && groups && offsets && (workspace || NS == 0), NSA_ERR_INVALID, "inverted_index: null pointer");
  NSA_REQUIRE(slots == nullptr || (T <= (1 << kSlotBits) && MG < (1 << (31 - kSlotBits))), NSA_ERR_UNSUPPORTED,
              "inverted_index: the slot output serves T <= %d and fewer than %d query groups", 1 << kSlotBits, 1 << (31 - kSlotBits));
  IdxParams ip{block_indices, idx_stride[0], idx_stride[1], idx_stride[2], idx_stride[3],
               B, MG, H, T, NS, block_size, chunk_size, causal, group_size, slots};
  return run_inverted_index(ip, groups, offsets, static_cast<int32_t*>(workspace),
                            static_cast<cudaStream_t>(stream));
}

extern "C" int nsa_inverted_index(const int32_t* block_indices, const int64_t idx_stride[4],
                                  int32_t B, int32_t MG, int32_t H, int32_t T, int64_t NS,
                                  int32_t block_size, int32_t chunk_size, int32_t causal,
                                  int32_t group_size, int32_t* groups, int32_t* offsets,
                                  void* workspace, size_t workspace_bytes, void* stream) {
  return nsa_inverted_index_slots(block_indices, idx_stride, B, MG, H, T, NS, block_size, chunk_size, causal, group_size,
                                  groups, offsets, nullptr, workspace, workspace_bytes, stream);
}

// workspace layout: delta f32 [B,H,M] | counts i32 [B,H,NS] | offsets i32 [B,H,NS+1] | groups i32 [B,H,MG*T]
static void bwd_ws_layout(int32_t B, int64_t M, int32_t H, int64_t NS, int64_t MG, int32_t T,
                          size_t off[5]) {
  off[0] = 0;
  off[1] = off[0] + align_up(static_cast<size_t>(B) * H * M * 4, 256);
  off[2] = off[1] + align_up(static_cast<size_t>(B) * H * NS * 4, 256);
  off[3] = off[2] + align_up(static_cast<size_t>(B) * H * (NS + 1) * 4, 256);
  off[4] = off[3] + align_up(static_cast<size_t>(B) * H * MG * T * 4, 256);
  off[5] = off[4] + 256;   // scheduling counter of the dK/dV kernel
}

extern "C" size_t nsa_sel_bwd_workspace_bytes(int32_t B, int64_t M, int32_t H, int64_t N, int32_t T,
                                              int32_t block_size, int32_t group_size) {
  if (block_size <= 0 || group_size <= 0) return 0;
  size_t off[6];
  bwd_ws_layout(B, M, H, cdiv64(N, block_size), cdiv64(M, group_size), T, off);
  return off[5];
}

static int bwd_common_checks(const char* op, int32_t B, int64_t M, int32_t H, int32_t D, int32_t T,
                             int32_t block_size, int32_t chunk_size, int32_t group_size, int32_t dtype,
                             const nsa_kv_source* kv, bool allow_ptr = false) {
  NSA_REQUIRE(B >= 0 && M >= 0 && H >= 0, NSA_ERR_INVALID, "%s: negative size", op);
  NSA_REQUIRE(group_size >= 1 && group_size <= 128, NSA_ERR_INVALID,
              "%s: group_size must be in [1,128], got %d", op, group_size);
  NSA_REQUIRE(block_size > 0 && chunk_size > 0 && T > 0, NSA_ERR_INVALID, "%s: block_size, chunk_size, T must be > 0", op);
  NSA_REQUIRE(dtype == NSA_BF16 || dtype == NSA_F16, NSA_ERR_UNSUPPORTED,
              "%s: only bf16 and fp16 are built (dtype %d)", op, dtype);
  NSA_REQUIRE(D == 64 || D == 128, NSA_ERR_UNSUPPORTED, "%s: head dim %d not built (64, 128)", op, D);
  NSA_REQUIRE(kv != nullptr, NSA_ERR_INVALID, "%s: kv source is null", op);
  NSA_REQUIRE(B <= 65535 && H <= 65535, NSA_ERR_INVALID, "%s: B and H must be <= 65535", op);
  NSA_REQUIRE(kv->mode != NSA_KV_PTR || allow_ptr, NSA_ERR_UNSUPPORTED,
              "%s: per-slot pointer tables serve the forward and dQ; dK/dV takes block base tables (nsa_sel_bwd_dkv_ptr)", op);
  NSA_REQUIRE(kv->mode != NSA_KV_PAGED || B == 1, NSA_ERR_INVALID, "%s: paged K/V needs B == 1", op);
  NSA_REQUIRE(cdiv64(M, group_size) <= 0x7fffffff && cdiv64(kv->n_tokens, block_size) <= 0x7fffffff, NSA_ERR_INVALID,
              "%s: too many groups / blocks", op);
  return NSA_OK;
}

extern "C" size_t nsa_sel_bwd_pds_bytes(int32_t B, int64_t M, int32_t H, int32_t T, int32_t group_size) {
  if (group_size <= 0 || B <= 0 || H <= 0 || T <= 0 || M <= 0) return 0;
  return static_cast<size_t>(B) * cdiv64(M, group_size) * H * T * 16384;
}

extern "C" int nsa_sel_bwd_dq(const void* q, const int64_t q_stride[3], const nsa_kv_source* kv,
                              const int32_t* block_indices, const int64_t idx_stride[4],
                              const void* out, const int64_t out_stride[3], const float* lse,
                              const void* d_out, const int64_t do_stride[3], void* dq,
                              const int64_t dq_stride[3], float* delta, int32_t B, int64_t M, int32_t H,
                              int32_t D, int32_t T, int32_t block_size, int32_t chunk_size,
                              int32_t causal, int32_t group_size, float scale, int32_t dtype,
                              void* stream) {
  return nsa_sel_bwd_dq_pds(q, q_stride, kv, block_indices, idx_stride, out, out_stride, lse, d_out, do_stride, dq,
                            dq_stride, delta, B, M, H, D, T, block_size, chunk_size, causal, group_size, scale,
                            nullptr, 0, nullptr, dtype, stream);
}

extern "C" int nsa_sel_bwd_dq_pds(const void* q, const int64_t q_stride[3], const nsa_kv_source* kv,
                                  const int32_t* block_indices, const int64_t idx_stride[4],
                                  const void* out, const int64_t out_stride[3], const float* lse,
                                  const void* d_out, const int64_t do_stride[3], void* dq,
                                  const int64_t dq_stride[3], float* delta, int32_t B, int64_t M, int32_t H,
                                  int32_t D, int32_t T, int32_t block_size, int32_t chunk_size,
                                  int32_t causal, int32_t group_size, float scale, void* pds, size_t pds_bytes,
                                  int32_t* pds_written, int32_t dtype, void* stream) {
  if (pds_written != nullptr) *pds_written = 0;
  int rc;
  if ((rc = bwd_common_checks("sel_bwd_dq", B, M, H, D, T, block_size, chunk_size, group_size, dtype, kv, true))) return rc;
  if (B == 0 || H == 0 || M == 0) return NSA_OK;
  NSA_REQUIRE((block_indices || kv->mode == NSA_KV_PTR) && lse && delta, NSA_ERR_INVALID, "sel_bwd_dq: null pointer");
  const int esz = 2;
  if ((rc = check_strides16("q", q, q_stride, 3, esz))) return rc;
  if ((rc = check_strides16("out", out, out_stride, 3, esz))) return rc;
  if ((rc = check_strides16("d_out", d_out, do_stride, 3, esz))) return rc;
  if ((rc = check_strides16("dq", dq, dq_stride, 3, esz))) return rc;
  BwdParams p{};
  if ((rc = make_kvsrc(kv, D, esz, block_size, &p.kv))) return rc;
  {
    // the page geometry runs on the tcgen05 kernel; every other shape on the general one
    bool launched = false;
    // the P / dS tiles are written only when the caller wants to know that they were (pds_written),
    // the buffer holds every (group, head, slot) pair and the lists are short enough for the storing kernel (64 slots)
    void* tiles = (pds != nullptr && pds_written != nullptr && T <= 64 &&
                   pds_bytes >= nsa_sel_bwd_pds_bytes(B, M, H, T, group_size) && aligned16(pds)) ? pds : nullptr;
    rc = try_launch_sel_bwd_dq_tc(q, q_stride, kv, block_indices, idx_stride, out, out_stride, lse, d_out, do_stride,
                                  dq, dq_stride, delta, B, M, H, D, T, block_size, chunk_size, causal, group_size,
                                  scale, dtype, static_cast<cudaStream_t>(stream), &launched, tiles);
    if (rc) return rc;
    if (launched) {
      if (tiles != nullptr) *pds_written = 1;
      return NSA_OK;
    }
  }
  p.q = static_cast<const char*>(q); p.q_sb = q_stride[0]; p.q_sm = q_stride[1]; p.q_sh = q_stride[2];
  p.o = static_cast<const char*>(out); p.o_sb = out_stride[0]; p.o_sm = out_stride[1]; p.o_sh = out_stride[2];
  p.dO = static_cast<const char*>(d_out); p.do_sb = do_stride[0]; p.do_sm = do_stride[1]; p.do_sh = do_stride[2];
  p.dq = static_cast<char*>(dq); p.dq_sb = dq_stride[0]; p.dq_sm = dq_stride[1]; p.dq_sh = dq_stride[2];
  p.lse = lse; p.delta = delta;
  p.ids = block_indices; p.i_sb = idx_stride[0]; p.i_sg = idx_stride[1]; p.i_sh = idx_stride[2]; p.i_st = idx_stride[3];
  p.B = B; p.H = H; p.T = T; p.block_size = block_size; p.chunk_size = chunk_size; p.causal = causal;
  p.G = group_size; p.MG = static_cast<int>(cdiv64(M, group_size)); p.M = M;
  p.NS = cdiv64(kv->n_tokens, block_size);
  p.scale = scale; p.scale_log2 = scale * kLog2e;
  return dispatch_bwd(kv, p, dtype, D, static_cast<cudaStream_t>(stream));
}

extern "C" int nsa_sel_bwd_dkv(const void* q, const int64_t q_stride[3], const nsa_kv_source* kv,
                               const int32_t* groups, const int32_t* offsets, const float* lse,
                               const float* delta, const void* d_out, const int64_t do_stride[3],
                               void* dk, void* dv, int32_t B, int64_t M, int32_t H, int32_t D, int32_t T,
                               int32_t block_size, int32_t chunk_size, int32_t causal,
                               int32_t group_size, float scale, void* workspace, size_t workspace_bytes,
                               int32_t dtype, void* stream) {
  return nsa_sel_bwd_dkv_pds(q, q_stride, kv, groups, offsets, nullptr, nullptr, 0, lse, delta, d_out, do_stride, dk, dv,
                             B, M, H, D, T, block_size, chunk_size, causal, group_size, scale, workspace,
                             workspace_bytes, dtype, stream);
}

extern "C" int nsa_sel_bwd_dkv_pds(const void* q, const int64_t q_stride[3], const nsa_kv_source* kv,
                                   const int32_t* groups, const int32_t* offsets, const int32_t* slots,
                                   const void* pds, size_t pds_bytes, const float* lse,
                                   const float* delta, const void* d_out, const int64_t do_stride[3],
                                   void* dk, void* dv, int32_t B, int64_t M, int32_t H, int32_t D, int32_t T,
                                   int32_t block_size, int32_t chunk_size, int32_t causal,
                                   int32_t group_size, float scale, void* workspace, size_t workspace_bytes,
                                   int32_t dtype, void* stream) {
  int rc;
  if ((rc = bwd_common_checks("sel_bwd_dkv", B, M, H, D, T, block_size, chunk_size, group_size, dtype, kv))) return rc;
  const int64_t N = kv->n_tokens;
  if (B == 0 || H == 0 || N == 0) return NSA_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int esz = 2;
  NSA_REQUIRE(dk && dv && aligned16(dk) && aligned16(dv), NSA_ERR_LAYOUT, "sel_bwd_dkv: dk/dv must be 16-byte aligned");
  if (M == 0) {
    NSA_CUDA_OK(cudaMemsetAsync(dk, 0, static_cast<size_t>(B) * N * H * D * esz, s));
    NSA_CUDA_OK(cudaMemsetAsync(dv, 0, static_cast<size_t>(B) * N * H * D * esz, s));
    return NSA_OK;
  }
  NSA_REQUIRE(groups && offsets && lse && delta, NSA_ERR_INVALID, "sel_bwd_dkv: null pointer");
  if ((rc = check_strides16("q", q, q_stride, 3, esz))) return rc;
  if ((rc = check_strides16("d_out", d_out, do_stride, 3, esz))) return rc;
  BwdParams p{};
  if ((rc = make_kvsrc(kv, D, esz, block_size, &p.kv))) return rc;
  {
    bool launched = false;
    int32_t* counter = (workspace != nullptr && workspace_bytes >= 256) ? static_cast<int32_t*>(workspace) : nullptr;
    if (pds != nullptr && slots != nullptr) {
      // P and dS of every pair were stored by the dQ kernel: stream them instead of recomputing S and dP
      NSA_REQUIRE(pds_bytes >= nsa_sel_bwd_pds_bytes(B, M, H, T, group_size) && aligned16(pds), NSA_ERR_WORKSPACE,
                  "sel_bwd_dkv: the P/dS buffer is too small or misaligned");
      rc = try_launch_sel_bwd_dkv_pds_tc(q, q_stride, kv, groups, slots, offsets, pds, d_out, do_stride, dk, dv, B, M, H,
                                         D, T, block_size, group_size, dtype, counter, s, &launched);
      if (rc) return rc;
      if (launched) return NSA_OK;
      NSA_REQUIRE(false, NSA_ERR_UNSUPPORTED, "sel_bwd_dkv: the stored-probabilities kernel does not serve this call");
    }
    rc = try_launch_sel_bwd_dkv_tc(q, q_stride, kv, groups, offsets, lse, delta, d_out, do_stride, dk, dv, B, M, H, D,
                                   T, block_size, chunk_size, causal, group_size, scale, dtype, counter, s, &launched);
    if (rc) return rc;
    if (launched) return NSA_OK;
  }
  p.q = static_cast<const char*>(q); p.q_sb = q_stride[0]; p.q_sm = q_stride[1]; p.q_sh = q_stride[2];
  p.dO = static_cast<const char*>(d_out); p.do_sb = do_stride[0]; p.do_sm = do_stride[1]; p.do_sh = do_stride[2];
  p.dk = static_cast<char*>(dk); p.dv = static_cast<char*>(dv);
  p.lse = lse; p.delta = const_cast<float*>(delta);
  p.groups = groups; p.offsets = offsets;
  p.B = B; p.H = H; p.T = T; p.block_size = block_size; p.chunk_size = chunk_size; p.causal = causal;
  p.G = group_size; p.MG = static_cast<int>(cdiv64(M, group_size)); p.M = M; p.NS = cdiv64(N, block_size);
  p.scale = scale; p.scale_log2 = scale * kLog2e;
  return dispatch_bwd(nullptr, p, dtype, D, s);
}

extern "C" int nsa_sel_bwd_dkv_ptr(const void* q, const int64_t q_stride[3], const int64_t* base_k,
                                   const int64_t* base_v, const int64_t* base_dk, const int64_t* base_dv,
                                   const int64_t base_stride[2], int32_t max_base,
                                   const int32_t* n_blocks_per_head, int64_t batch_stride_kv_bytes,
                                   int64_t batch_stride_dkv_bytes, int64_t stride_bn, int64_t stride_dbn,
                                   int32_t blocks_per_chunk, int64_t in_chunk_block_bytes_kv,
                                   int64_t in_chunk_block_bytes_dkv, const int32_t* groups,
                                   const int32_t* offsets, int64_t NS, const float* lse, const float* delta,
                                   const void* d_out, const int64_t do_stride[3], int32_t B, int64_t M,
                                   int32_t H, int32_t D, int32_t T, int32_t block_size, int32_t group_size,
                                   float scale, int32_t dtype, void* stream) {
  nsa_kv_source dummy{};
  dummy.mode = NSA_KV_DENSE;
  dummy.n_tokens = NS * block_size;
  int rc;
  if ((rc = bwd_common_checks("sel_bwd_dkv_ptr", B, M, H, D, T, block_size, 1, group_size, dtype, &dummy))) return rc;
  if (B == 0 || H == 0 || M == 0 || NS == 0) return NSA_OK;
  NSA_REQUIRE(base_k && base_v && base_dk && base_dv && base_stride, NSA_ERR_INVALID, "sel_bwd_dkv_ptr: null base table");
  NSA_REQUIRE(groups && offsets && lse && delta, NSA_ERR_INVALID, "sel_bwd_dkv_ptr: null pointer");
  NSA_REQUIRE(max_base > 0, NSA_ERR_INVALID, "sel_bwd_dkv_ptr: max_base must be > 0");
  NSA_REQUIRE(blocks_per_chunk >= 0, NSA_ERR_INVALID, "sel_bwd_dkv_ptr: blocks_per_chunk must be >= 0");
  NSA_REQUIRE(blocks_per_chunk == 0 || (in_chunk_block_bytes_kv > 0 && in_chunk_block_bytes_dkv > 0), NSA_ERR_INVALID,
              "sel_bwd_dkv_ptr: chunk-level bases need in_chunk_block_bytes_kv/dkv > 0");
  NSA_REQUIRE(stride_bn > 0 && (stride_bn * 2) % 16 == 0, NSA_ERR_LAYOUT,
              "sel_bwd_dkv_ptr: K/V token stride must be a positive multiple of 16 bytes");
  NSA_REQUIRE(stride_dbn >= D && stride_dbn % 2 == 0, NSA_ERR_LAYOUT,
              "sel_bwd_dkv_ptr: stride_dbn must be the fp32 scratch stride (>= D, even)");
  const int esz = 2;
  if ((rc = check_strides16("q", q, q_stride, 3, esz))) return rc;
  if ((rc = check_strides16("d_out", d_out, do_stride, 3, esz))) return rc;
  BwdParams p{};
  p.kv.mode = NSA_KV_DENSE;
  p.kv.n_tokens = NS * block_size;
  p.q = static_cast<const char*>(q); p.q_sb = q_stride[0]; p.q_sm = q_stride[1]; p.q_sh = q_stride[2];
  p.dO = static_cast<const char*>(d_out); p.do_sb = do_stride[0]; p.do_sm = do_stride[1]; p.do_sh = do_stride[2];
  p.lse = lse; p.delta = const_cast<float*>(delta);
  p.groups = groups; p.offsets = offsets;
  p.B = B; p.H = H; p.T = T; p.block_size = block_size; p.chunk_size = 1; p.causal = 0;
  p.G = group_size; p.MG = static_cast<int>(cdiv64(M, group_size)); p.M = M; p.NS = NS;
  p.scale = scale; p.scale_log2 = scale * kLog2e;
  p.tab.on = 1;
  p.tab.base_k = base_k; p.tab.base_v = base_v; p.tab.base_dk = base_dk; p.tab.base_dv = base_dv;
  p.tab.base_sh = base_stride[0]; p.tab.base_sb = base_stride[1]; p.tab.max_base = max_base;
  p.tab.n_blocks_per_head = n_blocks_per_head;
  p.tab.batch_kv_bytes = batch_stride_kv_bytes; p.tab.batch_dkv_bytes = batch_stride_dkv_bytes;
  p.tab.in_chunk_kv_bytes = in_chunk_block_bytes_kv; p.tab.in_chunk_dkv_bytes = in_chunk_block_bytes_dkv;
  p.tab.blocks_per_chunk = blocks_per_chunk;
  p.tab.s_bn = stride_bn; p.tab.s_dbn = stride_dbn;
  return dispatch_bwd(nullptr, p, dtype, D, static_cast<cudaStream_t>(stream));
}

extern "C" int nsa_sel_bwd(const void* q, const int64_t q_stride[3], const nsa_kv_source* kv,
                           const int32_t* block_indices, const int64_t idx_stride[4],
                           const void* out, const int64_t out_stride[3], const float* lse,
                           const void* d_out, const int64_t do_stride[3], void* dq,
                           const int64_t dq_stride[3], void* dk, void* dv, int32_t B, int64_t M,
                           int32_t H, int32_t D, int32_t T, int32_t block_size, int32_t chunk_size,
                           int32_t causal, int32_t group_size, float scale, void* workspace,
                           size_t workspace_bytes, int32_t dtype, void* stream) {
  int rc;
  if ((rc = bwd_common_checks("sel_bwd", B, M, H, D, T, block_size, chunk_size, group_size, dtype, kv))) return rc;
  const int64_t N = kv->n_tokens;
  const int64_t NS = cdiv64(N, block_size), MG = cdiv64(M, group_size);
  NSA_REQUIRE(workspace_bytes >= nsa_sel_bwd_workspace_bytes(B, M, H, N, T, block_size, group_size),
              NSA_ERR_WORKSPACE, "sel_bwd: workspace too small");
  if (B == 0 || H == 0) return NSA_OK;
  NSA_REQUIRE(workspace != nullptr, NSA_ERR_INVALID, "sel_bwd: workspace is null");
  size_t off[6];
  bwd_ws_layout(B, M, H, NS, MG, T, off);
  char* ws = static_cast<char*>(workspace);
  float* delta = reinterpret_cast<float*>(ws + off[0]);
  int32_t* counts = reinterpret_cast<int32_t*>(ws + off[1]);
  int32_t* offsets = reinterpret_cast<int32_t*>(ws + off[2]);
  int32_t* groups = reinterpret_cast<int32_t*>(ws + off[3]);
  if (M > 0) {
    NSA_REQUIRE(block_indices != nullptr, NSA_ERR_INVALID, "sel_bwd: block_indices is null");
    IdxParams ip{block_indices, idx_stride[0], idx_stride[1], idx_stride[2], idx_stride[3],
                 B, static_cast<int>(MG), H, T, NS, block_size, chunk_size, causal, group_size, nullptr};
    if ((rc = run_inverted_index(ip, groups, offsets, counts, static_cast<cudaStream_t>(stream)))) return rc;
    if ((rc = nsa_sel_bwd_dq(q, q_stride, kv, block_indices, idx_stride, out, out_stride, lse, d_out, do_stride,
                             dq, dq_stride, delta, B, M, H, D, T, block_size, chunk_size, causal, group_size,
                             scale, dtype, stream))) return rc;
  }
  return nsa_sel_bwd_dkv(q, q_stride, kv, groups, offsets, lse, delta, d_out, do_stride, dk, dv, B, M, H, D, T,
                         block_size, chunk_size, causal, group_size, scale, ws + off[4], 256, dtype, stream);
}
