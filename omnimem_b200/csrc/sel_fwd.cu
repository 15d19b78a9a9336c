// Selection attention forward, general geometry (any block size, group size <= 128, D in {64, 128}, bf16 / fp16):
// a thread block is one (batch, query group, head) or a part of its rows; a warp owns 16 query rows; the K/V rows come in
// tiles of one block each through a ring (sel_rows.cuh) or packed into tiles of 64 (sel_packed.cuh); S = Q K^T and
// O += P V run on mma.sync m16n8k16 with fp32 accumulation and an online softmax in the exp2 domain.
#include "sel_packed.cuh"
#include "sel_rows.cuh"

namespace nsa {
namespace {

struct FwdParams {
  const char* q;
  int64_t q_sb, q_sm, q_sh;
  char* out;
  int64_t o_sb, o_sm, o_sh;
  float* lse;               // [B,H,M]
  const int32_t* ids;
  int64_t i_sb, i_sg, i_sh, i_st;
  KVSrc kv;
  int B, H, T, block_size, chunk_size, causal, G;
  int parts;                // thread blocks that share a group's rows
  int64_t M;
  float scale_log2;
};

// W warps of 16 query rows each share one ring; p.parts such thread blocks take a group; with W = 1 the tiles of the list may be dealt out to KS warps
// with rings of their own, whose partial results are merged at the end (few groups on many SMs).
// What bounds it for small groups: the gathered K/V rows, which every list fetches for itself, through the L2 to SM
// path.  32760 queries x 12 heads, 15-query groups, 16 blocks of 30 tokens: 397 us = 16 TB/s of rows against the
// 18 TB/s that bulk copies reach here (5911 us with one warp per 70 KB thread block, 124 TF -> 243 TF of products).
// One K/V stage and 12 warps per SM: 397 us; two stages and 7 warps: 661 us; 16- or 32-byte loads straight into
// fragments, no shared memory: 780 us.
// A group of more than 64 queries is dealt out to thread blocks of one warp that walk the list each for itself: 3120 queries
// x 12 heads, 16 blocks of 64, D = 128, groups of 48 / 64 / 128: 117 / 116 / 117 us; with four warps per ring 131 / 131 / 131 us,
// with eight 470 / 320 / 247 us.  9360 queries, causal, groups of 64 / 128: 201 / 200 us; with four warps 193 / 196 us.
template <typename T, int D, int W, int KS, bool TMA>
__global__ void __launch_bounds__(32 * W * KS) sel_fwd_rows_kernel(const __grid_constant__ RingMaps maps, const FwdParams p,
                                                                   const int stages, int32_t* status) {
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

  float o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  float m_ref[2] = {-INFINITY, -INFINITY}, l_i[2] = {0.f, 0.f};
  uint32_t q[D / 16][4];
  load_a_frag<D>(q, p.q + (b * p.q_sb + m0 * p.q_sm + h * p.q_sh) * ESZ, p.q_sm * ESZ, n_q);

  bool ok = true;
  for (int i = 0; i < ring.count && ok; ++i) {
    const RingTile now = tile_of(i);
    const int n = now.n, brought = now.clear;
    if (!ring.template wait<0>()) { ok = false; break; }
    const int n16 = (n + 15) >> 4;
    float s[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    mma_rows_t<T, D, ROWS>(s, q, ring.tile(0), n16);
    ok = ring.template release<0>(i, src, tile_of);
    // scaled first, then masked: the scale may be zero or negative
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[j][e] *= p.scale_log2;
    if (n < ROWS) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (8 * j + 2 * t4 + (e & 1) >= n) s[j][e] = -INFINITY;
    }
    float mx[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) mx[r] = fmaxf(mx[r], fmaxf(s[j][2 * r], s[j][2 * r + 1]));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    }
    // the accumulator is rescaled only when a maximum has grown by more than 2^8 (and in the first step)
    if (__any_sync(0xffffffffu, mx[0] > m_ref[0] + 8.f || mx[1] > m_ref[1] + 8.f)) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m_new = fmaxf(m_ref[r], mx[r]);
        const float corr = fast_exp2(m_ref[r] - m_new);
        m_ref[r] = m_new;
        l_i[r] *= corr;
#pragma unroll
        for (int d = 0; d < D / 8; ++d) { o[d][2 * r] *= corr; o[d][2 * r + 1] *= corr; }
      }
    }
    uint32_t pa[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float e[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) e[x] = fast_exp2(s[j][x] - m_ref[x >> 1]);
      l_i[0] += e[0] + e[1];
      l_i[1] += e[2] + e[3];
      pa[j >> 1][(j & 1) * 2] = pack2<T>(e[0], e[1]);
      pa[j >> 1][(j & 1) * 2 + 1] = pack2<T>(e[2], e[3]);
    }
    ok = ring.template wait<1>() && ok;
    if (!ok) break;
    if (TMA && n < brought) ring_clear_rows<D, ROWS>(ring.tile(1), n, brought);
    mma_rows<T, D, ROWS>(o, pa, ring.tile(1), n16);
    if (TMA && n < brought) fence_async_shared();            // the cleared rows before the next copy into this tile
    ok = ring.template release<1>(i, src, tile_of);
    ring.step();
  }
  if (!ok) atomicExch(status, NSA_ERR_CUDA);

#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l_i[r] += __shfl_xor_sync(0xffffffffu, l_i[r], 1);
    l_i[r] += __shfl_xor_sync(0xffffffffu, l_i[r], 2);
  }
  __syncthreads();                                        // the rings are done with: their memory stages what follows
  if constexpr (KS > 1) {
    // partial sums of warps 1 .. KS - 1 in fragment order: [D / 8][32 lanes] float4, then maxima and sums
    float* part_mem = reinterpret_cast<float*>(smem) + (warp - 1) * (D / 8 * 128 + 128);
    if (warp > 0) {
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        reinterpret_cast<float4*>(part_mem)[n * 32 + lane] = make_float4(o[n][0], o[n][1], o[n][2], o[n][3]);
      reinterpret_cast<float4*>(part_mem + D / 8 * 128)[lane] = make_float4(m_ref[0], m_ref[1], l_i[0], l_i[1]);
    }
    __syncthreads();
    if (warp > 0) return;
    for (int k = 0; k < KS - 1; ++k) {
      const float* from = reinterpret_cast<const float*>(smem) + k * (D / 8 * 128 + 128);
      const float4 ml = reinterpret_cast<const float4*>(from + D / 8 * 128)[lane];
      const float m_new[2] = {fmaxf(m_ref[0], ml.x), fmaxf(m_ref[1], ml.y)};
      float mine[2], theirs[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m = m_new[r] == -INFINITY ? 0.f : m_new[r];   // neither part saw a key: all sums are 0
        mine[r] = fast_exp2(m_ref[r] - m);
        theirs[r] = fast_exp2((r ? ml.y : ml.x) - m);
        l_i[r] = l_i[r] * mine[r] + (r ? ml.w : ml.z) * theirs[r];
        m_ref[r] = m_new[r];
      }
#pragma unroll
      for (int n = 0; n < D / 8; ++n) {
        const float4 x = reinterpret_cast<const float4*>(from)[n * 32 + lane];
        o[n][0] = o[n][0] * mine[0] + x.x * theirs[0];
        o[n][1] = o[n][1] * mine[0] + x.y * theirs[0];
        o[n][2] = o[n][2] * mine[1] + x.z * theirs[1];
        o[n][3] = o[n][3] * mine[1] + x.w * theirs[1];
      }
    }
    __syncwarp();
  }
  if (n_q <= 0) return;
  const float inv[2] = {l_i[0] > 0.f ? 1.f / l_i[0] : 0.f, l_i[1] > 0.f ? 1.f / l_i[1] : 0.f};
  store_rows<T, D>(o, inv[0], inv[1], smem_u32(smem) + row_warp * 16 * (D * 2 + 16),
                   p.out + (b * p.o_sb + m0 * p.o_sm + h * p.o_sh) * ESZ, p.o_sm * ESZ, n_q);
  if (t4 == 0) {
    float* lse = p.lse + (static_cast<int64_t>(b) * p.H + h) * p.M + m0;
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (gid + 8 * r < n_q) lse[gid + 8 * r] = l_i[r] > 0.f ? (m_ref[r] + log2f(l_i[r])) * kLn2 : -INFINITY;
  }
}

// ------------------------------------------------------------------------------ packed tiles
template <typename T, int D>
__global__ void __launch_bounds__(256) sel_fwd_packed_kernel(const FwdParams p) {
  constexpr int PITCH = D + 8;
  constexpr int ESZ = sizeof(T);
  constexpr int KK = D / 16;     // k-steps of S = Q K^T
  constexpr int DN = D / 8;      // n8 tiles of O
  extern __shared__ __align__(1024) uint8_t smem[];

  const int g = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t4 = lane & 3;
  const int64_t m0 = static_cast<int64_t>(g) * p.G;
  const int n_q = static_cast<int>(p.M - m0 < p.G ? p.M - m0 : p.G);
  const int q_chunk = static_cast<int>(m0 / p.chunk_size);

  T* tiles = reinterpret_cast<T*>(smem);                       // [2][2][64][PITCH]
  const SlotTable st = carve_slot_table(reinterpret_cast<char*>(smem) + 4 * kPackedRows * PITCH * ESZ, p.T);
  auto stageK = [&](int s) { return tiles + (s * 2) * kPackedRows * PITCH; };
  auto stageV = [&](int s) { return tiles + (s * 2 + 1) * kPackedRows * PITCH; };

  const int total = build_slot_table<ESZ>(st, p.kv, p.ids, b * p.i_sb + g * p.i_sg + h * p.i_sh, p.i_st,
                                          p.T, b, h, D, p.block_size, p.chunk_size, p.causal != 0, q_chunk);

  char* out_row0 = p.out + (b * p.o_sb + m0 * p.o_sm + h * p.o_sh) * ESZ;
  float* lse_row0 = p.lse + (static_cast<int64_t>(b) * p.H + h) * p.M + m0;
  if (total == 0) {  // no visible key: O = 0, LSE = -inf
    for (int i = threadIdx.x; i < n_q * (D / 8); i += blockDim.x) {
      const int r = i / (D / 8), c = i % (D / 8);
      *reinterpret_cast<uint4*>(out_row0 + r * p.o_sm * ESZ + c * 16) = make_uint4(0, 0, 0, 0);
    }
    for (int r = threadIdx.x; r < n_q; r += blockDim.x) lse_row0[r] = -INFINITY;
    return;
  }

  const int64_t k_row_bytes = kv_row_bytes(p.kv, false, D, ESZ);
  const int64_t v_row_bytes = kv_row_bytes(p.kv, true, D, ESZ);
  const char* q_base = p.q + (b * p.q_sb + m0 * p.q_sm + h * p.q_sh) * ESZ;
  const int ntiles = (total + kPackedRows - 1) / kPackedRows;
  const int rows_pad = (blockDim.x >> 5) * 16;

  // Q goes through stage 1 (128 rows) while tile 0 lands in stage 0.
  issue_rows<T, D, PITCH>(stageK(1), q_base, p.q_sm * ESZ, n_q, rows_pad);
  cp_async_commit();
  issue_kv_tile<T, D, PITCH>(stageK(0), stageV(0), st, p.T, 0, total, k_row_bytes, v_row_bytes, p.q);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();

  uint32_t qf[KK][4];
  {
    const T* sQ = stageK(1) + (warp * 16 + (lane & 15)) * PITCH + (lane >> 4) * 8;
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) ldmatrix_x4(qf[kk], sQ + kk * 16);
  }
  __syncthreads();

  float o[DN][4];
#pragma unroll
  for (int n = 0; n < DN; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
  float m_i[2] = {-INFINITY, -INFINITY};
  float l_i[2] = {0.f, 0.f};
  const bool warp_active = warp * 16 < n_q;

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
      float s[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) { s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f; }
      const T* kb = sK + ((lane & 7) + ((lane >> 4) << 3)) * PITCH + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
#pragma unroll
        for (int n16 = 0; n16 < 4; ++n16) {
          if (n16 * 16 < nvalid) {
            uint32_t bf[4];
            ldmatrix_x4(bf, kb + n16 * 16 * PITCH + kk * 16);
            mma16816<T>(s[2 * n16], qf[kk], bf[0], bf[1]);
            mma16816<T>(s[2 * n16 + 1], qf[kk], bf[2], bf[3]);
          }
        }
      }
      // mask + online softmax (rows gid and gid + 8), exp2 domain
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int n = 0; n < 8; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = n * 8 + 2 * t4 + (e & 1);
          const float v = (col < nvalid) ? s[n][e] * p.scale_log2 : -INFINITY;
          s[n][e] = v;
          mx[e >> 1] = fmaxf(mx[e >> 1], v);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
        const float m_new = fmaxf(m_i[r], mx[r]);   // finite: every tile has a valid column
        const float corr = fast_exp2(m_i[r] - m_new);
        m_i[r] = m_new;
        l_i[r] *= corr;
#pragma unroll
        for (int n = 0; n < DN; ++n) { o[n][2 * r] *= corr; o[n][2 * r + 1] *= corr; }
      }
      uint32_t pa[4][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const float p0 = fast_exp2(s[n][0] - m_i[0]);
        const float p1 = fast_exp2(s[n][1] - m_i[0]);
        const float p2 = fast_exp2(s[n][2] - m_i[1]);
        const float p3 = fast_exp2(s[n][3] - m_i[1]);
        l_i[0] += p0 + p1;
        l_i[1] += p2 + p3;
        pa[n >> 1][(n & 1) * 2] = pack2<T>(p0, p1);
        pa[n >> 1][(n & 1) * 2 + 1] = pack2<T>(p2, p3);
      }
      const T* vb = sV + ((lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + (lane >> 4) * 8;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j * 16 < nvalid) {
#pragma unroll
          for (int d16 = 0; d16 < D / 16; ++d16) {
            uint32_t bf[4];
            ldmatrix_x4_trans(bf, vb + j * 16 * PITCH + d16 * 16);
            mma16816<T>(o[2 * d16], pa[j], bf[0], bf[1]);
            mma16816<T>(o[2 * d16 + 1], pa[j], bf[2], bf[3]);
          }
        }
      }
    }
    __syncthreads();
  }

  if (warp_active) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_i[r] += __shfl_xor_sync(0xffffffffu, l_i[r], 1);
      l_i[r] += __shfl_xor_sync(0xffffffffu, l_i[r], 2);
      const int row = warp * 16 + gid + 8 * r;
      if (row < n_q) {
        const float inv = l_i[r] > 0.f ? 1.f / l_i[r] : 0.f;
        char* orow = out_row0 + row * p.o_sm * ESZ;
#pragma unroll
        for (int n = 0; n < DN; ++n)
          *reinterpret_cast<uint32_t*>(orow + (n * 8 + 2 * t4) * ESZ) =
              pack2<T>(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
        if (t4 == 0)
          lse_row0[row] = l_i[r] > 0.f ? (m_i[r] + log2f(l_i[r])) * kLn2 : -INFINITY;
      }
    }
  }
}

size_t packed_fwd_smem(int D, int T) { return 4 * kPackedRows * (D + 8) * 2 + slot_table_bytes(T); }
template <typename T, int D>
int launch_packed(const FwdParams& p, int MG, cudaStream_t stream) {
  const size_t smem = packed_fwd_smem(D, p.T);
  NSA_CUDA_OK(cudaFuncSetAttribute(sel_fwd_packed_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem)));
  sel_fwd_packed_kernel<T, D><<<dim3(MG, p.H, p.B), cdiv(p.G, 16) * 32, smem, stream>>>(p);
  NSA_LAUNCH_OK("sel_fwd_packed_kernel");
  return NSA_OK;
}
// Where the packed tiles are the faster ones.  3120 queries x 12 heads, 16 blocks each, packed / row kernel: D = 128, blocks
// of 1 and groups of 8 / 64: 50 / 50, 15 / 50 us; blocks of 8, groups of 32 / 64 / 128: 53 / 50, 29 / 50, 33 / 51 us; of 16: 98 / 50,
// 51 / 50, 55 / 51 us; D = 64, blocks of 16, groups of 48 / 64: 33 / 27, 21 / 27 us.  With cp.async loads, D = 128, blocks of 16, groups
// of 32 / 64: 99 / 65, 50 / 60 us; of 64, groups of 64 / 128: 174 / 148, 131 / 143 us; D = 64: 64 / 63, 54 / 63 us.
bool packed_fwd_is_better(bool tma, int G, int block_size, int D) {
  if (block_size < 4) return G >= 8 || D == 64 || !tma;
  if (block_size < 16) return G > (tma && D == 128 ? 32 : 16);
  if (block_size < 24) return tma ? D == 64 && G > 48 : G > (D == 64 ? 32 : 48);
  if (!tma) return G >= (D == 64 ? 60 : 113);
  // by the rows that a block leaves free in its last tile: blocks of 33, D = 64, groups of 64: 65 / 99 us; D = 128, groups of
  // 128: 112 / 180 us
  const int rows = cdiv(block_size, 32) * 32;
  if (D == 128) return G > 96 && rows * 5 >= block_size * 8;
  return rows * 5 >= block_size * 6 ? G > 48 && (G <= 72 || G > 96) : G > 112 && block_size > 32;   // (64, 128: 80 / 93 us)
}

// -------------------------------------------------------------------------------------- launch
template <typename T, int D, int W, int KS, bool TMA>
int launch_rows(const RingMaps& maps, FwdParams p, int MG, int32_t* status, cudaStream_t stream) {
  // stages: one for a single warp (the thread blocks that share an SM are the depth), three where several warps wait for
  // the same ring; never less than the epilogue's staging needs
  constexpr int stages = W <= 2 ? 1 : 3;
  static_assert(W * 16 * (D * 2 + 16) <= stages * 2 * kRingTile<D, 32>, "the epilogue stages its rows in the ring");
  static_assert((KS - 1) * (D / 8 * 128 + 128) * 4 <= KS * 2 * kRingTile<D, 32>, "the partial results are merged in the ring");
  const size_t smem = static_cast<size_t>(KS) * stages * 2 * kRingTile<D, 32> + KS * kRingBars * 8 + 16 +
                      ring_list_bytes(p.T);
  NSA_REQUIRE(smem <= 226 * 1024, NSA_ERR_UNSUPPORTED, "sel_fwd: T=%d needs too much shared memory", p.T);
  auto kernel = sel_fwd_rows_kernel<T, D, W, KS, TMA>;
  NSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  p.parts = cdiv(p.G, 16 * W);
  kernel<<<dim3(static_cast<unsigned>(MG) * p.parts, p.H, p.B), 32 * W * KS, smem, stream>>>(maps, p, stages, status);
  NSA_LAUNCH_OK("sel_fwd_rows_kernel");
  return NSA_OK;
}

template <typename T, int D, bool TMA>
int launch_loader(const RingMaps& maps, const FwdParams& p, int MG, int32_t* st, cudaStream_t s) {
  // A warp per 16 rows, and as many warps per list as still fit the chip at once: 12 warps per SM at D = 128 (registers),
  // 16 at D = 64.  Measured, D = 128, 16 blocks of 30, one / two / four warps per list: 384 lists 22.7 / 18.5 / 15.5 us,
  // 768 lists 25.9 / 23.0 / 28.0 us, 1248 lists 31.6 / 40.8 / 41.0 us.  With more lists than that two or four warps share a
  // ring where they fill it, and always where the loads are a warp's own (cp.async).
  const bool short_list = ring_list_bytes(p.T) <= 64 * 1024;                   // (each warp's ring needs its room)
  const int64_t units = static_cast<int64_t>(MG) * cdiv(p.G, 16) * p.H * p.B, room = 148 * (D == 128 ? 12 : 16);
  if (!TMA || units * 2 > room || !short_list) {
    if (p.G > 16 && p.G <= 32) return launch_rows<T, D, 2, 1, TMA>(maps, p, MG, st, s);
    if (TMA ? p.G > 48 && p.G <= 64 : p.G > 32) return launch_rows<T, D, 4, 1, TMA>(maps, p, MG, st, s);
  }
  if (units * 4 <= room && short_list) return launch_rows<T, D, 1, 4, TMA>(maps, p, MG, st, s);
  if (units * 2 <= room && short_list) return launch_rows<T, D, 1, 2, TMA>(maps, p, MG, st, s);
  return launch_rows<T, D, 1, 1, TMA>(maps, p, MG, st, s);
}

template <typename T, int D>
int launch(const nsa_kv_source* kv, const FwdParams& p, int MG, cudaStream_t s) {
  int32_t* st = nullptr;
  int rc = device_status_address(&st);
  if (rc) return rc;
  RingMaps maps{};
  const bool tma = make_ring_maps(kv, p.B, p.H, D, p.block_size, 32, &maps);
  if (packed_fwd_is_better(tma, p.G, p.block_size, D) && packed_fwd_smem(D, p.T) <= 200 * 1024) return launch_packed<T, D>(p, MG, s);
  return tma ? launch_loader<T, D, true>(maps, p, MG, st, s) : launch_loader<T, D, false>(maps, p, MG, st, s);
}

}  // namespace

int try_launch_sel_fwd_tc(const void* q, const int64_t* q_stride, const nsa_kv_source* kv, const int32_t* ids,
                          const int64_t* idx_stride, void* out, const int64_t* out_stride, float* lse, int B,
                          int64_t M, int H, int D, int T, int block_size, int chunk_size, int causal, int G,
                          float scale, int dtype, int32_t* status, cudaStream_t stream, bool* launched);

int try_launch_sel_range_fwd_tc(const void* q, const int64_t* q_stride, const nsa_kv_source* kv, int first_block,
                                int n_blocks, void* out, const int64_t* out_stride, float* lse, int B, int64_t M,
                                int H, int D, int block_size, float scale, int dtype, int splits,
                                cudaStream_t stream, bool* launched);
int range_fwd_splits(int B, int64_t M, int H, int n_blocks);

int check_strides16(const char* what, const void* ptr, const int64_t* stride, int n, int esz) {
  NSA_REQUIRE(ptr != nullptr, NSA_ERR_INVALID, "%s: null pointer", what);
  NSA_REQUIRE(aligned16(ptr), NSA_ERR_LAYOUT, "%s: base address must be 16-byte aligned", what);
  for (int i = 0; i < n; ++i)
    NSA_REQUIRE((stride[i] * esz) % 16 == 0, NSA_ERR_LAYOUT,
                "%s: stride %d (%lld elements) is not a multiple of 16 bytes", what, i,
                static_cast<long long>(stride[i]));
  return NSA_OK;
}

int make_kvsrc(const nsa_kv_source* in, int D, int esz, int block_size, KVSrc* out) {
  NSA_REQUIRE(in != nullptr, NSA_ERR_INVALID, "kv source is null");
  NSA_REQUIRE(in->mode == NSA_KV_DENSE || in->mode == NSA_KV_PAGED || in->mode == NSA_KV_PTR, NSA_ERR_INVALID,
              "kv source: unknown mode %d", in->mode);
  NSA_REQUIRE(in->n_tokens >= 0, NSA_ERR_INVALID, "kv source: n_tokens < 0");
  out->mode = in->mode;
  out->k = static_cast<const char*>(in->k);
  out->v = static_cast<const char*>(in->v);
  out->n_tokens = in->n_tokens;
  out->block_table = in->block_table;
  out->max_blocks = in->max_blocks;
  out->page_tokens = in->page_tokens;
  out->ptr_k = in->ptr_k; out->ptr_v = in->ptr_v; out->ptr_sn = in->ptr_stride_n;
  out->k_sb = in->k_stride[0]; out->k_sn = in->k_stride[1]; out->k_sh = in->k_stride[2];
  out->v_sb = in->v_stride[0]; out->v_sn = in->v_stride[1]; out->v_sh = in->v_stride[2];
  if (in->mode == NSA_KV_PTR) {
    NSA_REQUIRE(in->ptr_k && in->ptr_v, NSA_ERR_INVALID, "pointer kv source: null table");
    NSA_REQUIRE((in->ptr_stride_n * esz) % 16 == 0 && in->ptr_stride_n >= D, NSA_ERR_LAYOUT,
                "pointer kv source: token stride must be >= D and a multiple of 16 bytes");
    return NSA_OK;
  }
  if (in->n_tokens == 0) return NSA_OK;
  if (in->mode == NSA_KV_DENSE) {
    int rc = check_strides16("k", in->k, in->k_stride, 3, esz);
    if (rc) return rc;
    rc = check_strides16("v", in->v, in->v_stride, 3, esz);
    if (rc) return rc;
  } else {
    NSA_REQUIRE(in->k && in->v && in->block_table, NSA_ERR_INVALID, "paged kv source: null pointer");
    NSA_REQUIRE(aligned16(in->k) && aligned16(in->v), NSA_ERR_LAYOUT, "page pools must be 16-byte aligned");
    NSA_REQUIRE(in->page_tokens == block_size, NSA_ERR_INVALID,
                "paged kv source: block_size (%d) must equal page_tokens (%d)", block_size, in->page_tokens);
    NSA_REQUIRE(in->max_blocks > 0, NSA_ERR_INVALID, "paged kv source: max_blocks must be > 0");
    NSA_REQUIRE((static_cast<int64_t>(D) * esz) % 16 == 0, NSA_ERR_LAYOUT, "page rows must be 16-byte multiples");
  }
  return NSA_OK;
}

}  // namespace nsa

using namespace nsa;

extern "C" int nsa_sel_fwd(const void* q, const int64_t q_stride[3], const nsa_kv_source* kv,
                           const int32_t* block_indices, const int64_t idx_stride[4], void* out,
                           const int64_t out_stride[3], float* lse, int32_t B, int64_t M, int32_t H,
                           int32_t D, int32_t T, int32_t block_size, int32_t chunk_size,
                           int32_t causal, int32_t group_size, float scale, int32_t dtype,
                           void* stream) {
  NSA_REQUIRE(B >= 0 && M >= 0 && H >= 0, NSA_ERR_INVALID, "sel_fwd: negative size");
  NSA_REQUIRE(group_size >= 1 && group_size <= 128, NSA_ERR_INVALID,
              "sel_fwd: group_size must be in [1,128], got %d", group_size);
  NSA_REQUIRE(block_size > 0 && chunk_size > 0, NSA_ERR_INVALID, "sel_fwd: block_size and chunk_size must be > 0");
  NSA_REQUIRE(T > 0, NSA_ERR_INVALID, "sel_fwd: T must be > 0");
  NSA_REQUIRE(dtype == NSA_BF16 || dtype == NSA_F16, NSA_ERR_UNSUPPORTED,
              "sel_fwd: only bf16 and fp16 are built (dtype %d)", dtype);
  NSA_REQUIRE(D == 64 || D == 128, NSA_ERR_UNSUPPORTED, "sel_fwd: head dim %d not built (64, 128)", D);
  if (B == 0 || M == 0 || H == 0) return NSA_OK;
  NSA_REQUIRE(static_cast<int64_t>(B) <= 65535 && H <= 65535, NSA_ERR_INVALID, "sel_fwd: B and H must be <= 65535");
  NSA_REQUIRE(kv && (kv->mode == NSA_KV_DENSE || B == 1), NSA_ERR_INVALID, "sel_fwd: paged K/V needs B == 1");
  NSA_REQUIRE((block_indices || kv->mode == NSA_KV_PTR) && lse, NSA_ERR_INVALID, "sel_fwd: null pointer");
  const int esz = 2;
  int rc = check_strides16("q", q, q_stride, 3, esz);
  if (rc) return rc;
  rc = check_strides16("out", out, out_stride, 3, esz);
  if (rc) return rc;
  FwdParams p;
  rc = make_kvsrc(kv, D, esz, block_size, &p.kv);
  if (rc) return rc;
  p.q = static_cast<const char*>(q);
  p.q_sb = q_stride[0]; p.q_sm = q_stride[1]; p.q_sh = q_stride[2];
  p.out = static_cast<char*>(out);
  p.o_sb = out_stride[0]; p.o_sm = out_stride[1]; p.o_sh = out_stride[2];
  p.lse = lse;
  p.ids = block_indices;
  p.i_sb = idx_stride[0]; p.i_sg = idx_stride[1]; p.i_sh = idx_stride[2]; p.i_st = idx_stride[3];
  p.B = B; p.H = H; p.T = T; p.block_size = block_size; p.chunk_size = chunk_size;
  p.causal = causal; p.G = group_size; p.M = M;
  p.scale_log2 = scale * kLog2e;
  const int64_t MG = cdiv64(M, group_size);
  NSA_REQUIRE(MG <= 0x7fffffff, NSA_ERR_INVALID, "sel_fwd: too many query groups");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  {
    // the page geometry runs on the tcgen05 kernel; every other shape on the general one
    bool launched = false;
    rc = try_launch_sel_fwd_tc(q, q_stride, kv, block_indices, idx_stride, out, out_stride, lse, B, M, H, D, T,
                               block_size, chunk_size, causal, group_size, scale, dtype, nullptr, s, &launched);
    if (rc) return rc;
    if (launched) return NSA_OK;
  }
  if (dtype == NSA_BF16) {
    return D == 128 ? launch<__nv_bfloat16, 128>(kv, p, static_cast<int>(MG), s)
                    : launch<__nv_bfloat16, 64>(kv, p, static_cast<int>(MG), s);
  }
  return D == 128 ? launch<__half, 128>(kv, p, static_cast<int>(MG), s)
                  : launch<__half, 64>(kv, p, static_cast<int>(MG), s);
}

extern "C" size_t nsa_range_fwd_workspace_bytes(int32_t B, int64_t M, int32_t H, int32_t D, int32_t n_blocks) {
  if (B <= 0 || M <= 0 || H <= 0 || D <= 0 || n_blocks <= 0) return 0;
  const int splits = nsa::range_fwd_splits(B, M, H, n_blocks);
  if (splits == 1) return 0;
  const size_t outs = static_cast<size_t>(splits) * B * M * H * D * 2;
  return ((outs + 255) & ~static_cast<size_t>(255)) + static_cast<size_t>(splits) * B * H * M * 4;
}

extern "C" int nsa_range_fwd(const void* q, const int64_t* q_stride, const nsa_kv_source* kv, int32_t first_block,
                             int32_t n_blocks, void* out, const int64_t* out_stride, float* lse, int32_t B,
                             int64_t M, int32_t H, int32_t D, int32_t block_size, float scale, void* workspace,
                             size_t workspace_bytes, int32_t dtype, void* stream) {
  using namespace nsa;
  NSA_REQUIRE(q && kv && out && lse && q_stride && out_stride, NSA_ERR_INVALID, "range_fwd: null pointer");
  NSA_REQUIRE(first_block >= 0 && n_blocks >= 0, NSA_ERR_INVALID, "range_fwd: first_block %d, n_blocks %d",
              first_block, n_blocks);
  if (B == 0 || M == 0 || H == 0) return NSA_OK;
  NSA_REQUIRE(static_cast<int64_t>(B) <= 65535 && H <= 65535, NSA_ERR_INVALID, "range_fwd: B and H must be <= 65535");
  NSA_REQUIRE(kv->mode == NSA_KV_DENSE || B == 1, NSA_ERR_INVALID, "range_fwd: paged K/V needs B == 1");
  int rc = check_strides16("q", q, q_stride, 3, 2);
  if (rc) return rc;
  rc = check_strides16("out", out, out_stride, 3, 2);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // spans of the range on thread blocks of their own, when that fills the machine better and the
  // caller gave the room for their partial results (the merged output is written contiguous)
  int splits = n_blocks > 0 ? range_fwd_splits(B, M, H, n_blocks) : 1;
  const size_t outs_bytes = (static_cast<size_t>(splits) * B * M * H * D * 2 + 255) & ~static_cast<size_t>(255);
  const bool contiguous = out_stride[2] == D && out_stride[1] == static_cast<int64_t>(H) * D &&
                          (B == 1 || out_stride[0] == M * H * D);
  if (splits > 1 && (workspace == nullptr || !aligned16(workspace) || !contiguous || B * splits > 65535 ||
                     workspace_bytes < outs_bytes + static_cast<size_t>(splits) * B * H * M * 4))
    splits = 1;
  bool launched = false;
  if (splits > 1) {
    char* part_out = static_cast<char*>(workspace);
    float* part_lse = reinterpret_cast<float*>(part_out + outs_bytes);
    const int64_t part_stride[3] = {M * H * D, static_cast<int64_t>(H) * D, D};
    rc = try_launch_sel_range_fwd_tc(q, q_stride, kv, first_block, n_blocks, part_out, part_stride, part_lse, B, M, H,
                                     D, block_size, scale, dtype, splits, s, &launched);
    if (rc) return rc;
    if (launched) return nsa_merge_partials(part_out, part_lse, splits, B, M, H, D, out, lse, dtype, stream);
  }
  rc = try_launch_sel_range_fwd_tc(q, q_stride, kv, first_block, n_blocks, out, out_stride, lse, B, M, H, D,
                                   block_size, scale, dtype, 1, s, &launched);
  if (rc) return rc;
  NSA_REQUIRE(launched, NSA_ERR_UNSUPPORTED,
              "range_fwd: built for bf16, D = 128, 64-token blocks, H > 1, dense or paged K/V, at most 1024 blocks; "
              "list the blocks and call nsa_sel_fwd for anything else");
  return NSA_OK;
}
