// Selection attention backward, dK / dV of blocks of at most 32 tokens (any group size, bf16 / fp16, D in {64, 128}) on
// the tcgen05 tensor cores.
//
// A block of 30 tokens is far from the 128 rows of a tensor-core tile, but its bucket of query groups is not: a thread
// block owns one (batch, head, block), stacks the rows of the bucket's groups in pieces of 16 (a group of 15 is one
// piece with a zero row) to tiles of 64 (D = 128) or 128 (D = 64) query rows and computes per tile
//     S = Q K^T, dP = dO V^T           M = 64 or 128 query rows, N = 32 tokens, K = D
//     dV^T += dO^T P, dK^T += Q^T dS   M = D (rows of the head dim), N = 32 tokens, K = 16 per piece
// with the accumulators in TMEM for the whole bucket.  At D = 64 the last two are one product: dO and Q lie one behind
// the other as the two 64-row halves of its A operand and P, dS are the halves of its B operand; of the four quadrants
// of the result two are wanted.  Buckets are walked in ascending group order without atomics: bit-reproducible.
//
//   warps 0-3  one or two pieces of 16 query rows each: P and dS from TMEM into one swizzled tile (32 + 32 columns); one
//              lane per piece issues its copies, dO as soon as dV^T of the tile before is done, then Q
//   warp 4     issues the products
//
// One stage of rows per thread block; the four thread blocks of an SM overlap each other.
// What bounds it: the chain copy -> S, dP -> exponentials -> dV, dK of a thread block against the bytes that shared memory
// can keep in flight.  32760 queries x 12 heads, D = 128, 16 blocks of 30, groups of 15, bf16: 1106 us on mma.sync, 620 us
// with tiles of 128 rows and two thread blocks per SM, 549 us as it is.  2 x 3120 queries x 16 heads, D = 64, 64 blocks of
// 24, groups of 12, fp16: 699 us, 371 us as it is (410 us with three thread blocks per SM), 531 us with tiles of 64 rows.
// (256 threads for the exponentials: 632 / 500 us.)
#include "sel_rows.cuh"

#include <type_traits>

namespace nsa {
namespace {

using namespace tc;

constexpr int kTok = 32, kPiece = 16;
template <int D> constexpr int kRows = D == 128 ? 64 : 128;                   // query rows of a tile
constexpr int kComputeThreads = 128, kThreads = 160;
constexpr uint32_t kTmemCols = 128;                // S 32, dP 32, dV^T and dK^T 32 each
constexpr uint32_t kColS = 0, kColDP = 32, kColDV = 64, kColDK = 96;

template <int D> constexpr uint32_t kHalf = kRows<D> * 128;                    // 64 columns of one operand's tile
template <int D> constexpr uint32_t kOperand = kRows<D> * D * 2;
// Four thread blocks share an SM if each takes no more than 56 KiB: the barriers lie in the last row of the V tile when
// the block has no 32nd token (that column of dP is masked whatever it holds), else behind it.
constexpr uint32_t kBars = 128;
template <int D> constexpr uint32_t kTiles = 2 * kOperand<D> + kRows<D> * 128 + 2 * kTok * D * 2;
template <int D> __host__ __device__ constexpr uint32_t smem_bytes(int block_size) { return kTiles<D> + (block_size < kTok ? 0 : kBars); }

__device__ __forceinline__ void piece_copy(uint32_t dst, const CUtensorMap* map, int col, int h, int row, int unit, int b, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
               ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(col), "r"(h), "r"(row), "r"(unit), "r"(b) : "memory");
}

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, 4) sel_bwd_dkv_rows_tc_kernel(const __grid_constant__ RingMaps maps, const DkvRowsArgs p,
                                                                          int32_t* status) {
  constexpr int ESZ = 2, HALVES = D / 64, ROWS = kRows<D>, kPieces = ROWS / kPiece;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sDO = smem;                             // [half][ROWS][128 bytes]
  uint8_t* sQ = smem + kOperand<D>;
  uint8_t* sP = smem + 2 * kOperand<D>;            // [ROWS][P of 32 tokens, dS of 32 tokens]
  uint8_t* sK = sP + ROWS * 128;                   // [half][32 tokens][128 bytes]
  uint8_t* sV = sK + kTok * D * 2;
  const int loaded = p.block_size < kTok ? kTok - 1 : kTok;       // rows of the K and V tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + smem_bytes<D>(p.block_size) - kBars);
  uint64_t *full_do = bars, *full_q = bars + 1, *s_ready = bars + 2, *p_ready = bars + 3, *dv_done = bars + 4, *dk_done = bars + 5;
  int* abort = reinterpret_cast<int*>(bars + 6);
  uint32_t* tmem_word = reinterpret_cast<uint32_t*>(bars + 7);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int64_t t0 = static_cast<int64_t>(blk) * p.block_size;
  const int64_t left = p.kv.n_tokens - t0;
  const int n_rows = static_cast<int>(left < p.block_size ? left : p.block_size);
  if (n_rows <= 0) return;
  const int64_t out_row = static_cast<int64_t>(p.H) * D * ESZ;
  const int64_t out_at = (static_cast<int64_t>(b) * p.kv.n_tokens + t0) * out_row + static_cast<int64_t>(h) * D * ESZ;
  const int64_t bh = static_cast<int64_t>(b) * p.H + h;
  const int32_t* offs = p.offsets + bh * (p.NS + 1);
  const int beg = offs[blk], n_ent = offs[blk + 1] - beg;
  const int32_t* bucket = p.groups + bh * p.MG * p.T + beg;
  const BlockRef br = resolve_block<ESZ>(p.kv, b, h, blk, D, p.block_size, 1, false, 0);
  if (n_ent == 0 || br.k == nullptr) {
    for (int i = tid; i < n_rows * (D / 8); i += kThreads) {
      const int64_t at = out_at + (i / (D / 8)) * out_row + i % (D / 8) * 16;
      *reinterpret_cast<uint4*>(p.dk + at) = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(p.dv + at) = make_uint4(0, 0, 0, 0);
    }
    return;
  }

  if (tid == 0) {
    *abort = 0;
    mbar_init(full_do, kPieces);
    mbar_init(full_q, kPieces);
    mbar_init(s_ready, 1);
    mbar_init(p_ready, kComputeThreads);
    mbar_init(dv_done, 1);
    mbar_init(dk_done, 1);
    fence_barrier_init();
  }
  if (warp == 4) tmem_alloc(tmem_word, kTmemCols);
  // this block's K and V rows (zeros up to 31 or 32)
  {
    const int64_t k_row = kv_row_bytes(p.kv, false, D, ESZ), v_row = kv_row_bytes(p.kv, true, D, ESZ);
    for (int i = tid; i < loaded * (D / 8); i += kThreads) {
      const int r = i / (D / 8), c = i % (D / 8), bytes = r < n_rows ? 16 : 0;
      const int64_t at = r < n_rows ? r : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sK) + ring_at<kTok>(r, c)), "l"(br.k + at * k_row + c * 16), "r"(bytes) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sV) + ring_at<kTok>(r, c)), "l"(br.v + at * v_row + c * 16), "r"(bytes) : "memory");
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_async_shared();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tmem_word;
  const int subs = (p.G + kPiece - 1) / kPiece;                  // pieces of a group
  const int64_t pieces = static_cast<int64_t>(n_ent) * subs;
  const int tiles = static_cast<int>((pieces + kPieces - 1) / kPieces);

  if (warp < 4) {
    const int piece = ROWS == 64 ? warp : tid / kPiece;
    const bool issuer = (lane & (ROWS == 64 ? 31 : 15)) == 0;
    // group and first row of this thread's piece of tile i; -1: none
    const auto group_of = [&](int i, int& r0) {
      const int64_t x = static_cast<int64_t>(i) * kPieces + piece;
      if (x >= pieces) return -1;
      const int e = subs == 1 ? static_cast<int>(x) : static_cast<int>(x / subs);
      r0 = static_cast<int>(x - static_cast<int64_t>(e) * subs) * kPiece;
      return bucket[e];
    };
    const auto copy = [&](uint8_t* tile, uint64_t* bar, const CUtensorMap& whole, const CUtensorMap& tail, int g, int r0) {
      if (g < 0) {
        mbar_arrive(bar);
        return;
      }
      mbar_expect_tx(bar, kPiece * D * ESZ);
      const bool cut = g >= p.whole;
      const CUtensorMap* map = cut ? &tail : &whole;
      const int row = cut ? g * p.G + r0 : r0, unit = cut ? 0 : g;
#pragma unroll
      for (int c = 0; c < HALVES; ++c) piece_copy(smem_u32(tile) + c * kHalf<D> + piece * (kPiece * 128), map, c * 64, h, row, unit, b, bar);
    };
    int r0 = 0, r0_next = 0;
    int g = group_of(0, r0);
    if (issuer) {
      copy(sDO, full_do, maps.b, maps.b_tail, g, r0);
      copy(sQ, full_q, maps.a, maps.a_tail, g, r0);
    }
    const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
    bool ok = true;
    int filled = 1;                                              // tiles whose copies were issued
    for (int i = 0; i < tiles; ++i) {
      // rows of the piece, and how many of the block's tokens its group may see
      const int g_next = i + 1 < tiles ? group_of(i + 1, r0_next) : -1;
      constexpr int RT = ROWS == 64 ? 2 : 1;                     // rows per thread: lane / 4 and + 8 of the piece, or its own
      float lse2[2] = {INFINITY, INFINITY}, delta[2] = {0.f, 0.f};
      int vis = 0;
      if (g >= 0) {
        const int64_t g0 = static_cast<int64_t>(g) * p.G, rows = p.M - g0 < p.G ? p.M - g0 : p.G;
#pragma unroll
        for (int y = 0; y < RT; ++y) {
          const int r = r0 + (ROWS == 64 ? (lane >> 2) + 8 * y : tid % kPiece);
          if (r < rows) {
            lse2[y] = p.lse[bh * p.M + g0 + r] * kLog2e;
            delta[y] = p.delta[bh * p.M + g0 + r];
          }
        }
        vis = n_rows;
        if (p.causal) {
          const int64_t seen = (g0 / p.chunk_size + 1) * p.chunk_size - t0;
          vis = static_cast<int>(seen < vis ? seen : vis);
        }
      }
      ok = __all_sync(0xffffffffu, mbar_wait(s_ready, i & 1, abort));
      if (!ok) break;
      tc_fence_after();
      if constexpr (ROWS == 64) {
        uint32_t s[16], dp[16];                                  // [8-token column][row lane / 4: 2 tokens, row + 8: 2 tokens]
        tmem_ld_16x256b_x4_nowait(tm + lanes + kColS, s);
        tmem_ld_16x256b_x4_nowait(tm + lanes + kColDP, dp);
        tmem_ld_wait();
        uint32_t pw[4][2], dw[4][2];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            float e[2], d[2];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              const int x = 4 * c + 2 * y + z;
              const bool in = 8 * c + 2 * (lane & 3) + z < vis;
              const float pe = fast_exp2(__uint_as_float(s[x]) * p.scale_log2 - lse2[y]);
              e[z] = in ? pe : 0.f;
              d[z] = in ? pe * (__uint_as_float(dp[x]) - delta[y]) * p.scale : 0.f;
            }
            pw[c][y] = pack2<T>(e[0], e[1]);
            dw[c][y] = pack2<T>(d[0], d[1]);
          }
        const int row = (lane & 7) + ((lane >> 3) & 1) * 8, col = lane >> 4;     // of the 8 x 8 matrix this lane addresses
        const uint32_t row_at = smem_u32(sP) + static_cast<uint32_t>(warp * kPiece + row) * 128;
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
          stmatrix_x4(row_at + (((c + col) ^ (row & 7)) << 4), pw[c][0], pw[c][1], pw[c + 1][0], pw[c + 1][1]);
          stmatrix_x4(row_at + (((4 + c + col) ^ (row & 7)) << 4), dw[c][0], dw[c][1], dw[c + 1][0], dw[c + 1][1]);
        }
      } else {
        uint32_t s[32], dp[32];
        tmem_ld32_nowait(tm + lanes + kColS, s);
        tmem_ld32_nowait(tm + lanes + kColDP, dp);
        tmem_ld_wait();
        const uint32_t row_at = smem_u32(sP) + static_cast<uint32_t>(tid) * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) {                            // 8 tokens: a 16-byte piece of P and one of dS
          uint32_t pw[4], dw[4];
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            float e[2], d[2];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              const int j = c * 8 + y * 2 + z;
              const float pe = fast_exp2(__uint_as_float(s[j]) * p.scale_log2 - lse2[0]);
              e[z] = j < vis ? pe : 0.f;
              d[z] = j < vis ? pe * (__uint_as_float(dp[j]) - delta[0]) * p.scale : 0.f;
            }
            pw[y] = pack2<T>(e[0], e[1]);
            dw[y] = pack2<T>(d[0], d[1]);
          }
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(row_at + ((c ^ (tid & 7)) << 4)), "r"(pw[0]), "r"(pw[1]), "r"(pw[2]), "r"(pw[3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(row_at + (((c + 4) ^ (tid & 7)) << 4)), "r"(dw[0]), "r"(dw[1]), "r"(dw[2]), "r"(dw[3]) : "memory");
        }
      }
      fence_async_shared();
      tc_fence_before();
      mbar_arrive(p_ready);
      g = g_next;
      r0 = r0_next;
      if (i + 1 < tiles) {
        if (issuer) {
          ok = mbar_wait(dv_done, i & 1, abort);
          if (ok) copy(sDO, full_do, maps.b, maps.b_tail, g, r0);
          ok = ok && mbar_wait(dk_done, i & 1, abort);
          if (ok) copy(sQ, full_q, maps.a, maps.a_tail, g, r0);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        ++filled;
      }
    }
    ok = ok && __all_sync(0xffffffffu, mbar_wait(dk_done, (tiles - 1) & 1, abort));
    if (!ok && issuer) {                                          // copies in flight end before the thread block does
      atomicExch(status, NSA_ERR_CUDA);
      mbar_wait(full_do, (filled - 1) & 1, abort);
      mbar_wait(full_q, (filled - 1) & 1, abort);
    }
    // dV^T and dK^T (thread = head dim) -> rows of tokens in the dead Q / dO tiles -> 16-byte pieces of global rows
    constexpr uint32_t pitch = D * 2 + 16;
    const uint32_t stage = smem_u32(smem);
    tc_fence_after();
#pragma unroll
    for (int mat = 0; mat < 2; ++mat) {
      if (!ok || (D == 64 && mat != warp / 2)) continue;          // D = 64: lanes 0-63 hold dV^T, 64-127 dK^T
      uint32_t x[32];
      tmem_ld32_nowait(tm + lanes + (mat ? kColDK : kColDV), x);
      tmem_ld_wait();
      const uint32_t at = stage + mat * (kTok * pitch) + static_cast<uint32_t>(tid & (D - 1)) * 2;
#pragma unroll
      for (int j = 0; j < kTok; ++j) {
        const T v = from_f32<T>(__uint_as_float(x[j]));
        asm volatile("st.shared.b16 [%0], %1;" ::"r"(at + j * pitch), "h"(*reinterpret_cast<const uint16_t*>(&v)) : "memory");
      }
    }
    named_barrier(1, kComputeThreads);                            // every warp comes here, also after a wait that gave up
    for (int i = tid; ok && i < 2 * kTok * (D / 8); i += kComputeThreads) {
      const int mat = i / (kTok * (D / 8)), x = i % (kTok * (D / 8)), row = x / (D / 8), c = x % (D / 8);
      if (row < n_rows) {
        uint4 v;
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(stage + (mat * kTok + row) * pitch + c * 16));
        *reinterpret_cast<uint4*>((mat ? p.dk : p.dv) + out_at + row * out_row + c * 16) = v;
      }
    }
  } else {
    // ======================= products (warp-uniform control flow, one elected lane issues) =======================
    constexpr uint32_t types = std::is_same<T, __half>::value ? ~((1u << 7) | (1u << 10)) : ~0u;
    constexpr uint32_t id_s = instr_desc_bf16(ROWS, kTok, 0, 0) & types;
    constexpr uint32_t id_g = instr_desc_bf16(128, D == 128 ? kTok : 2 * kTok, 1, 1) & types;
    const uint32_t el = elect_one();
    const uint64_t dQ = smem_desc(smem_u32(sQ), 16, 1024), dDO = smem_desc(smem_u32(sDO), 16, 1024);
    const uint64_t dK = smem_desc(smem_u32(sK), 16, 1024), dV = smem_desc(smem_u32(sV), 16, 1024);
    const uint64_t dQmn = smem_desc(smem_u32(sQ), kHalf<D>, 1024), dDOmn = smem_desc(smem_u32(sDO), kHalf<D>, 1024);
    const uint64_t dP = smem_desc(smem_u32(sP), 16, 1024);
    bool ok = true;
    for (int i = 0; i < tiles && ok; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait(full_do, i & 1, abort)) && __all_sync(0xffffffffu, mbar_wait(full_q, i & 1, abort));
      if (!ok) break;
      tc_fence_after();
      if (el) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t q_at = (kk >> 2) * kHalf<D> + (kk & 3) * 32, k_at = (kk >> 2) * (kTok * 128) + (kk & 3) * 32;
          umma_ss(tm + kColS, desc_advance(dQ, q_at), desc_advance(dK, k_at), id_s, kk > 0);
        }
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t q_at = (kk >> 2) * kHalf<D> + (kk & 3) * 32, k_at = (kk >> 2) * (kTok * 128) + (kk & 3) * 32;
          umma_ss(tm + kColDP, desc_advance(dDO, q_at), desc_advance(dV, k_at), id_s, kk > 0);
        }
        umma_commit(s_ready);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait(p_ready, i & 1, abort));
      if (!ok) break;
      tc_fence_after();
      const int64_t rest = pieces - static_cast<int64_t>(i) * kPieces;
      const int n = rest < kPieces ? static_cast<int>(rest) : kPieces;      // rows of absent pieces are not summed
      if (el) {
        for (int kk = 0; kk < n; ++kk)
          umma_ss(tm + kColDV, desc_advance(dDOmn, kk * 2048), desc_advance(dP, kk * 2048), id_g, i > 0 || kk > 0);
        umma_commit(dv_done);
        if (D == 128)
          for (int kk = 0; kk < n; ++kk)
            umma_ss(tm + kColDK, desc_advance(dQmn, kk * 2048), desc_advance(dP, kk * 2048 + 64), id_g, i > 0 || kk > 0);
        umma_commit(dk_done);
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 4) tmem_dealloc(tm, kTmemCols);
}

template <typename T, int D>
int launch(const RingMaps& maps, const DkvRowsArgs& p, int32_t* status, cudaStream_t stream) {
  const uint32_t smem = smem_bytes<D>(p.block_size);
  static_assert(2 * kTok * (D * 2 + 16) <= 2 * kOperand<D>, "the epilogue stages its rows in the Q and dO tiles");
  auto kernel = sel_bwd_dkv_rows_tc_kernel<T, D>;
  NSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  kernel<<<dim3(static_cast<unsigned>(p.NS), p.H, p.B), kThreads, smem, stream>>>(maps, p, status);
  NSA_LAUNCH_OK("sel_bwd_dkv_rows_tc_kernel");
  return NSA_OK;
}

}  // namespace

// Serves blocks of at most 32 tokens whose query rows tensor maps can describe; everything else stays on the row kernel
// (larger blocks fill its tiles: at 64 tokens and D = 128 it needs 315 us where the smaller blocks needed 1106).
int try_launch_sel_bwd_dkv_rows_tc(DkvRowsArgs p, const int64_t* q_stride, const int64_t* do_stride, int D, int dtype,
                                   int32_t* status, cudaStream_t stream, bool* launched) {
  *launched = false;
  if (p.block_size > kTok || p.NS <= 0 || p.NS > 0x7fffffff || p.M <= 0) return NSA_OK;
  RingMaps maps{};
  if (!make_unit_maps(&maps.a, &maps.a_tail, p.q, q_stride, p.B, p.M, p.H, D, p.G, kPiece, false) ||
      !make_unit_maps(&maps.b, &maps.b_tail, p.dO, do_stride, p.B, p.M, p.H, D, p.G, kPiece, false))
    return NSA_OK;
  p.whole = static_cast<int>(p.M / p.G);
  *launched = true;
  if (dtype == NSA_BF16) return D == 128 ? launch<__nv_bfloat16, 128>(maps, p, status, stream) : launch<__nv_bfloat16, 64>(maps, p, status, stream);
  return D == 128 ? launch<__half, 128>(maps, p, status, stream) : launch<__half, 64>(maps, p, status, stream);
}

}  // namespace nsa
