// Selection attention forward, general geometry (any block size, group size <= 128, D in {64, 128}, bf16 / fp16):
// a thread block is one (batch, query group, head); each of its warps owns 16 query rows and all of them read the
// same ring of K/V tiles (sel_rows.cuh); S = Q K^T and O += P V run on mma.sync m16n8k16 with fp32 accumulation
// and an online softmax in the exp2 domain.
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
  int64_t M;
  float scale_log2;
};

// W warps of 16 query rows each share one ring; with W = 1 the tiles of the list may be dealt out to KS warps
// with rings of their own, whose partial results are merged at the end (few groups on many SMs).
// What bounds it for small groups: the gathered K/V rows, which every list fetches for itself, through the L2 to SM
// path.  32760 queries x 12 heads, 15-query groups, 16 blocks of 30 tokens: 397 us = 16 TB/s of rows against the
// 18 TB/s that bulk copies reach here (5911 us with one warp per 70 KB thread block, 124 TF -> 243 TF of products).
// One K/V stage and 12 warps per SM: 397 us; two stages and 7 warps: 661 us; 16- or 32-byte loads straight into
// fragments, no shared memory: 780 us.
template <typename T, int D, int W, int KS, bool TMA>
__global__ void __launch_bounds__(32 * W * KS) sel_fwd_rows_kernel(const __grid_constant__ RingMaps maps, const FwdParams p,
                                                                   const int stages, int32_t* status) {
  static_assert(W == 1 || KS == 1, "only single-warp groups are split");
  constexpr int ESZ = sizeof(T), ROWS = 32;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t4 = lane & 3;
  const int g = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int64_t g0 = static_cast<int64_t>(g) * p.G;
  const int row_warp = W > 1 ? warp : 0, part = KS > 1 ? warp : 0;
  const int n_q = static_cast<int>(p.M - g0 < p.G ? p.M - g0 : p.G) - row_warp * 16;   // rows of this warp (may be <= 0)
  const int64_t m0 = g0 + row_warp * 16;

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

template <typename T, int D, int W, int KS, bool TMA>
int launch_rows(const RingMaps& maps, const FwdParams& p, int MG, int32_t* status, cudaStream_t stream) {
  // stages: two per ring of a single warp (the thread blocks that share an SM are the depth), three where several
  // warps wait for the same ring; never less than the epilogue's staging needs
  const int stages = W <= 2 ? 1 : 3;
  static_assert(W * 16 * (D * 2 + 16) <= (W <= 2 ? 1 : 3) * 2 * kRingTile<D, 32>, "the epilogue stages its rows in the ring");
  static_assert((KS - 1) * (D / 8 * 128 + 128) * 4 <= KS * 2 * kRingTile<D, 32>, "the partial results are merged in the ring");
  const size_t smem = static_cast<size_t>(KS) * stages * 2 * kRingTile<D, 32> + KS * kRingBars * 8 + 16 +
                      ring_list_bytes(p.T);
  NSA_REQUIRE(smem <= 226 * 1024, NSA_ERR_UNSUPPORTED, "sel_fwd: T=%d needs too much shared memory", p.T);
  auto kernel = sel_fwd_rows_kernel<T, D, W, KS, TMA>;
  NSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  kernel<<<dim3(MG, p.H, p.B), 32 * W * KS, smem, stream>>>(maps, p, stages, status);
  NSA_LAUNCH_OK("sel_fwd_rows_kernel");
  return NSA_OK;
}

template <typename T, int D, bool TMA>
int launch_loader(const RingMaps& maps, const FwdParams& p, int MG, int32_t* st, cudaStream_t s) {
  if (p.G <= 16) {
    // as many warps per list as still fit the chip at once: 12 warps per SM at D = 128 (registers), 16 at D = 64.
    // Measured, D = 128, 16 blocks of 30, one / two / four warps per list: 384 lists 22.7 / 18.5 / 15.5 us,
    // 768 lists 25.9 / 23.0 / 28.0 us, 1248 lists 31.6 / 40.8 / 41.0 us
    const bool short_list = ring_list_bytes(p.T) <= 64 * 1024;                   // (each warp's ring needs its room)
    const int64_t units = static_cast<int64_t>(MG) * p.H * p.B, room = 148 * (D == 128 ? 12 : 16);
    if (units * 4 <= room && short_list) return launch_rows<T, D, 1, 4, TMA>(maps, p, MG, st, s);
    if (units * 2 <= room && short_list) return launch_rows<T, D, 1, 2, TMA>(maps, p, MG, st, s);
    return launch_rows<T, D, 1, 1, TMA>(maps, p, MG, st, s);
  }
  if (p.G <= 32) return launch_rows<T, D, 2, 1, TMA>(maps, p, MG, st, s);
  if (p.G <= 64) return launch_rows<T, D, 4, 1, TMA>(maps, p, MG, st, s);
  return launch_rows<T, D, 8, 1, TMA>(maps, p, MG, st, s);
}

template <typename T, int D>
int launch(const nsa_kv_source* kv, const FwdParams& p, int MG, cudaStream_t s) {
  int32_t* st = nullptr;
  int rc = device_status_address(&st);
  if (rc) return rc;
  RingMaps maps{};
  return make_ring_maps(kv, p.B, p.H, D, p.block_size, 32, &maps) ? launch_loader<T, D, true>(maps, p, MG, st, s)
                                                              : launch_loader<T, D, false>(maps, p, MG, st, s);
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
