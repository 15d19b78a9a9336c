// The row kernels: selection forward, dQ and dK/dV of every geometry that the tcgen05 kernels do not serve
// (any block size, groups of 1 to 128 queries, D in {64, 128}, bf16 / fp16), on mma.sync m16n8k16.
//
// A query group of this path is often far smaller than a tensor-core tile (15 queries against 30-token
// blocks), and every group reads its own blocks, so what bounds these kernels is how fast the gathered rows
// reach shared memory and how many warps hide each other's chains of small products, not the products
// themselves.  Hence: a warp works on 16 rows by itself, the gathered rows come in tiles of 16 to 64 rows through a
// ring that one thread fills with TMA copies (one instruction per operand and tile), and as many small thread
// blocks as registers allow share an SM, each with its own ring: one stage is enough, depth only costs warps.
// Operands that the tensor maps cannot describe (address tables, zero strides) go through the same ring with
// cp.async.
//
// Ring tile of one operand: [D / 64 halves][ROWS][128 bytes], 128-byte swizzle (16-byte chunk c of row r at
// c ^ (r & 7)).  The maps know the units (blocks, query groups): rows past the end of a unit arrive as zeros.
#pragma once

#include "common.cuh"
#include "tc_common.cuh"

namespace nsa {

template <int D, int ROWS> constexpr int kRingTile = ROWS * D * 2;     // bytes of one operand's tile
constexpr int kRingMaxStages = 4;
constexpr int kRingBars = 3 * kRingMaxStages;                           // barriers of one ring


// One tile: rows [r0, r0 + ROWS) of a unit, of which the first n count.
struct RingTile {
  uint64_t a, b;       // addresses of row r0 in the two operands (cp.async loader)
  int unit, r0, n;
  int clear;           // rows of the unit that the copy brings (n < clear: the others are zeroed after they land)
  int64_t aux;         // element of the fp32 row vectors (rings that carry them)
};

__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// byte offset of 16-byte chunk c (0 .. D / 8 - 1) of row r in a tile
template <int ROWS> __device__ __forceinline__ uint32_t ring_at(int r, int c) {
  return static_cast<uint32_t>((c >> 3) * (ROWS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// A operand (16 rows x D) from global memory: rows row0 + gid and + 8, k = 16 kk + 2 t4 (+1, +8, +9)
template <int D>
__device__ __forceinline__ void load_a_frag(uint32_t (&a)[D / 16][4], const char* base, int64_t row_bytes, int rows) {
  const int lane = threadIdx.x & 31, gid = lane >> 2, t4 = lane & 3;
  const char* lo = base + gid * row_bytes + t4 * 4;
  const char* hi = lo + 8 * row_bytes;
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    a[kk][0] = gid < rows ? __ldg(reinterpret_cast<const uint32_t*>(lo + kk * 32)) : 0u;
    a[kk][1] = gid + 8 < rows ? __ldg(reinterpret_cast<const uint32_t*>(hi + kk * 32)) : 0u;
    a[kk][2] = gid < rows ? __ldg(reinterpret_cast<const uint32_t*>(lo + kk * 32 + 16)) : 0u;
    a[kk][3] = gid + 8 < rows ? __ldg(reinterpret_cast<const uint32_t*>(hi + kk * 32 + 16)) : 0u;
  }
}

// A operand in shared memory: 16 rows of a ring tile, k-step kk
template <int ROWS>
__device__ __forceinline__ void ldsm_a(uint32_t (&a)[4], uint32_t tile, int row0, int kk) {
  const int lane = threadIdx.x & 31, c = 2 * kk;
  ldsm_x4(a, tile + (c >> 3) * (ROWS * 128) + static_cast<uint32_t>(row0 + (lane & 15)) * 128 +
                 ((((c & 7) + (lane >> 4)) ^ (lane & 7)) << 4));
}
// B operand of columns = tile rows (16 of them from j * 16), k-step kk: two n8 fragments
template <int ROWS>
__device__ __forceinline__ void ldsm_b(uint32_t (&b)[4], uint32_t tile, int j, int kk) {
  const int lane = threadIdx.x & 31, c = 2 * kk;
  ldsm_x4(b, tile + (c >> 3) * (ROWS * 128) + static_cast<uint32_t>(j * 16 + (lane & 7) + ((lane >> 4) << 3)) * 128 +
                 ((((c & 7) + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
}

// acc[n] (16 x 8 each) += A * rows(tile)^T: the tile's rows (n16 * 16 of them) are the columns of the product
template <typename T, int D, int ROWS>
__device__ __forceinline__ void mma_rows_t(float (&acc)[ROWS / 8][4], const uint32_t (&a)[D / 16][4], uint32_t tile, int n16) {
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
    for (int j = 0; j < ROWS / 16; ++j)
      if (j < n16) {
        uint32_t b[4];
        ldsm_b<ROWS>(b, tile, j, kk);
        mma16816<T>(acc[2 * j], a[kk], b[0], b[1]);
        mma16816<T>(acc[2 * j + 1], a[kk], b[2], b[3]);
      }
}
// two such products with tiles of ROWS rows, A being 16 rows (from a_row0) of a tile each: their chains of dependent
// products interleave
template <typename T, int D, int AROWS, int ROWS>
__device__ __forceinline__ void mma_rows_t2(float (&x)[ROWS / 8][4], uint32_t ax, uint32_t bx, float (&y)[ROWS / 8][4], uint32_t ay,
                                            uint32_t by, int a_row0, int n16) {
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    uint32_t a0[4], a1[4];
    ldsm_a<AROWS>(a0, ax, a_row0, kk);
    ldsm_a<AROWS>(a1, ay, a_row0, kk);
#pragma unroll
    for (int j = 0; j < ROWS / 16; ++j) {
      if (ROWS == 16 || j < n16) {
        uint32_t b0[4], b1[4];
        ldsm_b<ROWS>(b0, bx, j, kk);
        ldsm_b<ROWS>(b1, by, j, kk);
        mma16816<T>(x[2 * j], a0, b0[0], b0[1]);
        mma16816<T>(x[2 * j + 1], a0, b0[2], b0[3]);
        mma16816<T>(y[2 * j], a1, b1[0], b1[1]);
        mma16816<T>(y[2 * j + 1], a1, b1[2], b1[3]);
      }
    }
  }
}

// acc[n] (16 x 8 each, n < D / 8) += P * rows(tile): the tile's rows are summed over, P packed in pa[16 rows]
template <typename T, int D, int ROWS>
__device__ __forceinline__ void mma_rows(float (&acc)[D / 8][4], const uint32_t (&pa)[ROWS / 16][4], uint32_t tile, int n16) {
  const int lane = threadIdx.x & 31;
  const uint32_t row = tile + static_cast<uint32_t>((lane & 7) + ((lane >> 3) & 1) * 8) * 128;
#pragma unroll
  for (int j = 0; j < ROWS / 16; ++j) {
    if (j < n16) {
#pragma unroll
      for (int d16 = 0; d16 < D / 16; ++d16) {
        const int c = 2 * d16;
        uint32_t b[4];
        ldsm_x4_trans(b, row + j * 2048 + (c >> 3) * (ROWS * 128) + ((((c & 7) + (lane >> 4)) ^ (lane & 7)) << 4));
        mma16816<T>(acc[2 * d16], pa[j], b[0], b[1]);
        mma16816<T>(acc[2 * d16 + 1], pa[j], b[2], b[3]);
      }
    }
  }
}

// rows [n, end) of a tile := 0 (by one warp): rows that a copy brought but that do not count must
// not reach a product, not even times 0
template <int D, int ROWS>
__device__ __forceinline__ void ring_clear_rows(uint32_t tile, int n, int end) {
  const int lane = threadIdx.x & 31;
  for (int i = lane; i < (end - n) * (D / 8); i += 32) {
    const int r = n + i / (D / 8), c = i % (D / 8);
    asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(tile + ring_at<ROWS>(r, c)), "r"(0) : "memory");
  }
  __syncwarp();
}

// 16 x D accumulator -> 16-bit rows in shared memory ([16][D * 2 + 16 bytes]) -> whole 16-byte pieces of global rows
template <typename T, int D>
__device__ __forceinline__ void store_rows(const float (&acc)[D / 8][4], float s_lo, float s_hi, uint32_t stage, char* dst,
                                           int64_t row_bytes, int rows) {
  constexpr uint32_t pitch = D * 2 + 16;
  const int lane = threadIdx.x & 31;
  const uint32_t st = stage + static_cast<uint32_t>((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 16;
#pragma unroll
  for (int n = 0; n < D / 8; n += 2)
    tc::stmatrix_x4(st + n * 16, pack2<T>(acc[n][0] * s_lo, acc[n][1] * s_lo), pack2<T>(acc[n][2] * s_hi, acc[n][3] * s_hi),
                    pack2<T>(acc[n + 1][0] * s_lo, acc[n + 1][1] * s_lo), pack2<T>(acc[n + 1][2] * s_hi, acc[n + 1][3] * s_hi));
  __syncwarp();
#pragma unroll
  for (int i = 0; i < D / 16; ++i) {
    const int x = i * 32 + lane, r = x / (D / 8), c = x % (D / 8);
    if (r < rows) {
      uint4 v;
      asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                   : "r"(stage + r * pitch + c * 16));
      *reinterpret_cast<uint4*>(dst + r * row_bytes + c * 16) = v;
    }
  }
}

// Two row operands (K and V of the listed blocks, or Q and dO of the listed groups) that stream through a ring.
struct RingMaps {
  CUtensorMap a, b;             // whole units
  CUtensorMap a_tail, b_tail;   // the last unit when it is cut off by the end of the tensor
};
struct RingSource {
  const RingMaps* maps;
  int64_t a_row, b_row;         // bytes between rows (cp.async loader)
  int h, b;                     // head and batch coordinates (a page pool has neither)
  int unit_rows, whole;         // rows of a unit; units in front of the cut-off one
  int halves;                   // 1: the maps' last dimension is the 64-column half (one copy per tile), else the batch
};

// Fills tile memory `dst` with operand OP (0: a, 1: b) of tile t.  TMA: one thread; cp.async: a whole warp.
template <int D, int ROWS, bool TMA, int OP>
__device__ __forceinline__ void ring_fill(uint32_t dst, uint64_t* full, const RingTile& t, const RingSource& s) {
  if constexpr (TMA) {
    tc::mbar_expect_tx(full, static_cast<uint32_t>(kRingTile<D, ROWS>));
    const uint32_t bar = smem_u32(full);
    const bool tail = t.unit >= s.whole;
    const CUtensorMap* map = OP ? (tail ? &s.maps->b_tail : &s.maps->b) : (tail ? &s.maps->a_tail : &s.maps->a);
    const int r = tail ? t.unit * s.unit_rows + t.r0 : t.r0, u = tail ? 0 : t.unit;
    const int copies = s.halves ? 1 : D / 64, last = s.halves ? 0 : s.b;
    for (int c = 0; c < copies; ++c)
      asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                   ::"r"(dst + c * (ROWS * 128)), "l"(map), "r"(bar), "r"(c * 64), "r"(s.h), "r"(r), "r"(u), "r"(last) : "memory");
  } else {
    const int lane = threadIdx.x & 31;
    const char* from = reinterpret_cast<const char*>(OP ? t.b : t.a);
    const int64_t row = OP ? s.b_row : s.a_row;
#pragma unroll 4
    for (int i = lane; i < ROWS * (D / 8); i += 32) {
      const int r = i / (D / 8), c = i % (D / 8);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                   ::"r"(dst + ring_at<ROWS>(r, c)), "l"(from + (r < t.n ? r * row : 0) + c * 16), "r"(r < t.n ? 16 : 0) : "memory");
    }
    cp_async_arrive(full);
  }
}

// The ring of a thread block: a stage is one tile of either operand, read by `readers` warps.  A single reader has a
// barrier per operand and refills each as soon as it is done with it.  Several readers share one barrier per stage and
// let go of both operands together; then warp 0 refills the first operand and warp 1 the second (issuing a copy costs
// its warp some hundred cycles, so the two share it).  `get(i)` gives the ring's i-th tile.  AUX (several readers
// only): two fp32 values per row come along, from aux_a and aux_b at RingTile::aux.
template <int D, int ROWS, bool TMA, bool AUX = false>
struct Ring {
  uint32_t mem;                 // shared-memory address of stage 0
  uint64_t* bars;               // full of each operand, empty: [3][stage]
  int* abort;
  int count, stages, warp, readers;      // tiles of this ring, ...
  const float *aux_a, *aux_b;
  uint32_t aux_mem;             // [stage][2][ROWS] floats
  int stage, parity;            // of the stage being read

  __device__ __forceinline__ uint64_t* full(int op, int s) const { return bars + (readers == 1 ? op : 0) * kRingMaxStages + s; }
  __device__ __forceinline__ uint64_t* empty(int s) const { return bars + 2 * kRingMaxStages + s; }
  __device__ __forceinline__ uint32_t at(int op, int s) const { return mem + static_cast<uint32_t>(2 * s + op) * kRingTile<D, ROWS>; }
  __device__ __forceinline__ uint32_t tile(int op) const { return at(op, stage); }

  // initialises the barriers (a block barrier has to follow)
  __device__ __forceinline__ void init() {
    stage = 0;
    parity = 0;
    if (warp == 0 && (threadIdx.x & 31) == 0) {
      for (int i = 0; i < stages; ++i) {
        const int fills = (TMA ? 1 : 32) * (readers == 1 ? 1 : 2) + (AUX ? 32 : 0);
        tc::mbar_init(full(0, i), fills);
        if (readers == 1) tc::mbar_init(full(1, i), fills);
        tc::mbar_init(empty(i), readers);
      }
      tc::fence_barrier_init();
    }
  }
  template <int OP> __device__ __forceinline__ void fill(int s, const RingTile& t, const RingSource& src) {
    if (!TMA || (threadIdx.x & 31) == 0) ring_fill<D, ROWS, TMA, OP>(at(OP, s), full(OP, s), t, src);
    if constexpr (AUX && OP == 1) {
#pragma unroll
      for (int y = 0; y < 2 * ROWS; y += 32) {
        const int i = y + (threadIdx.x & 31), r = i % ROWS, which = i / ROWS;
        const float* from = (which ? aux_b : aux_a) + t.aux + (r < t.n ? r : 0);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                     ::"r"(aux_mem + static_cast<uint32_t>((s * 2 + which) * ROWS + r) * 4), "l"(from), "r"(r < t.n ? 4 : 0) : "memory");
      }
      cp_async_arrive(full(0, s));
    }
  }
  // this warp's share of stage s := tile i
  template <typename Get> __device__ __forceinline__ void fill_both(int s, int i, const RingSource& src, Get&& get) {
    if (readers == 1) {
      const RingTile t = get(i);
      fill<0>(s, t, src);
      fill<1>(s, t, src);
    } else if (warp == 0) {
      fill<0>(s, get(i), src);
    } else if (warp == 1) {
      fill<1>(s, get(i), src);
    }
  }
  template <typename Get> __device__ __forceinline__ void start(const RingSource& src, Get&& get) {
    for (int i = 0; i < stages && i < count; ++i) fill_both(i, i, src, get);
  }
  template <int OP> __device__ __forceinline__ bool wait() {
    return (OP == 1 && readers > 1) || tc::mbar_wait(full(OP, stage), parity, abort);
  }
  // by every reading warp after its last access to operand OP of tile i (several readers: to the stage)
  template <int OP, typename Get> __device__ __forceinline__ bool release(int i, const RingSource& src, Get&& get) {
    const int next = i + stages;
    if (readers == 1) {
      __syncwarp();
      if (next < count) fill<OP>(stage, get(next), src);
      return true;
    }
    if (OP == 0) return true;
    __syncwarp();
    if ((threadIdx.x & 31) == 0) tc::mbar_arrive(empty(stage));
    if (warp > 1 || next >= count) return true;
    if (!tc::mbar_wait(empty(stage), parity, abort)) return false;
    fill_both(stage, next, src, get);
    return true;
  }
  __device__ __forceinline__ void step() {
    if (++stage == stages) { stage = 0; parity ^= 1; }
  }
};

// A visible block of one (batch, group, head) list: its 32-row tiles are tiles [first, first of the next slot).
struct RingSlot {
  uint64_t a, b;       // cp.async loader: addresses of row 0 of either operand; TMA: the unit, the rows that a copy brings
  int n_vis, first;    // rows that count, first tile
};
inline size_t ring_list_bytes(int T) { return (static_cast<size_t>(T) + 1) * sizeof(RingSlot); }

// The visible blocks of a list, in list order and with a sentinel at the end, written by one warp; returns their tiles.
template <int ESZ, bool TMA>
__device__ __forceinline__ int ring_list(RingSlot* out, const KVSrc& kv, const int32_t* ids, int64_t ids_off, int64_t ids_st,
                                         int T, int b, int h, int D, int block_size, int chunk_size, bool causal, int q_chunk) {
  constexpr int ROWS = 32;
  const int lane = threadIdx.x & 31;
  int count = 0, slots = 0;
  for (int t0 = 0; t0 < T; t0 += 32) {
    BlockRef r{nullptr, nullptr, 0};
    int unit = 0;
    const int t = t0 + lane;
    if (t < T) {
      const int64_t at = ids_off + t * ids_st;
      if (kv.mode == NSA_KV_PTR) {
        const int64_t ak = kv.ptr_k[at], av = kv.ptr_v[at];
        if (ak != 0 && av != 0) {
          r.k = reinterpret_cast<const char*>(static_cast<uintptr_t>(ak));
          r.v = reinterpret_cast<const char*>(static_cast<uintptr_t>(av));
          r.n_vis = block_size;
        }
      } else {
        unit = ids[at];
        r = resolve_block<ESZ>(kv, b, h, unit, D, block_size, chunk_size, causal, q_chunk);
        if (r.n_vis > 0 && kv.mode == NSA_KV_PAGED) unit = kv.block_table[static_cast<int64_t>(h) * kv.max_blocks + unit];
      }
    }
    const int mine = (r.n_vis + ROWS - 1) / ROWS;
    int upto = mine;                                 // inclusive prefix sum over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += y;
    }
    const uint32_t some = __ballot_sync(0xffffffffu, mine > 0);
    if (mine > 0) {
      // (a cut-off last block of a dense tensor: what follows it is outside the tensor and arrives as zeros)
      const int64_t there = kv.mode == NSA_KV_DENSE ? kv.n_tokens - static_cast<int64_t>(unit) * block_size : block_size;
      out[slots + __popc(some & ((1u << lane) - 1))] =
          RingSlot{TMA ? static_cast<uint64_t>(unit) : reinterpret_cast<uint64_t>(r.k),
                   TMA ? static_cast<uint64_t>(there < block_size ? there : block_size) : reinterpret_cast<uint64_t>(r.v), r.n_vis,
                   count + upto - mine};
    }
    slots += __popc(some);
    count += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (lane == 0) out[slots].first = count;
  __syncwarp();
  return count;
}

// Tile i of a list: no block has more than `per_block` tiles and few (cut off, partly visible) have less, so the search
// starts at slot i / per_block and hardly ever goes on.
__device__ __forceinline__ const RingSlot& ring_slot(const RingSlot* list, int i, int per_block) {
  if (per_block == 1) return list[i];
  int s = i / per_block;
  while (list[s + 1].first <= i) ++s;
  return list[s];
}
template <bool TMA>
__device__ __forceinline__ RingTile ring_tile(const RingSlot* list, int i, int per_block, const RingSource& src) {
  const RingSlot& w = ring_slot(list, i, per_block);
  const int r0 = (i - w.first) * 32, n = min(32, w.n_vis - r0);
  if (!TMA) return RingTile{w.a + r0 * src.a_row, w.b + r0 * src.b_row, 0, r0, n, n, 0};
  return RingTile{0, 0, static_cast<int>(w.a), r0, n, min(32, static_cast<int>(w.b) - r0), 0};
}

template <int ESZ>
__device__ __forceinline__ RingSource kv_ring_source(const KVSrc& kv, const RingMaps& maps, int B, int b, int h, int D, int block_size) {
  const bool paged = kv.mode == NSA_KV_PAGED;
  return RingSource{&maps, kv_row_bytes(kv, false, D, ESZ), kv_row_bytes(kv, true, D, ESZ), paged ? 0 : h, b, block_size,
                    paged ? 0x7fffffff : static_cast<int>(kv.n_tokens / block_size), B == 1};
}

// ---- host side
// Maps of rows of one dense operand [B,N,H,D] in units of `unit` rows, boxes of `rows` rows x 64 columns; `tail`
// takes the unit that the end of the tensor cuts off.  False: not describable (the caller loads with cp.async).
// join_halves: with one batch element the map's last dimension is the 64-column half, so that one copy brings whole rows.
bool make_unit_maps(CUtensorMap* whole, CUtensorMap* tail, const void* base, const int64_t* stride, int B, int64_t N, int H,
                    int D, int unit, int rows, bool join_halves = true);
// The same for the K and V of a source (a pool's units are its pages).
bool make_ring_maps(const nsa_kv_source* kv, int B, int H, int D, int unit, int rows, RingMaps* maps);
int device_status_address(int32_t** out);

// dK / dV on the tensor cores (sel_bwd_dkv_rows_tc.cu).
struct DkvRowsArgs {
  const char *q, *dO;                    // [B,M,H,D]
  char *dk, *dv;                         // contiguous [B,N,H,D]
  const float *lse, *delta;              // [B,H,M]
  const int32_t *groups, *offsets;       // [B,H,MG*T], [B,H,NS+1]
  KVSrc kv;
  int B, H, T, block_size, chunk_size, causal, G, MG, whole;   // whole: query groups in front of a cut-off one
  int64_t M, NS;
  float scale, scale_log2;
};
int try_launch_sel_bwd_dkv_rows_tc(DkvRowsArgs p, const int64_t* q_stride, const int64_t* do_stride, int D, int dtype,
                                   int32_t* status, cudaStream_t stream, bool* launched);

}  // namespace nsa
