// Elementwise and row-wise work of a transformer layer around the attention, one pass per stop of the residual
// stream: residual add + layer norm + modulation, root-mean-square norm of the query / key projections + rotary
// embedding.  HBM-bound; 16-byte accesses, the whole row in registers.  Values are rounded to
// the activations' type where the eager tensors are.
#include "common.cuh"
#include "rope.cuh"

#include <type_traits>

namespace nsa {
namespace {

constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}
template <typename T> __device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = unpack2<T>(w[i]);
    f[2 * i] = x.x;
    f[2 * i + 1] = x.y;
  }
}
template <typename T> __device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack2<T>(f[0], f[1]), pack2<T>(f[2], f[3]), pack2<T>(f[4], f[5]), pack2<T>(f[6], f[7]));
}
template <typename T> __device__ __forceinline__ float round_to(float x) { return to_f32<T>(from_f32<T>(x)); }
// 8 values of a vector that is the sum of a T row and an fp32 row (either may be absent)
template <typename T> __device__ __forceinline__ void vector8(const void* mod, const float* e, int at, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = 0.f;
  if (mod != nullptr) unpack8<T>(__ldg(reinterpret_cast<const uint4*>(static_cast<const char*>(mod) + at * 2)), f);
  if (e != nullptr) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(e + at)), b = __ldg(reinterpret_cast<const float4*>(e + at + 4));
    f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
    f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
  }
}

struct NormParams {
  const char* x; const char* y;
  const void *gate_mod, *scale_mod, *shift_mod;
  const float *gate_e, *scale_e, *shift_e;
  char* x_out; char* h_out;
  int64_t rows;
  int d, gated, modulated;
  float eps;
};

// A thread owns one 16-byte column of R rows: the gate, scale and shift values of its column are read once per R rows
// (a warp per row read 15 KB of them for every 3 KB row), the row sums go through shared memory.
// 390 rows of 1536, gated residual, modulated norm: 9.1 -> 4.0 us; 4680 rows: 18.0 -> 15.4 us.
template <typename T, int R>
__global__ void __launch_bounds__(256) residual_norm_kernel(const NormParams p) {
  __shared__ float s_sum[2][8][R];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, at = threadIdx.x * 8;
  const bool on = at < p.d;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * R;
  const int n = static_cast<int>(p.rows - row0 < R ? p.rows - row0 : R);
  const int64_t base = (row0 * p.d + at) * 2, step = static_cast<int64_t>(p.d) * 2;
  chain_release();
  chain_wait();
  uint4 xs[R], ys[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {                                   // all loads first
    const bool there = on && r < n;
    xs[r] = there ? *reinterpret_cast<const uint4*>(p.x + base + r * step) : make_uint4(0, 0, 0, 0);
    ys[r] = there && p.y != nullptr ? *reinterpret_cast<const uint4*>(p.y + base + r * step) : make_uint4(0, 0, 0, 0);
  }
  float v[R][8], sum[R];
  float g[8], a[8], b[8];
  if (on) {
    if (p.gated) vector8<T>(p.gate_mod, p.gate_e, at, g);
    if (p.h_out != nullptr) {
      vector8<T>(p.scale_mod, p.scale_e, at, a);
      vector8<T>(p.shift_mod, p.shift_e, at, b);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    unpack8<T>(xs[r], v[r]);
    if (p.y != nullptr && on && r < n) {
      float y[8];
      unpack8<T>(ys[r], y);
      if (p.gated) {                                              // x + (y.float() * gate).to(T), rounded again
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = round_to<T>(y[e] * g[e]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) v[r][e] = round_to<T>(v[r][e] + y[e]);
      *reinterpret_cast<uint4*>(p.x_out + base + r * step) = pack8<T>(v[r]);
    }
    sum[r] = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) sum[r] += v[r][e];
  }
  if (p.h_out == nullptr) return;
  const auto row_sums = [&](float (&x)[R], int turn) {            // over the block
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = warp_sum(x[r]);
    if (warps == 1) return;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane == r) s_sum[turn][warp][r] = x[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      x[r] = 0.f;
      for (int w = 0; w < warps; ++w) x[r] += s_sum[turn][w][r];
    }
  };
  row_sums(sum, 0);
  float sq[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float mean = sum[r] / static_cast<float>(p.d);
    sq[r] = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[r][e] -= mean;
      sq[r] += on ? v[r][e] * v[r][e] : 0.f;
    }
  }
  row_sums(sq, 1);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (!on || r >= n) continue;
    const float rstd = rsqrtf(sq[r] / static_cast<float>(p.d) + p.eps);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[r][e] = v[r][e] * rstd * (p.modulated ? 1.f + a[e] : a[e]) + b[e];
    *reinterpret_cast<uint4*>(p.h_out + base + r * step) = pack8<T>(v[r]);
  }
}

template <typename T, int R> int launch_residual_norm(const NormParams& p, cudaStream_t s) {
  NSA_CUDA_OK(launch_chained(kChainSmall, residual_norm_kernel<T, R>, dim3(static_cast<unsigned>(cdiv64(p.rows, R))),
                             dim3(cdiv(p.d / 8, 32) * 32), 0, s, p));
  NSA_LAUNCH_OK("residual_norm_kernel");
  return NSA_OK;
}
// 4680 rows: 17.6 / 15.4 / 20.7 us with 1 / 2 / 4 rows per thread block; 1560 rows: 8.0 / 7.5 / 10.9 us; a few hundred
// rows want as many thread blocks as they can give.
template <typename T> int launch_residual_norm(const NormParams& p, cudaStream_t s) {
  return p.rows >= 4 * 148 ? launch_residual_norm<T, 2>(p, s) : launch_residual_norm<T, 1>(p, s);
}

struct RmsParams {
  const char* x; const void* w; char* out;
  int64_t rows, row_stride;
  int d;
  float eps;
};
template <typename T, int C>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) rms_rows_kernel(const RmsParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  chain_release();
  chain_wait();
  if (row >= p.rows) return;
  const int pieces = p.d / 8;
  const char* x = p.x + row * p.row_stride * 2;
  float v[C][8], sq = 0.f;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int i = c * 32 + lane;
    unpack8<T>(i < pieces ? *reinterpret_cast<const uint4*>(x + i * 16) : make_uint4(0, 0, 0, 0), v[c]);
#pragma unroll
    for (int e = 0; e < 8; ++e) sq += v[c][e] * v[c][e];
  }
  const float r = rsqrtf(warp_sum(sq) / static_cast<float>(p.d) + p.eps);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int i = c * 32 + lane;
    if (i >= pieces) continue;
    float w[8];
    vector8<T>(p.w, nullptr, i * 8, w);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[c][e] = v[c][e] * r * w[e];
    *reinterpret_cast<uint4*>(p.out + row * p.d * 2 + i * 16) = pack8<T>(v[c]);
  }
}

// Queries and keys of one token: norm over all heads, then the rotary embedding.  32 lanes x 16 bytes are whole
// heads (D / 8 divides 32), so a lane meets the same pairs of a head in every piece and needs only their four factors.
struct QkParams : RopeParams {
  const char* q; const char* k;
  const void *qw, *kw;
  char* q_out; char* k_out;
  int64_t S, row_stride, k_out_stride;
  int d, D;
  float eps;
};
template <typename T, int C>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) qk_norm_rope_kernel(const QkParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  int fr = 0, hr = 0, wr = 0;
  if (t < p.S) rope_position(p, t, fr, hr, wr);
  chain_release();
  chain_wait();
  if (t >= p.S) return;
  // (the tables too may have been written by the kernel in front of this one)
  const int j0 = lane % (p.D / 8) * 4;
  double2 f[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = rope_factor(p, j0 + i, fr, hr, wr);
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const char* x = (which ? p.k : p.q) + t * p.row_stride * 2;
    char* out = which ? p.k_out + t * p.k_out_stride * 2 : p.q_out + t * p.d * 2;
    float v[C][8], sq = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      unpack8<T>(*reinterpret_cast<const uint4*>(x + (c * 32 + lane) * 16), v[c]);
#pragma unroll
      for (int e = 0; e < 8; ++e) sq += v[c][e] * v[c][e];
    }
    const float r = rsqrtf(warp_sum(sq) / static_cast<float>(p.d) + p.eps);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      float w[8];
      vector8<T>(which ? p.kw : p.qw, nullptr, (c * 32 + lane) * 8, w);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[c][e] = v[c][e] * r * w[e];
      uint4 o = pack8<T>(v[c]);
      T* e = reinterpret_cast<T*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) rope_pair<T>(e[2 * i], e[2 * i + 1], f[i]);
      *reinterpret_cast<uint4*>(out + (c * 32 + lane) * 16) = o;
    }
  }
}

// calls f with the smallest built number of 16-byte pieces per lane that covers a row
template <typename F> int with_pieces(int pieces, F&& f) {
  const int c = cdiv(pieces, 32);
  if (c <= 1) return f(std::integral_constant<int, 1>());
  if (c <= 2) return f(std::integral_constant<int, 2>());
  if (c <= 4) return f(std::integral_constant<int, 4>());
  if (c <= 6) return f(std::integral_constant<int, 6>());
  return f(std::integral_constant<int, 8>());
}
unsigned row_blocks(int64_t rows) { return static_cast<unsigned>(cdiv64(rows, kWarpsPerBlock)); }

int check_rows(const char* what, int64_t rows, int d, int dtype) {
  NSA_REQUIRE(rows >= 0 && rows <= 0x7fffffffll && d > 0, NSA_ERR_INVALID, "%s: bad size", what);
  NSA_REQUIRE(d % 8 == 0 && d <= 2048, NSA_ERR_UNSUPPORTED, "%s: row length %d (a multiple of 8, at most 2048)", what, d);
  NSA_REQUIRE(dtype == NSA_BF16 || dtype == NSA_F16, NSA_ERR_UNSUPPORTED, "%s: bf16 / fp16 only", what);
  return NSA_OK;
}

}  // namespace
}  // namespace nsa

using namespace nsa;

extern "C" int nsa_residual_norm(const void* x, const void* y, const void* gate_mod, const float* gate_e,
                                 const void* scale_mod, const float* scale_e, const void* shift_mod, const float* shift_e,
                                 int32_t modulated, void* x_out, void* h_out, int64_t rows, int32_t d, float eps,
                                 int32_t dtype, void* stream) {
  int rc;
  if ((rc = check_rows("residual_norm", rows, d, dtype))) return rc;
  if (rows == 0) return NSA_OK;
  NSA_REQUIRE(x && (y == nullptr || x_out) && (y || h_out), NSA_ERR_INVALID, "residual_norm: null pointer");
  const void* ptrs[11] = {x, y, gate_mod, gate_e, scale_mod, scale_e, shift_mod, shift_e, x_out, h_out, nullptr};
  for (const void* q : ptrs) NSA_REQUIRE(aligned16(q), NSA_ERR_LAYOUT, "residual_norm: pointers must be 16-byte aligned");
  const NormParams p{static_cast<const char*>(x), static_cast<const char*>(y), gate_mod, scale_mod, shift_mod, gate_e, scale_e,
                     shift_e, static_cast<char*>(x_out), static_cast<char*>(h_out), rows, d,
                     gate_mod != nullptr || gate_e != nullptr, modulated, eps};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == NSA_BF16 ? launch_residual_norm<__nv_bfloat16>(p, s) : launch_residual_norm<__half>(p, s);
}

extern "C" int nsa_rms_rows(const void* x, int64_t row_stride, const void* weight, void* out, int64_t rows, int32_t d,
                            float eps, int32_t dtype, void* stream) {
  int rc;
  if ((rc = check_rows("rms_rows", rows, d, dtype))) return rc;
  if (rows == 0) return NSA_OK;
  NSA_REQUIRE(x && weight && out, NSA_ERR_INVALID, "rms_rows: null pointer");
  NSA_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(out) && row_stride % 8 == 0, NSA_ERR_LAYOUT,
              "rms_rows: rows must be 16-byte aligned");
  const RmsParams p{static_cast<const char*>(x), weight, static_cast<char*>(out), rows, row_stride, d, eps};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rc = with_pieces(d / 8, [&](auto c) -> int {
    NSA_CUDA_OK(dtype == NSA_BF16
                    ? launch_chained(kChainSmall, rms_rows_kernel<__nv_bfloat16, c.value>, dim3(row_blocks(rows)), dim3(kWarpsPerBlock * 32), 0, s, p)
                    : launch_chained(kChainSmall, rms_rows_kernel<__half, c.value>, dim3(row_blocks(rows)), dim3(kWarpsPerBlock * 32), 0, s, p));
    return NSA_OK;
  });
  if (rc) return rc;
  NSA_LAUNCH_OK("rms_rows_kernel");
  return NSA_OK;
}

extern "C" int nsa_qk_norm_rope(const void* q, const void* k, int64_t row_stride, const void* q_weight, const void* k_weight,
                                float eps, int64_t S, int32_t H, int32_t D, void* q_out, void* k_out, int64_t k_out_stride,
                                const nsa_rope* rope, int32_t dtype, void* stream) {
  int rc;
  const int d = H * D;
  if ((rc = check_rows("qk_norm_rope", S, d, dtype))) return rc;
  NSA_REQUIRE(D % 8 == 0 && 32 % (D / 8) == 0 && (d == 256 || d == 512 || d == 1024 || d == 1536 || d == 2048), NSA_ERR_UNSUPPORTED,
              "qk_norm_rope: built for rows of 256, 512, 1024, 1536 or 2048 elements and head dims that divide 256, got %d x %d", H, D);
  if (S == 0) return NSA_OK;
  NSA_REQUIRE(q && k && q_weight && k_weight && q_out && k_out && rope, NSA_ERR_INVALID, "qk_norm_rope: null pointer");
  NSA_REQUIRE(aligned16(q) && aligned16(k) && aligned16(q_weight) && aligned16(k_weight) && aligned16(q_out) && aligned16(k_out) &&
                  row_stride % 8 == 0 && k_out_stride % 8 == 0, NSA_ERR_LAYOUT, "qk_norm_rope: rows must be 16-byte aligned");
  QkParams p{{}, static_cast<const char*>(q), static_cast<const char*>(k), q_weight, k_weight, static_cast<char*>(q_out),
             static_cast<char*>(k_out), S, row_stride, k_out_stride, d, D, eps};
  if ((rc = set_rope(rope, S, D, &p))) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rc = with_pieces(d / 8, [&](auto c) -> int {
    NSA_CUDA_OK(dtype == NSA_BF16
                    ? launch_chained(kChainSmall, qk_norm_rope_kernel<__nv_bfloat16, c.value>, dim3(row_blocks(S)), dim3(kWarpsPerBlock * 32), 0, s, p)
                    : launch_chained(kChainSmall, qk_norm_rope_kernel<__half, c.value>, dim3(row_blocks(S)), dim3(kWarpsPerBlock * 32), 0, s, p));
    return NSA_OK;
  });
  if (rc) return rc;
  NSA_LAUNCH_OK("qk_norm_rope_kernel");
  return NSA_OK;
}
