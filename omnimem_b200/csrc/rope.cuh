// Rotary embedding of a chunk's tokens (causal_reorder_rope_apply,
// models/transformers/causal_wan_nsa_model.py:72-105): token t of the chunk, in the reordered order
// (f h w fs hs ws), sits at frame / row / column (fr, hr, wr) of the chunk's latent grid; complex pair j of a
// head takes its factor from the frame table (j < c_f, row start_frame + fr), the row table (next c_h pairs)
// or the column table (last c_w pairs); products in float64.
#pragma once

#include "common.cuh"

namespace nsa {

struct RopeParams {
  const double2* rope_f; const double2* rope_h; const double2* rope_w;
  int c_f, c_h, c_w;
  int grid_h, grid_w, pool_f, pool_h, pool_w, start_frame;
};

// frame / row / column of token t of a chunk stored in (f h w fs hs ws) order
template <typename I>
__device__ __forceinline__ void rope_position_t(const RopeParams& p, I t, int& fr, int& hr, int& wr) {
  const I pw = static_cast<I>(p.pool_w), ph = static_cast<I>(p.pool_h), pf = static_cast<I>(p.pool_f);
  const int ws = static_cast<int>(t % pw); t /= pw;
  const int hs = static_cast<int>(t % ph); t /= ph;
  const int fs = static_cast<int>(t % pf); t /= pf;
  const I wq = static_cast<I>(p.grid_w / p.pool_w), hq = static_cast<I>(p.grid_h / p.pool_h);
  const int wo = static_cast<int>(t % wq); t /= wq;
  const int ho = static_cast<int>(t % hq); t /= hq;
  fr = static_cast<int>(t) * p.pool_f + fs;
  hr = ho * p.pool_h + hs;
  wr = wo * p.pool_w + ws;
}
// (five divisions per call: in 32 bits whenever the token index allows, a 64-bit division costs
// several times as many instructions and this runs once per row and thread)
__device__ __forceinline__ void rope_position(const RopeParams& p, int64_t t, int& fr, int& hr, int& wr) {
  if (static_cast<uint64_t>(t) <= 0xffffffffull) rope_position_t<uint32_t>(p, static_cast<uint32_t>(t), fr, hr, wr);
  else rope_position_t<int64_t>(p, t, fr, hr, wr);
}
// factor of complex pair j of a head for a token at (fr, hr, wr): one load through a selected table instead of
// three branches (a warp's threads sit in different tables)
__device__ __forceinline__ double2 rope_factor(const RopeParams& p, int j, int fr, int hr, int wr) {
  const bool in_f = j < p.c_f, in_h = j < p.c_f + p.c_h;
  const double2* tb = in_f ? p.rope_f + j : in_h ? p.rope_h + (j - p.c_f) : p.rope_w + (j - p.c_f - p.c_h);
  const int len = in_f ? p.c_f : in_h ? p.c_h : p.c_w;
  const int at = in_f ? p.start_frame + fr : in_h ? hr : wr;
  return tb[static_cast<int64_t>(at) * len];
}
// float64 product, then float64 -> float32 -> T, as view_as_real(...).type_as(x) does
template <typename T>
__device__ __forceinline__ void rope_pair(T& re, T& im, const double2 w) {
  const double xr = static_cast<double>(to_f32<T>(re)), xi = static_cast<double>(to_f32<T>(im));
  re = from_f32<T>(static_cast<float>(xr * w.x - xi * w.y));
  im = from_f32<T>(static_cast<float>(xr * w.y + xi * w.x));
}

int set_rope(const nsa_rope* rope, int64_t S, int32_t D, RopeParams* p);

}  // namespace nsa
