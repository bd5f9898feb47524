// Where a freshly projected K or V element of token row `row`, model column `c` goes:
// the context cache during prefill, the private buffer cache (in-place append) otherwise.
#pragma once
#include "common.cuh"

namespace artab {

template <typename T>
__device__ __forceinline__ void scatter_k(const KvDest& kv, long row, int c, float val) {
  const int h = c / kv.head_dim, d = c - h * kv.head_dim;
  if (kv.mode == KV_PREFILL) {
    const long g = row / kv.n_ctx, i = row - g * kv.n_ctx;
    reinterpret_cast<T*>(kv.k_ctx)[((size_t)(g * kv.n_heads + h) * kv.n_ctx_pad + i) * kv.head_dim + d] =
        from_f32<T>(val);
  } else {
    const long b = row / kv.tokens_per_stream;
    const int j = (int)(row - b * kv.tokens_per_stream);
    if (j >= kv.n_kv_tokens) return;
    reinterpret_cast<T*>(kv.kv_buf)[(((size_t)(b * kv.n_heads + h) * kv.max_buf + kv.pos0 + j) * 2) * kv.head_dim + d] =
        from_f32<T>(val);
  }
}

template <typename T>
__device__ __forceinline__ void scatter_v(const KvDest& kv, long row, int c, float val) {
  const int h = c / kv.head_dim, d = c - h * kv.head_dim;
  if (kv.mode == KV_PREFILL) {
    const long g = row / kv.n_ctx, i = row - g * kv.n_ctx;
    if (kv.dtype == ARTAB_BF16) {  // transposed, split into a bf16 hi and lo part: [.., 2*Dh][Ncp]
      T* vb = reinterpret_cast<T*>(kv.v_ctx) + ((size_t)(g * kv.n_heads + h) * 2 * kv.head_dim) * kv.n_ctx_pad + i;
      const T hi = from_f32<T>(val);
      vb[(size_t)d * kv.n_ctx_pad] = hi;
      vb[(size_t)(kv.head_dim + d) * kv.n_ctx_pad] = from_f32<T>(val - to_f32<T>(hi));
    } else {
      reinterpret_cast<T*>(kv.v_ctx)[((size_t)(g * kv.n_heads + h) * kv.n_ctx_pad + i) * kv.head_dim + d] =
          from_f32<T>(val);
    }
  } else {
    const long b = row / kv.tokens_per_stream;
    const int j = (int)(row - b * kv.tokens_per_stream);
    if (j >= kv.n_kv_tokens) return;
    reinterpret_cast<T*>(
        kv.kv_buf)[(((size_t)(b * kv.n_heads + h) * kv.max_buf + kv.pos0 + j) * 2 + 1) * kv.head_dim + d] =
        from_f32<T>(val);
  }
}

// four neighbouring values into the cache type
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&v)[4]) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  }
}

// K (which = 1) or V (2) of token row `row`, columns c .. c + 3 (inside one head), four elements at a time
template <typename T>
__device__ __forceinline__ void scatter4(const KvDest& kv, int which, unsigned row, int c, const float (&v)[4]) {
  const int h = c / kv.head_dim, d = c - h * kv.head_dim;
  if (kv.mode == KV_PREFILL) {
    const unsigned g = row / (unsigned)kv.n_ctx, i = row - g * kv.n_ctx;
    const size_t gh = (size_t)g * kv.n_heads + h;
    if (which == 2 && sizeof(T) == 2) {  // transposed, bf16 hi and lo parts
      T* p = reinterpret_cast<T*>(kv.v_ctx) + (gh * 2 * kv.head_dim + d) * kv.n_ctx_pad + i;
#pragma unroll
      for (int e = 0; e < 4; ++e, p += kv.n_ctx_pad) {
        const T hi = from_f32<T>(v[e]);
        p[0] = hi;
        p[(size_t)kv.head_dim * kv.n_ctx_pad] = from_f32<T>(v[e] - to_f32<T>(hi));
      }
    } else {
      store4<T>(reinterpret_cast<T*>(which == 1 ? kv.k_ctx : kv.v_ctx) + (gh * kv.n_ctx_pad + i) * kv.head_dim + d, v);
    }
  } else {
    const unsigned b = row / (unsigned)kv.tokens_per_stream, j = row - b * kv.tokens_per_stream;
    if ((int)j >= kv.n_kv_tokens) return;
    store4<T>(reinterpret_cast<T*>(kv.kv_buf) +
                  ((((size_t)b * kv.n_heads + h) * kv.max_buf + kv.pos0 + j) * 2 + which - 1) * kv.head_dim + d, v);
  }
}

}  // namespace artab
