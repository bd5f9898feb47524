// Context attention in fp32 FMA: queries of many streams against one shared (or one per-group) context.
//
// This is the context kernel of the fp32 mode and of head sizes the tensor-core kernel is not built for.  A
// warp owns 2, 4 or 8 query rows and walks the keys in tiles of 32 (attn_tile.cuh); the eight warps of a CTA share
// the K / V tiles, which asynchronous copies bring into the lane order of the tile loop while the previous
// 64 keys are worked on.  Per tile and 8 rows that is 28 - 56 16-byte shared-memory reads for 8 * 32 * 2 * Dh FMAs;
// its predecessor read six words for every eight FMAs.
#include "attn.cuh"
#include "attn_tile.cuh"

namespace artab {

namespace {

constexpr int kWarps = 8;
constexpr int kStage = 64;   // keys of a stage: two tiles

template <int DH, int NR>
struct Smem {
  static constexpr int QP = DH + 4;
  float4 kv[2][2][16 * DH];                                  // [stage][tile]: K in lane order, then V
  float q[kWarps][NR][QP];
  float pw[kWarps][NR * (DH > 32 ? DH : 32)];                // softmax numerators, later the warp's result
  float ml[kWarps][NR * 2];
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const uint32_t n = valid ? 16u : 0u;  // 0 source bytes: the 16 destination bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}

// four neighbouring elements from an address that only has the element's alignment
template <typename T>
__device__ __noinline__ float4 load4_any(const T* p) {
  return make_float4(to_f32<T>(p[0]), to_f32<T>(p[1]), to_f32<T>(p[2]), to_f32<T>(p[3]));
}

template <typename T, int DH, int NR>
__global__ void __launch_bounds__(kWarps * 32, 2) ctx_attn_fma_kernel(const CtxAttnArgs a) {
  extern __shared__ __align__(128) uint8_t raw[];
  using S = Smem<DH, NR>;
  S& sm = *reinterpret_cast<S*>(raw);
  constexpr int D4 = DH / 4, NI = DH / 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int h = blockIdx.y;
  const int g = blockIdx.z / a.n_splits, split = blockIdx.z - g * a.n_splits;
  const int rows_in_group = a.n_groups == 1 ? a.rows : a.rows_per_group;
  const long group_row0 = a.n_groups == 1 ? 0 : (long)g * a.rows_per_group;
  const int q0 = (blockIdx.x * kWarps + warp) * NR;          // first row of this warp in its group

  const int tiles = (a.n_ctx + kStage - 1) / kStage;
  const int tps = (tiles + a.n_splits - 1) / a.n_splits;
  const int k_begin = split * tps * kStage;
  const int k_end = min(a.n_ctx, k_begin + tps * kStage);

  const T* Q = reinterpret_cast<const T*>(a.q);
  const T* Kc = reinterpret_cast<const T*>(a.k_ctx) + (size_t)(g * a.n_heads + h) * a.n_ctx_pad * DH;
  const T* Vc = reinterpret_cast<const T*>(a.v_ctx) + (size_t)(g * a.n_heads + h) * a.n_ctx_pad * DH * (a.v_transposed ? 2 : 1);

  // A caller's own K / V may start anywhere, and transposed V may have any pitch: wide loads need 16-byte aligned
  // arrays and pitches of whole float4s.
  const bool wide = (((uintptr_t)a.k_ctx | (uintptr_t)a.v_ctx) & 15) == 0 && (!a.v_transposed || (a.n_ctx_pad & 3) == 0);

  // keys [k0, k0 + 64) -> stage st; float4 (key, dims 4d .. 4d + 3) of K sits at [d / 4][key % 4][d % 4][key / 4], of V at
  // [key % NI][key / NI][d]
  auto stage = [&](int k0, int st) {
    for (int i = tid; i < kStage * D4; i += kWarps * 32) {
      const int key = i / D4, d = i - key * D4, t = key >> 5, kt = key & 31;
      float4* kd = &sm.kv[st][t][((d >> 2) * 4 + (kt & 3)) * 32 + (d & 3) * 8 + (kt >> 2)];
      float4* vd = &sm.kv[st][t][8 * DH + (kt & (NI - 1)) * 32 + kt / NI * D4 + d];
      const bool valid = k0 + key < k_end;
      const size_t at = (size_t)(valid ? k0 + key : 0) * DH + 4 * d;
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!wide) {
        *kd = valid ? load4_any(Kc + at) : z;
        if (!a.v_transposed) *vd = valid ? load4_any(Vc + at) : z;
      } else if constexpr (sizeof(T) == 4) {
        cp_async16(kd, Kc + at, valid);
        if (!a.v_transposed) cp_async16(vd, Vc + at, valid);
      } else {
        *kd = valid ? load4(Kc + at) : z;
        if (!a.v_transposed) *vd = valid ? load4(Vc + at) : z;
      }
    }
    if constexpr (sizeof(T) == 2) {
      if (a.v_transposed) {  // hi and lo parts, [2 Dh][Ncp]
        for (int i = tid; i < DH * (kStage / 4); i += kWarps * 32) {
          const int d = i / (kStage / 4), key = 4 * (i - d * (kStage / 4)), t = key >> 5, kt = key & 31;
          float v[4] = {0.f, 0.f, 0.f, 0.f};
          const T* vp = Vc + (size_t)d * a.n_ctx_pad + k0 + key;
          if (!wide) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (k0 + key + e < k_end) v[e] = to_f32<T>(vp[e]) + to_f32<T>(vp[(size_t)DH * a.n_ctx_pad + e]);
          } else if (k0 + key < k_end) {   // a pitch of whole float4s: the last one may reach into the padding
            const float4 hi = load4(vp), lo = load4(vp + (size_t)DH * a.n_ctx_pad);
            v[0] = hi.x + lo.x; v[1] = hi.y + lo.y; v[2] = hi.z + lo.z; v[3] = hi.w + lo.w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            reinterpret_cast<float*>(&sm.kv[st][t][8 * DH + ((kt + e) & (NI - 1)) * 32 + (kt + e) / NI * D4])[d] =
                k0 + key + e < k_end ? v[e] : 0.f;
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  for (int i = lane; i < NR * DH; i += 32) {
    const int r = i / DH, d = i - r * DH;
    sm.q[warp][r][d] = q0 + r < rows_in_group ? to_f32<T>(Q[((size_t)(group_row0 + q0 + r) * a.n_heads + h) * DH + d]) : 0.f;
  }
  TileState<DH, NR, S::QP> st;
  st.init();
  const float sc = a.scale * kLog2e;
  if (k_begin < k_end) stage(k_begin, 0);
  int cur = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += kStage, cur ^= 1) {
    if (k0 + kStage < k_end) {
      stage(k0 + kStage, cur ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < 2; ++t) {
      const int n_valid = k_end - k0 - 32 * t;
      if (n_valid <= 0) break;
      const float4* tile = sm.kv[cur][t] + lane;
      st.tile(&sm.q[warp][0][0], sm.pw[warp], n_valid, sc, [&](int j, int kk) { return tile[(4 * j + kk) * 32]; },
              [&](int i) { return tile[8 * DH + 32 * i]; });
    }
    __syncthreads();   // the stage may be refilled
  }
  __syncwarp();
  st.flush(sm.pw[warp], sm.ml[warp]);
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < NR * D4; i += 32) {
    const int r = i / D4, d = 4 * (i - r * D4);
    if (q0 + r >= rows_in_group) continue;
    const long row = group_row0 + q0 + r;
    const float m = sm.ml[warp][2 * r], l = sm.ml[warp][2 * r + 1];
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    const float4 o = *reinterpret_cast<const float4*>(&sm.pw[warp][r * DH + d]);
    const size_t ro = ((size_t)split * a.rows + row) * a.n_heads + h;
    float* dst = a.out + (a.out_lane_major ? lane_major_index(row, h * DH + d, a.n_heads * DH) : ro * DH + d);
    const float4 y = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    if (((uintptr_t)a.out & 15) == 0) {
      *reinterpret_cast<float4*>(dst) = y;
    } else {
      dst[0] = y.x; dst[1] = y.y; dst[2] = y.z; dst[3] = y.w;
    }
    if (d == 0) a.lse[ro] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
  }
}

template <typename T, int DH, int NR>
int launch_variant(const CtxAttnArgs& a, cudaStream_t s) {
  const int rows_in_group = a.n_groups == 1 ? a.rows : a.rows_per_group;
  const size_t smem = sizeof(Smem<DH, NR>);
  static SmemConfig configured;
  const cudaError_t e = configured.ensure(ctx_attn_fma_kernel<T, DH, NR>, smem, true);
  ARTAB_REQUIRE(e == cudaSuccess, ARTAB_ELAUNCH, "ctx_attn_fma_kernel: shared memory refused: %s", cudaGetErrorString(e));
  const dim3 grid((rows_in_group + kWarps * NR - 1) / (kWarps * NR), a.n_heads, a.n_groups * a.n_splits);
  prof_begin(PROF_CTX, s);
  ctx_attn_fma_kernel<T, DH, NR><<<grid, kWarps * 32, smem, s>>>(a);
  prof_end(s);
  count_launch();
  return check_launch("ctx_attn_fma_kernel");
}

template <typename T, int DH>
int launch_dh(const CtxAttnArgs& a, cudaStream_t s) {
  // eight rows per warp reuse a key tile best; with fewer rows in a group half-empty warps cost more than that
  switch (ctx_attn_fma_rows(a.n_groups == 1 ? a.rows : a.rows_per_group)) {
    case 2 * kWarps: return launch_variant<T, DH, 2>(a, s);
    case 4 * kWarps: return launch_variant<T, DH, 4>(a, s);
    default: return launch_variant<T, DH, 8>(a, s);
  }
}

template <typename T>
int launch_t(const CtxAttnArgs& a, cudaStream_t s) {
  switch (a.head_dim) {
    case 16: return launch_dh<T, 16>(a, s);
    case 32: return launch_dh<T, 32>(a, s);
    default: return launch_dh<T, 64>(a, s);
  }
}

}  // namespace

int ctx_attn_fma_rows(int rows_in_group) {
  const int r = (rows_in_group + kWarps - 1) / kWarps;
  return kWarps * (r <= 2 ? 2 : r <= 4 ? 4 : 8);
}

int launch_ctx_attn_fma(const CtxAttnArgs& a, cudaStream_t s) {
  if (a.rows <= 0) return ARTAB_OK;
  ARTAB_REQUIRE(a.n_ctx > 0 && a.n_splits >= 1, ARTAB_EINVAL, "context attention: empty context or no splits");
  ARTAB_REQUIRE(a.head_dim == 16 || a.head_dim == 32 || a.head_dim == 64, ARTAB_EINVAL,
                "context attention: head_dim %d not supported (16, 32, 64)", a.head_dim);
  return a.dtype == ARTAB_BF16 ? launch_t<__nv_bfloat16>(a, s) : launch_t<float>(a, s);
}

}  // namespace artab
