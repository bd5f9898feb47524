// fp32 attention of a few query rows over tiles of 32 keys by one warp: what the whole-sequence decode and the
// context attention of the fp32 mode share.
#pragma once
#include "common.cuh"

namespace artab {

// One halving step of a sum over lanes: the lane pair that differs in bit MASK splits its V values, each
// keeps the half its bit names and receives the other lane's share of it.  V == 1: plain sum.
template <int V, int MASK>
__device__ __forceinline__ void halve(float* v) {
  const bool up = (threadIdx.x & MASK) != 0;
  if constexpr (V > 1) {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      const float give = up ? v[i] : v[i + V / 2];
      const float keep = up ? v[i + V / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, MASK);
    }
  } else {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], MASK);
  }
}

// ---- attention: tiles of 32 keys ----
// Scores: lane (ds, kg) multiplies dims 4 ds + 16 j .. + 3 of keys 4 kg .. 4 kg + 3 with four query rows at a
// time; halving over ds leaves it row ds and its four keys.  P.V: lane (ks, dg) owns dims 4 dg .. 4 dg + 3 and
// keys ks * NI .. ks * NI + NI - 1.
template <int DH, int NR, int QP>   // QP: floats between query rows
struct TileState {
  static constexpr int NQ = DH / 16;       // 4-dim blocks of a key per lane
  static constexpr int KSL = 128 / DH;     // key slices of P.V
  static constexpr int NI = 32 / KSL;      // keys of a slice
  static constexpr int G = NR < 4 ? NR : 4, NG = NR / G;  // query rows are taken G at a time
  static constexpr int NKL = G == 4 ? 4 : 2;              // keys a lane is left with
  float m[NG], l[NG], acc[NR][4];          // reference (log2 units) and sum share of the lane's row of every group

  __device__ __forceinline__ void init() {
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      m[g] = -INFINITY;
      l[g] = 0.f;
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[r][e] = 0.f;
  }

  // load_k(j, kk) -> the lane's dims of its key kk; load_v(i) -> the lane's dims of key i of its slice
  template <class LoadK, class LoadV>
  __device__ __forceinline__ void tile(const float* q, float* pw, int n_valid, float sc, LoadK load_k, LoadV load_v) {
    const int lane = threadIdx.x & 31, ds = lane >> 3, kg = lane & 7;
    const int row = G == 4 ? ds : ds >> 1;
    const int key0 = 4 * kg + (G == 4 ? 0 : 2 * (ds & 1));
    __syncwarp();  // the previous tile's numerators have been read
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      float s[G * 4];
#pragma unroll
      for (int i = 0; i < G * 4; ++i) s[i] = 0.f;
#pragma unroll
      for (int j = 0; j < NQ; ++j) {
        float4 k[4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) k[kk] = load_k(j, kk);
#pragma unroll
        for (int r = 0; r < G; ++r) {
          const float4 x = *reinterpret_cast<const float4*>(q + (g * G + r) * QP + 4 * ds + 16 * j);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            s[4 * r + kk] = fmaf(x.x, k[kk].x, fmaf(x.y, k[kk].y, fmaf(x.z, k[kk].z, fmaf(x.w, k[kk].w, s[4 * r + kk]))));
        }
      }
      halve<G * 4, 16>(s);
      halve<G * 2, 8>(s);
      float mx = -INFINITY;
#pragma unroll
      for (int kk = 0; kk < NKL; ++kk) {
        s[kk] = key0 + kk < n_valid ? s[kk] * sc : -INFINITY;
        mx = fmaxf(mx, s[kk]);
      }
      if (__any_sync(0xffffffffu, mx > m[g] + 8.0f)) {  // some score passes its row's reference by 2^8: raise it
#pragma unroll
        for (int o = 1; o < (G == 4 ? 8 : 16); o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mn = fmaxf(m[g], mx);
        const float alpha = m[g] == mn ? 1.0f : exp2f(m[g] - mn);
        l[g] *= alpha;
        m[g] = mn;
#pragma unroll
        for (int r = 0; r < G; ++r) {
          const float ar = __shfl_sync(0xffffffffu, alpha, (G == 4 ? 8 : 16) * r);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[g * G + r][e] *= ar;
        }
      }
      const float ref = m[g] == -INFINITY ? 0.f : m[g];   // no key of this row yet: exp2(-inf - 0) = 0
#pragma unroll
      for (int kk = 0; kk < NKL; ++kk) {
        s[kk] = exp2f(s[kk] - ref);
        l[g] += s[kk];
      }
      float* o = pw + (g * G + row) * 32 + key0;
      if constexpr (NKL == 4) *reinterpret_cast<float4*>(o) = make_float4(s[0], s[1], s[2], s[3]);
      else *reinterpret_cast<float2*>(o) = make_float2(s[0], s[1]);
    }
    __syncwarp();
    const float* pp = pw + lane / (DH / 4) * NI;
#pragma unroll
    for (int i = 0; i < NI; i += 4) {
      float4 x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = load_v(i + e);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const float4 p = *reinterpret_cast<const float4*>(pp + r * 32 + i);
        acc[r][0] = fmaf(p.x, x[0].x, fmaf(p.y, x[1].x, fmaf(p.z, x[2].x, fmaf(p.w, x[3].x, acc[r][0]))));
        acc[r][1] = fmaf(p.x, x[0].y, fmaf(p.y, x[1].y, fmaf(p.z, x[2].y, fmaf(p.w, x[3].y, acc[r][1]))));
        acc[r][2] = fmaf(p.x, x[0].z, fmaf(p.y, x[1].z, fmaf(p.z, x[2].z, fmaf(p.w, x[3].z, acc[r][2]))));
        acc[r][3] = fmaf(p.x, x[0].w, fmaf(p.y, x[1].w, fmaf(p.z, x[2].w, fmaf(p.w, x[3].w, acc[r][3]))));
      }
    }
  }

  // partial result of this warp: row r at part + r * DH, {reference, sum} at ml + 2 r
  __device__ __forceinline__ void flush(float* part, float* ml) {
    const int lane = threadIdx.x & 31, dg = lane & (DH / 4 - 1);
    constexpr int NS = DH == 16 ? 3 : DH == 32 ? 2 : 1;   // halving steps over the key slices
    constexpr int V = NR * 4 >> NS, W = V < 4 ? V : 4;
    float* v = &acc[0][0];
    halve<NR * 4, 16>(v);
    if constexpr (NS > 1) halve<NR * 2, 8>(v);
    if constexpr (NS > 2) halve<NR, 4>(v);
    const int at = (lane >> (5 - NS)) * V;                // first (row, dim) index this lane is left with
#pragma unroll
    for (int i = 0; i < V; i += W) {
      float* o = part + ((at + i) >> 2) * DH + 4 * dg + ((at + i) & 3);
      if constexpr (W == 4) *reinterpret_cast<float4*>(o) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      else if constexpr (W == 2) *reinterpret_cast<float2*>(o) = make_float2(v[i], v[i + 1]);
      else o[0] = v[i];
    }
    constexpr int LPR = G == 4 ? 8 : 16;                  // lanes that hold shares of one row
#pragma unroll
    for (int g = 0; g < NG; ++g) {
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) l[g] += __shfl_xor_sync(0xffffffffu, l[g], o);
      if ((lane & (LPR - 1)) == 0) *reinterpret_cast<float2*>(ml + 2 * (g * G + lane / LPR)) = make_float2(m[g], l[g]);
    }
  }
};

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                     __uint_as_float(w.y & 0xffff0000u));
}

}  // namespace artab
