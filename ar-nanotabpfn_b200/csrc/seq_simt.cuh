// Whole-sequence decode on fp32 FMA, in fp32 and in bf16 mode, for the jobs it is the faster path of (seq.cu).
//
// A launch-per-layer decode step spends its time on dependent launches and on a few CTAs walking all
// the weights: at 64 streams of a 6-layer d_model 128 model a layer took 116 us for 20 us worth of
// FMAs on one CTA's share of the chip.  Here a cluster of C CTAs (C = heads, at most 8) owns `spc`
// streams = 2 * spc token rows and walks embedder -> layers -> head -> sampler for every target:
//
//   projections   column slices, one per CTA (W2: row slices, so the hidden tile never leaves its CTA)
//   attention     CTA c owns head c: context tiles of its head, private K/V rows of its head
//   exchanges     4 - 5 per layer, R x D floats each, as st.async stores that complete an mbarrier of
//                 the receiver: one one-way trip of the cluster network, no cluster barrier in the loop
//   weights       one contiguous byte stream per CTA in the order of use, and the context re-tiled so
//                 that a tile is contiguous: a producer thread keeps a ring of bulk copies in flight
//                 across phases, layers and targets
//
// Two uses of a landing area are always separated by another exchange in which every CTA takes part
// after it has read the area, so the areas need no "free" signal.  All waits are bounded.
//
// What bounds it: a CTA does a few thousand instructions per layer and warp, one dependent phase after
// the other, so every phase is written for few instructions and few shared-memory reads: a 16-byte
// shared-memory load costs the SM four cycles however many lanes read the same address, so products are
// register tiles (4 columns x R rows per thread, k split over the lanes and added up with shuffles), and
// the pieces used at several places are out of line (the first version inlined everything: 300 KB of
// code, 40 - 60 K cycles per layer, most of them instruction fetch and index arithmetic).
#pragma once
#include <type_traits>

#include "attn_tile.cuh"
#include "cluster.cuh"
#include "seq.cuh"

namespace artab {

namespace {

constexpr int kWarps = kSeqWarps;      // compute warps
constexpr int kT = kSeqThreads;        // compute threads
constexpr int kP = kSeqPitch;          // floats between the rows of every activation array

extern __shared__ __align__(1024) uint8_t g_seq_smem[];

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float gelu_erf(float v) { return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f)); }
__device__ __forceinline__ void sync_compute() { asm volatile("bar.sync 1, %0;" ::"n"(kT) : "memory"); }
// the same, and whether `v` is non-zero in any compute thread: one answer for all of them
__device__ __forceinline__ bool sync_compute_any(int v) {
  int any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 1, %2, q;\n\t"
      "selp.s32 %0, 1, 0, p;\n\t}"
      : "=r"(any)
      : "r"(v), "n"(kT)
      : "memory");
  return any != 0;
}

// mbarriers (full / empty per ring slot, one per exchange) and what a bounded wait needs, at the start of
// shared memory: a wait site hands over nothing but the barrier.
struct Bars {
  uint64_t full[kSeqMaxSlots], empty[kSeqMaxSlots];
  uint64_t x[6];
  long long limit;
  int abort_flag;
};
static_assert(sizeof(Bars) <= kSeqBarBytes, "barrier block");
__device__ __forceinline__ Bars* the_bars() { return reinterpret_cast<Bars*>(g_seq_smem); }
__device__ __forceinline__ uint8_t* slot_ptr(int slot) { return g_seq_smem + kSeqBarBytes + (size_t)slot * kSeqSlotBytes; }

__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity) {
  volatile Bars* b = the_bars();
  const long long t0 = clock64();
  for (;;) {
    if (b->abort_flag) return;  // first: after an abort no wait may block again
    if (clock64() - t0 > b->limit) {
      b->abort_flag = 1;
      return;
    }
    if (mbar_try(bar, parity)) return;
  }
}
// Bounded wait.  The data behind every barrier of this kernel (bulk copies, st.async of a peer) land in this
// CTA's own shared memory and are counted by the barrier itself.
__device__ __forceinline__ void wait_bar(uint32_t bar, uint32_t parity) {
  if (!mbar_test(bar, parity)) wait_slow(bar, parity);
}

// consumer side of the ring: every compute warp walks every slab in order.  The state is one word,
// slot | phase << 16, so that it stays in a register across the out-of-line pieces.
__device__ __forceinline__ const float4* ring_acquire(uint32_t ring) {
  wait_bar(smem_u32(&the_bars()->full[ring & 0xffffu]), ring >> 16);
  return reinterpret_cast<const float4*>(slot_ptr(ring & 0xffffu));
}
__device__ __forceinline__ void ring_release(uint32_t& ring, int n_slots) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&the_bars()->empty[ring & 0xffffu])) : "memory");
  ++ring;
  if ((ring & 0xffffu) == (uint32_t)n_slots) ring = (ring & 0x10000u) ^ 0x10000u;
}

// One matrix slice, out of line: act[R][K] . W[K][N] (act rows LDA floats apart), then what to do with it.
//
// W comes through the ring in units of 32 k x 16 columns (2 KB), k blocks outermost, in the lane order of the
// reads below: lane (s, g) holds k 4s .. 4s + 3 of columns 4g .. 4g + 3.  A warp takes one column tile and
// every kw-th k block: 4 + R 16-byte reads for 16 R FMAs per lane; the eight k slices of a warp are added
// with shuffles that halve the values each time, the kw warps of a column tile through shared memory.
enum ProjectMode : int { PROJ_SEND = 0, PROJ_SPLIT = 1, PROJ_GELU = 2, PROJ_STORE = 3 };
//   out, ld   row r, column n at out + r * ld + n (PROJ_SPLIT: column n % split of CTA n / split)
//   bar       PROJ_SEND / PROJ_SPLIT: the exchange's barrier
//   aux       PROJ_SPLIT: split.  PROJ_STORE: columns below aux are rounded to bf16 (queries of a bf16 cache)
//   bias      PROJ_GELU
template <int R, int LDA>
__device__ __noinline__ uint32_t project(uint32_t ring, int n_slots, const float* act, float* red, SeqMat m, ProjectMode mode,
                                         float* out, int ld, int C, uint32_t bar, int aux, const float* bias) {
  constexpr int V = R >= 2 ? R / 2 : 1;                  // values a lane ends up with
  constexpr int W = V < 4 ? V : 4;                       // of these neighbouring columns
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = lane >> 2, g = lane & 3;
  const int my_kw = (int)__fdividef((float)warp + 0.5f, (float)m.tiles), t = warp - my_kw * m.tiles;
  const bool active = my_kw < m.kw;
  const int total = m.tiles * m.octs, step = m.kw * m.tiles;
  int u = active ? my_kw * m.tiles + t : total;
  const float* x = act + my_kw * 32 + 4 * s;
  constexpr bool PACKED = R <= 8;                        // sixteen rows would need 128 accumulator registers
  float2 acc2[PACKED ? R * 4 : 1];
  float v[R * 4];
#pragma unroll
  for (int i = 0; i < R * 4; ++i) {
    v[i] = 0.f;
    if constexpr (PACKED) acc2[i] = make_float2(0.f, 0.f);
  }
#pragma unroll 1
  for (int u0 = 0; u0 < total; u0 += kSeqSlabUnits) {
    const float4* slab = ring_acquire(ring);
    const int end = min(u0 + kSeqSlabUnits, total);
#pragma unroll 1
    for (; u < end; u += step, x += 32 * m.kw) {
      const float4* wp = slab + (u - u0) * 128 + lane;
      float4 w[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) w[c] = wp[32 * c];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(x + r * LDA);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if constexpr (PACKED) {
            acc2[4 * r + c] = fma2(make_float2(a.x, a.y), make_float2(w[c].x, w[c].y), acc2[4 * r + c]);
            acc2[4 * r + c] = fma2(make_float2(a.z, a.w), make_float2(w[c].z, w[c].w), acc2[4 * r + c]);
          } else {
            v[4 * r + c] = fmaf(a.x, w[c].x, fmaf(a.y, w[c].y, fmaf(a.z, w[c].z, fmaf(a.w, w[c].w, v[4 * r + c]))));
          }
        }
      }
    }
    ring_release(ring, n_slots);
  }
  if constexpr (PACKED) {
#pragma unroll
    for (int i = 0; i < R * 4; ++i) v[i] = acc2[i].x + acc2[i].y;
  }
  if (active) {
    halve<4 * R, 16>(v);
    halve<2 * R, 8>(v);
    halve<R, 4>(v);
  }
  if (m.kw > 1) {
    float* mine = red + (warp * 32 + lane) * V;
    if (active && my_kw > 0) {
#pragma unroll
      for (int i = 0; i < V; i += W) {
        if constexpr (W == 4) *reinterpret_cast<float4*>(mine + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        else if constexpr (W == 2) *reinterpret_cast<float2*>(mine + i) = make_float2(v[i], v[i + 1]);
        else mine[i] = v[i];
      }
    }
    sync_compute();
    if (my_kw == 0) {
#pragma unroll 1
      for (int k = 1; k < m.kw; ++k) {
        const float* o = mine + k * m.tiles * 32 * V;
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] += o[i];
      }
    }
  }
  if (active && my_kw == 0) {
    // the halving left lane (s, g) with these rows and columns of the 16-column tile
    const int r0 = R >= 8 ? s * (R / 8) : R == 4 ? s >> 1 : R == 2 ? s >> 2 : 0;
    int n = 16 * t + 4 * g + (R >= 8 ? 0 : R == 4 ? 2 * (s & 1) : R == 2 ? (s & 3) : s >> 1);
    const bool mine = R > 1 || !(s & 1);
    if (mode == PROJ_GELU) {
#pragma unroll
      for (int c = 0; c < W; ++c) {
        const float b = bias[n + c];
#pragma unroll
        for (int i = c; i < V; i += W) v[i] = gelu_erf(v[i] + b);
      }
    }
    if (mode == PROJ_STORE && n < aux) {
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = __bfloat162float(__float2bfloat16_rn(v[i]));
    }
    if (mode >= PROJ_GELU) {
      if (mine) {
#pragma unroll
        for (int i = 0; i < V; ++i) out[(r0 + i / 4) * ld + n + (i & 3)] = v[i];
      }
    } else {
      int c0 = 0, c1 = C;
      if (mode == PROJ_SPLIT) {
        c0 = (int)__fdividef((float)n + 0.5f, (float)aux);
        c1 = c0 + 1;
        n -= c0 * aux;
      }
      if (mine) {
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
#pragma unroll
          for (int i = 0; i < V; i += W)
            st_async<W>(map_to_rank(smem_u32(out + (r0 + i / 4) * ld + n), c), v + i, map_to_rank(bar, c));
        }
      }
    }
  }
  if (mode >= PROJ_GELU) sync_compute();
  return ring;
}

// The C partial sums of this CTA's DS columns of the MLP output, [C][rows][DS], added up and sent to every CTA.
__device__ __noinline__ void sum_send(const float* part, int rows, int DS, float* out, uint32_t bar, int C) {
  const int n4 = DS >> 2;
  const float inv = 1.0f / (float)n4;
#pragma unroll 1
  for (int i = threadIdx.x; i < rows * n4; i += kT) {
    const int r = (int)(((float)i + 0.5f) * inv), n = 4 * (i - r * n4);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int c = 0; c < C; ++c) {
      const float4 t = *reinterpret_cast<const float4*>(part + (c * rows + r) * DS + n);
      v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
    }
    const uint32_t at = smem_u32(out + r * kP + n);
#pragma unroll 1
    for (int c = 0; c < C; ++c) st_async<4>(map_to_rank(at, c), v, map_to_rank(bar, c));
  }
}

// dst row r <- LayerNorm(res row r + bias + sum over c of src[c][r]), one warp per row, D = 64, 128 or 192.
// Rows of dst / res are ld floats apart, rows of the n_src source blocks kP.  `bar`: the exchange barrier that
// completes when the sources have arrived (0: none).
__device__ __noinline__ void layer_norm(float* dst, int dst_ld, const float* res, int res_ld, const float* src, int n_src,
                                        const float* bias, int rows, int D, const float* gamma, const float* beta,
                                        uint32_t bar, uint32_t parity) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_d = D == 64 ? 1.0f / 64 : D == 128 ? 1.0f / 128 : 1.0f / 192;
  float2 g[3], b[3], v[3];
  if (warp < rows) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (64 * i < D) {
        g[i] = reinterpret_cast<const float2*>(gamma + 64 * i)[lane];
        b[i] = reinterpret_cast<const float2*>(beta + 64 * i)[lane];
        v[i] = bias ? reinterpret_cast<const float2*>(bias + 64 * i)[lane] : make_float2(0.f, 0.f);
      }
  }
  if (bar && warp < rows) wait_bar(bar, parity);  // a polling warp takes issue slots: only those that will read
#pragma unroll 1
  for (int r = warp; r < rows; r += kWarps) {
    float2 x[3];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (64 * i < D) {
        float2 t = v[i];
        const float2* sp = reinterpret_cast<const float2*>(src + r * kP + 64 * i) + lane;
#pragma unroll 2
        for (int c = 0; c < n_src; ++c) {
          const float2 y = sp[c * rows * (kP / 2)];
          t.x += y.x;
          t.y += y.y;
        }
        const float2 y = reinterpret_cast<const float2*>(res + r * res_ld + 64 * i)[lane];
        x[i] = make_float2(t.x + y.x, t.y + y.y);
        sum += x[i].x + x[i].y;
      }
    const float mean = warp_sum(sum) * inv_d;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (64 * i < D) {
        x[i].x -= mean;
        x[i].y -= mean;
        ss = fmaf(x[i].x, x[i].x, fmaf(x[i].y, x[i].y, ss));
      }
    const float var = fmaf(warp_sum(ss), inv_d, 1e-5f);
    float rstd = rsqrtf(var);
    rstd *= fmaf(-0.5f * var * rstd, rstd, 1.5f);   // one Newton step: rsqrtf alone is good to 2^-22
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (64 * i < D)
        reinterpret_cast<float2*>(dst + r * dst_ld + 64 * i)[lane] =
            make_float2(fmaf(x[i].x * rstd, g[i].x, b[i].x), fmaf(x[i].y * rstd, g[i].y, b[i].y));
  }
  sync_compute();
}

// Diagnostic builds (-DARTAB_TIMELINE): the first compute thread of every CTA stamps clock64() at the phase
// boundaries of the last target: marks 16 * layer + {0 layer begins, 1 fold sent, 2 LayerNorm 1, 3 Q|K|V,
// 4 context keys, 5 private keys, 6 partial results merged, 7 attention rows received, 8 out-projection sent,
// 9 LayerNorm 2, 10 first MLP matrix, 11 second sent, 12 LayerNorm 3}.
#ifdef ARTAB_TIMELINE
__device__ long long g_seq_tl[256][16 * kSeqMaxLayers + 8];
#define SEQ_TL(id) do { if (tid == 0 && t == a.t1 - 1) g_seq_tl[blockIdx.x & 255][id] = clock64(); } while (0)
#else
#define SEQ_TL(id) do { } while (0)
#endif

// Void results are zeros, not what the memory held before.  Out of line and from the arguments alone: nothing of it is
// live while the kernel works.
__device__ __noinline__ void zero_results(const SeqArgs& a) {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int stream0 = (int)(blockIdx.x / a.C) * a.spc, n = a.t1 - a.t0;
  if (rank != 0) return;
#pragma unroll 1
  for (int i = threadIdx.x; i < min(a.spc, a.B - stream0) * n; i += kT + 32) {
    const size_t o = (size_t)(stream0 + i / n) * a.Nt + a.t0 + i % n;
    a.samples[o] = 0.f;
    if (a.logdens) a.logdens[o] = 0.f;
    if (a.comp) a.comp[o] = 0;
  }
}

template <typename CT, int DH, int R, bool SHARED>
__global__ void __launch_bounds__(kT + 32, 1) seq_simt_kernel(const __grid_constant__ SeqArgs a) {
  constexpr int S = R / 2;              // streams this variant holds (a.spc of them in use)
  constexpr int kParts = kWarps + kSeqBufferParts;
  const int D = a.D, C = a.C, L = a.L, K = a.n_comp, n_slots = a.n_slots;
  uint32_t crank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const int rank = (int)crank;
  const int stream0 = (int)(blockIdx.x / C) * a.spc;
  const int ns = min(a.spc, a.B - stream0);  // streams of this cluster
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int hc = a.hc, DS = a.DS, HS = a.HS, NB = a.NB;

  Bars* bars = the_bars();
  float* red = reinterpret_cast<float*>(g_seq_smem + a.off_red);  // partial sums of a product; attention scratch
  float* x_attn = reinterpret_cast<float*>(g_seq_smem + a.off_areas);  // exchange 0: attention output     [R][kP]
  float* x_wo = x_attn + R * kP;                         // exchange 1: out-projection       [R][kP]
  float* x_fold = x_wo + R * kP;                         // exchange 4: folded feature attention [R][kP]
  float* x_gather = x_fold + R * kP;                     // exchange 3: MLP output           [R][kP] (reduce + gather form)
  float* res = x_gather + (a.mlp_direct ? 0 : R * kP);   // residual stream                  [R][kP], the same in every CTA
  float* z = res + R * kP;                               // final LayerNorm, target rows     [S][kP]
  float* hid = z + S * kP;                               // hidden slice of the MLP          [R][kP]
  float* qkv = hid + R * kP;                             // q | k | v of this CTA's heads    [R][kP]
  float* x_mlp = qkv + R * kP;                           // exchange 2: MLP partial sums     [C][R][kP] or [C][R][DS]
  float* x_head = x_mlp + (a.mlp_direct ? C * R * kP : C * R * DS);  // exchange 5: head partial sums [C][S][NB]
  float* head_c = x_head + C * S * NB;                   // per component: bb x 3, mean / std / weight bias [6][32]
  float* xm = head_c + 6 * 32;                           // feature means: previous target [S], this one [S]
  float* ys = xm + 2 * S;                                // last sampled y [S]

  if (tid == 0) {
#pragma unroll 1
    for (int i = 0; i < n_slots; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars->full[i])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&bars->empty[i])), "r"(kWarps) : "memory");
    }
#pragma unroll 1
    for (int i = 0; i < 6; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars->x[i])) : "memory");
    bars->abort_flag = 0;
    bars->limit = a.wait_cycles;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // peers may write here only once the barriers exist
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  dep_wait();
  dep_trigger();
  volatile int* abort_flag = &bars->abort_flag;

  int slot = 0, filled = 0;   // producer thread: next ring slot, slots ever filled
  uint32_t phase = 1;         // empty barriers: the first round passes at once
  if (warp == kWarps) {
    // ------------------------------- producer -------------------------------
    if (lane == 0) {
      auto put = [&](const void* src, uint32_t bytes) {
        if (*abort_flag) return;
        wait_bar(smem_u32(&bars->empty[slot]), phase);
        if (*abort_flag) return;
        const uint32_t full = smem_u32(&bars->full[slot]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(slot_ptr(slot))),
                     "l"(src), "r"(bytes), "r"(full)
                     : "memory");
        filled |= 1 << slot;
        if (++slot == n_slots) {
          slot = 0;
          phase ^= 1;
        }
      };
      constexpr uint32_t kTile = 64 * DH * 4;   // context tile: 32 K rows and 32 V rows
      // One loop over the matrices of a target in the order the compute threads use them: per layer fold,
      // Q|K|V, [context], out-projection, W1, W2, then the two matrices of the head.
#pragma unroll 1
      for (int t = a.t0; t < a.t1 && !*abort_flag; ++t) {
        const uint8_t* w = a.weights + (size_t)rank * a.rank_bytes;
#pragma unroll 1
        for (int l = 0; l <= L; ++l) {
#pragma unroll 1
          for (int kind = 0; kind < (l == L ? 2 : 5); ++kind) {
            const int mi = l == L ? (kind == 0 ? SEQ_W1 : SEQ_WB) : kind == 0 ? SEQ_DS : kind == 1 ? SEQ_QKV : kind == 2 ? SEQ_DS : kind == 3 ? SEQ_W1 : SEQ_W2;
            if (l < L && kind == 2) {
              const int n_grp = SHARED ? 1 : ns;
#pragma unroll 1
              for (int hh = 0; hh < hc; ++hh) {
#pragma unroll 1
                for (int s = 0; s < n_grp; ++s) {
                  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.ctx) +
                                       (((size_t)l * a.G + (SHARED ? 0 : stream0 + s)) * a.H + rank * hc + hh) * a.n_ctx_tiles * kTile;
#pragma unroll 1
                  for (int j = 0; j < a.n_ctx_tiles; j += a.tiles_per_slab) {
                    const uint32_t bytes = (uint32_t)min(a.tiles_per_slab, a.n_ctx_tiles - j) * kTile;
                    put(src, bytes);
                    src += bytes;
                  }
                }
              }
            }
            const int units = a.mat[mi].tiles * a.mat[mi].octs;
#pragma unroll 1
            for (int u = 0; u < units; u += kSeqSlabUnits) {
              const uint32_t bytes = (uint32_t)min(kSeqSlabUnits, units - u) * 2048u;
              put(w, bytes);
              w += bytes;
            }
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------- compute --------------------------------
    uint32_t ring = 0;
    uint32_t xphase = 0;  // one bit per exchange
    const uint32_t xbar0 = smem_u32(&bars->x[0]);
    auto expect = [&](int x, int floats) {  // one thread announces what this CTA will receive
      if (tid == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(xbar0 + 8 * x), "r"(floats * 4) : "memory");
    };
    auto xparity = [&](int x) {  // parity of this use; the next one has the other
      const uint32_t p = (xphase >> x) & 1;
      xphase ^= 1u << x;
      return p;
    };

    // LayerNorm vectors and biases of this rank: in shared memory when the plan found room for them
    const float* vec = reinterpret_cast<const float*>(a.weights + (size_t)rank * a.rank_bytes + a.vec_off);
    if (a.vec_smem) {
      const float4* src = reinterpret_cast<const float4*>(vec);
      float4* dst = reinterpret_cast<float4*>(g_seq_smem + a.vec_smem);
      const int n = (L * (7 * D + HS) + 2 * D + HS) / 4;
#pragma unroll 1
      for (int i = tid; i < n; i += kT) dst[i] = __ldg(src + i);
      vec = reinterpret_cast<const float*>(dst);
    }
    // constants of the head, feature means of targets t0 - 1 and t0, the last sampled value
    if (warp == 0) {
      const int k = lane < K ? lane : 0;
#pragma unroll
      for (int i = 0; i < 3; ++i) head_c[32 * i + lane] = __ldg(a.bb + 3 * k + i);
      head_c[96 + lane] = __ldg(a.mean_bias + k);
      head_c[128 + lane] = __ldg(a.std_bias + k);
      head_c[160 + lane] = __ldg(a.weight_bias + k);
      if (lane < S) ys[lane] = a.t0 > 0 && lane < ns ? a.samples[(size_t)(stream0 + lane) * a.Nt + a.t0 - 1] : 0.f;
    }
#pragma unroll 1
    for (int i = warp; i < 2 * S; i += kWarps) {
      const int s = i >> 1, t = a.t0 - 1 + (i & 1);
      float sum = 0.f;
      if (t >= 0 && s < ns) {
        const float* xr = a.xt + (size_t)(stream0 + s) * a.xt_stride + (size_t)t * a.F;
#pragma unroll 1
        for (int f = lane; f < a.F; f += 32) sum += __ldg(xr + f);
      }
      sum = warp_sum(sum) / (float)a.F;
      if (lane == 0) xm[(i & 1) * S + s] = sum;
    }
    sync_compute();

    bool dead = false;
#pragma unroll 1
    for (int t = a.t0; t < a.t1; ++t) {
      const int len = t;               // private keys visible in this step (the buffer token's own among them)
      // ---- embedder: row 2s buffer (x_{t-1}, y_{t-1}), row 2s + 1 target x_t; one warp per row ----
#pragma unroll 1
      for (int r = warp; r < R; r += kWarps) {
        const int s = r >> 1;
        const bool buf = !(r & 1);
        const float xmean = buf ? xm[s] : xm[S + s], y = ys[s];
        const float* mk = a.marker + (buf ? ARTAB_MARK_BUFFER : ARTAB_MARK_TARGET) * D;
        const float* ar = a.ar_tokens + (t % a.S_ar) * D;
#pragma unroll 1
        for (int d = lane; d < D; d += 32) {
          float e = fmaf(xmean, __ldg(a.wx + d), __ldg(a.bx + d));
          if (buf) e += fmaf(y, __ldg(a.wy + d), __ldg(a.by + d));
          e += __ldg(mk + d);
          if (buf) e += __ldg(ar + d);
          res[r * kP + d] = buf && t == 0 ? 0.f : e;
        }
      }
      // what the end of the step needs from memory: the next target's features, the random numbers
      float nx = 0.f, ex = 1.f, no = 0.f;
      if (warp < ns) {
        const size_t b = stream0 + warp;
        if (t + 1 < a.Nt) {
          const float* xr = a.xt + b * a.xt_stride + (size_t)(t + 1) * a.F;
#pragma unroll 1
          for (int f = lane; f < a.F; f += 32) nx += __ldg(xr + f);
        }
        if (lane < K) ex = __ldg(a.expo + ((size_t)t * a.B + b) * K + lane);
        no = __ldg(a.normal + (size_t)t * a.B + b);
      }
      sync_compute();

#pragma unroll 1
      for (int l = 0; l < L; ++l) {
        // per layer: LayerNorm 1 gamma, beta | LayerNorm 2 gamma, beta | b2 | LayerNorm 3 gamma, beta | b1 slice
        const float* w = vec + l * (7 * D + HS);
        SEQ_TL(16 * l);
        // ---- feature attention over one token (one folded matrix) + LayerNorm 1 ----
        expect(4, R * D);
        ring = project<R, kP>(ring, n_slots, res, red, a.mat[SEQ_DS], PROJ_SEND, x_fold + rank * DS, kP, C,
                              xbar0 + 8 * 4, 0, nullptr);
        SEQ_TL(16 * l + 1);
        layer_norm(res, kP, res, kP, x_fold, 1, nullptr, R, D, w, w + D, xbar0 + 8 * 4, xparity(4));
        SEQ_TL(16 * l + 2);
        // ---- Q | K | V of this CTA's heads; K / V rows of the buffer tokens go to their cache slots ----
        ring = project<R, kP>(ring, n_slots, res, red,
                              a.mat[SEQ_QKV], PROJ_STORE, qkv, kP, C, 0,
                              sizeof(CT) == 2 ? hc * DH : 0, nullptr);
        CT* const kv_layer = reinterpret_cast<CT*>(a.kv_buf) + ((size_t)l * a.B + stream0) * a.H * a.max_buf * 2 * DH;
        if (t > 0) {
          constexpr int PH = 2 * DH / 4;   // 4-element pieces of a K row and a V row
#pragma unroll 1
          for (int i = tid; i < ns * hc * PH; i += kT) {
            const int sh = i / PH, e = 4 * (i - sh * PH);   // e: element of the K row, then of the V row
            int s = sh, hh = 0;
            if (hc > 1) {
              s = sh / hc;
              hh = sh - s * hc;
            }
            const float4 v = *reinterpret_cast<const float4*>(qkv + 2 * s * kP + ((e >= DH ? 2 : 1) * hc + hh) * DH + (e & (DH - 1)));
            CT* o = kv_layer + ((size_t)(s * a.H + rank * hc + hh) * a.max_buf + (t - 1)) * 2 * DH + e;
            if constexpr (sizeof(CT) == 4) {
              *reinterpret_cast<float4*>(o) = v;
            } else {
              const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
              *reinterpret_cast<uint2*>(o) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            }
          }
          sync_compute();
        }
        SEQ_TL(16 * l + 3);
        // ---- attention of this CTA's heads ----
        expect(0, R * D);
#pragma unroll 1
        for (int hh = 0; hh < hc; ++hh) {
          const float* q = qkv + hh * DH;
          float* part = red;                             // [kParts][R][DH]
          float* ml = part + kParts * R * DH;            // [kParts][R][2]
          float* pw = ml + kParts * R * 2 + warp * 32 * R;  // softmax numerators of a tile, [32][rows]
          const float sc = a.scale_log2e;
          int turn = 0;
          if constexpr (SHARED) {
            TileState<DH, R, kP> st;
            st.init();
#pragma unroll 1
            for (int i = 0; i < a.n_ctx_tiles; i += a.tiles_per_slab) {
              const float4* slab = ring_acquire(ring) + lane;
              if (turn == warp) {
                const int nt = min(a.tiles_per_slab, a.n_ctx_tiles - i);
#pragma unroll 1
                for (int j = 0; j < nt; ++j, slab += 16 * DH)
                  st.tile(q, pw, a.n_ctx - (i + j) * 32, sc, [&](int jj, int kk) { return slab[(4 * jj + kk) * 32]; },
                          [&](int ii) { return slab[8 * DH + 32 * ii]; });
              }
              ring_release(ring, n_slots);
              if (++turn == kWarps) turn = 0;
            }
            st.flush(part + warp * R * DH, ml + warp * R * 2);
          } else {
#pragma unroll 1
            for (int s = 0; s < ns; ++s) {
              TileState<DH, 2, kP> st;
              st.init();
              turn = 0;  // every stream spreads over the warps in the same way
#pragma unroll 1
              for (int i = 0; i < a.n_ctx_tiles; i += a.tiles_per_slab) {
                const float4* slab = ring_acquire(ring) + lane;
                if (turn == warp) {
                  const int nt = min(a.tiles_per_slab, a.n_ctx_tiles - i);
#pragma unroll 1
                  for (int j = 0; j < nt; ++j, slab += 16 * DH)
                    st.tile(q + 2 * s * kP, pw, a.n_ctx - (i + j) * 32, sc, [&](int jj, int kk) { return slab[(4 * jj + kk) * 32]; },
                            [&](int ii) { return slab[8 * DH + 32 * ii]; });
                }
                ring_release(ring, n_slots);
                if (++turn == kWarps) turn = 0;
              }
              st.flush(part + (warp * R + 2 * s) * DH, ml + (warp * R + 2 * s) * 2);
            }
          }
          SEQ_TL(16 * l + 4);
          // Private keys: (stream, part) items over the warps, those with the fewest context tiles first.  A part
          // is every nb-th tile of the stream, its result a partial of its own: what a stream gets does not
          // depend on where in the cluster it sits.
          const int nb = min(kSeqBufferParts, (len + 31) >> 5);
#pragma unroll 1
          for (int u = kWarps - 1 - warp; u < S * nb; u += kWarps) {
            const int s = u & (S - 1), jb = u / S;
            if (s >= ns) continue;
            const CT* kv = kv_layer + (size_t)(s * a.H + rank * hc + hh) * a.max_buf * 2 * DH;
            TileState<DH, 2, kP> st;
            st.init();
#pragma unroll 1
            for (int k0 = 32 * jb; k0 < len; k0 += 32 * nb) {
              // every load of the tile is issued before the first is used: one memory round trip
              constexpr int NQ = TileState<DH, 2, kP>::NQ, NI = TileState<DH, 2, kP>::NI;
              float4 kr[NQ * 4], vr[NI];
              const int last = len - 1;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int j = 0; j < NQ; ++j)
                  kr[4 * j + kk] = load4(kv + (size_t)min(k0 + 4 * (lane & 7) + kk, last) * 2 * DH + 4 * (lane >> 3) + 16 * j);
#pragma unroll
              for (int i = 0; i < NI; ++i)
                vr[i] = load4(kv + (size_t)min(k0 + lane / (DH / 4) * NI + i, last) * 2 * DH + DH + 4 * (lane & (DH / 4 - 1)));
              st.tile(q + 2 * s * kP, pw, len - k0, sc, [&](int jj, int kk) { return kr[4 * jj + kk]; }, [&](int ii) { return vr[ii]; });
            }
            st.flush(part + ((kWarps + jb) * R + 2 * s) * DH, ml + ((kWarps + jb) * R + 2 * s) * 2);
          }
          SEQ_TL(16 * l + 5);
          sync_compute();
          // merge the partial softmaxes: four lanes per (row, 4 dims), each every fourth part
          const int parts = kWarps + nb;
#pragma unroll 1
          for (int i = tid; i < R * DH; i += kT) {
            const int w0 = i & 3, r = (i >> 2) / (DH / 4), d = 4 * ((i >> 2) & (DH / 4 - 1));
            float2 f[kParts / 4];
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < kParts / 4; ++j) {
              const int w = w0 + 4 * j;
              f[j] = w < parts ? *reinterpret_cast<const float2*>(ml + (w * R + r) * 2) : make_float2(-INFINITY, 0.f);
              top = fmaxf(top, f[j].x);
            }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            float o[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < kParts / 4; ++j) {
              if (f[j].x == -INFINITY) continue;   // no keys in this part
              const float e = exp2f(f[j].x - top);
              const float4 p = *reinterpret_cast<const float4*>(part + ((w0 + 4 * j) * R + r) * DH + d);
              o[0] = fmaf(e, p.x, o[0]);
              o[1] = fmaf(e, p.y, o[1]);
              o[2] = fmaf(e, p.z, o[2]);
              o[3] = fmaf(e, p.w, o[3]);
              o[4] = fmaf(e, f[j].y, o[4]);
            }
#pragma unroll
            for (int e = 0; e < 5; ++e) {
              o[e] += __shfl_xor_sync(0xffffffffu, o[e], 1);
              o[e] += __shfl_xor_sync(0xffffffffu, o[e], 2);
            }
            const float inv = 1.0f / o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] *= inv;
            const uint32_t at = smem_u32(x_attn + r * kP + (rank * hc + hh) * DH + d);
#pragma unroll 1
            for (int c = w0; c < C; c += 4) st_async<4>(map_to_rank(at, c), o, map_to_rank(xbar0, c));
          }
          if (hh + 1 < hc) sync_compute();  // the scratch is reused by the next head
        }
        SEQ_TL(16 * l + 6);
        {
          const uint32_t par = xparity(0);
          if (warp == 0) wait_bar(xbar0, par);  // one warp polls, the others sleep at the barrier
        }
        // Also: the scratch has been read, the projections may overwrite it.  And where a job ends whose waits gave
        // up: until here every exchange barrier has been armed at most once since, so none is armed twice in a phase,
        // and the peers, which get nothing more from here, give up in turn.
        dead = sync_compute_any(*abort_flag);
        if (dead) break;
        // ---- out-projection, MLP; the last layer has results for the target rows only ----
        auto post = [&](auto rows_const, auto ld_const, int off) {
          constexpr int RR = decltype(rows_const)::value, LD = decltype(ld_const)::value;
          SEQ_TL(16 * l + 7);
          float* rs = res + off;
          expect(1, RR * D);
          ring = project<RR, LD>(ring, n_slots, x_attn + off, red, a.mat[SEQ_DS], PROJ_SEND, x_wo + rank * DS, kP,
                                 C, xbar0 + 8, 0, nullptr);
          SEQ_TL(16 * l + 8);
          layer_norm(rs, LD, rs, LD, x_wo, 1, nullptr, RR, D, w + 2 * D, w + 3 * D, xbar0 + 8, xparity(1));
          SEQ_TL(16 * l + 9);
          ring = project<RR, LD>(ring, n_slots, rs, red, a.mat[SEQ_W1], PROJ_GELU, hid, kP, C, 0, 0, w + 7 * D);
          SEQ_TL(16 * l + 10);
          if (a.mlp_direct) {
            expect(2, C * RR * D);
            ring = project<RR, kP>(ring, n_slots, hid, red, a.mat[SEQ_W2], PROJ_SEND, x_mlp + rank * RR * kP,
                                   kP, C, xbar0 + 16, 0, nullptr);
            SEQ_TL(16 * l + 11);
            layer_norm(rs, LD, rs, LD, x_mlp, C, w + 4 * D, RR, D, w + 5 * D, w + 6 * D, xbar0 + 16, xparity(2));
          } else {
            expect(2, RR * D);
            expect(3, RR * D);
            ring = project<RR, kP>(ring, n_slots, hid, red,
                                   a.mat[SEQ_W2], PROJ_SPLIT, x_mlp + rank * RR * DS,
                                   DS, C, xbar0 + 16, DS, nullptr);
            SEQ_TL(16 * l + 11);
            wait_bar(xbar0 + 16, xparity(2));
            sum_send(x_mlp, RR, DS, x_gather + rank * DS, xbar0 + 24, C);
            layer_norm(rs, LD, rs, LD, x_gather, 1, w + 4 * D, RR, D, w + 5 * D, w + 6 * D, xbar0 + 24, xparity(3));
          }
        };
        if (l + 1 < L)
          post(std::integral_constant<int, R>{}, std::integral_constant<int, kP>{}, 0);
        else
          post(std::integral_constant<int, S>{}, std::integral_constant<int, 2 * kP>{}, kP);
        SEQ_TL(16 * l + 12);
      }

      if (dead) break;
      SEQ_TL(16 * L);
      // ---- mixture head on the target rows: every CTA ends up with all raw outputs ----
      layer_norm(z, kP, res + kP, 2 * kP, nullptr, 0, nullptr, S, D, vec + L * (7 * D + HS), vec + L * (7 * D + HS) + D, 0, 0);
      ring = project<S, kP>(ring, n_slots, z, red, a.mat[SEQ_W1], PROJ_GELU, hid, kP, C, 0, 0, vec + L * (7 * D + HS) + 2 * D);
      expect(5, C * S * NB);
      ring = project<S, kP>(ring, n_slots, hid, red, a.mat[SEQ_WB], PROJ_SEND, x_head + rank * S * NB, NB, C,
                            xbar0 + 8 * 5, 0, nullptr);
      SEQ_TL(16 * L + 1);
      const uint32_t head_parity = xparity(5);
      if (warp < ns) {
        wait_bar(xbar0 + 8 * 5, head_parity);
        SEQ_TL(16 * L + 2);
        // every CTA of the cluster samples the same value; rank 0 writes it
        const int s = warp;
        float raw[3] = {head_c[lane], head_c[32 + lane], head_c[64 + lane]};
        float mean = 0.f, stdv = 1.f, lw = -INFINITY;
        if (lane < K) {
#pragma unroll 1
          for (int c = 0; c < C; ++c)
#pragma unroll
            for (int i = 0; i < 3; ++i) raw[i] += x_head[(c * S + s) * NB + 3 * lane + i];
          mean = raw[0] + head_c[96 + lane];
          const float sr = raw[1] + head_c[128 + lane];
          const float sp = sr > 20.f ? sr : log1pf(expf(sr));  // F.softplus, beta 1, threshold 20
          stdv = fminf(sp, 2.0f) + 1e-3f;
          lw = raw[2] + head_c[160 + lane];
        }
        const float mx = warp_max(lw);
        const float se = warp_sum(lane < K ? expf(lw - mx) : 0.f);
        const float logw = lw - mx - logf(se);
        // torch.multinomial(w, 1) == argmax_k(w_k / Exp(1)_k); first maximum wins
        float bv = lane < K ? expf(logw) / ex : -1.f;
        int best = lane;
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
          const int oi = __shfl_xor_sync(0xffffffffu, best, o);
          if (ov > bv || (ov == bv && oi < best)) {
            bv = ov;
            best = oi;
          }
        }
        const float y = __shfl_sync(0xffffffffu, mean, best) + __shfl_sync(0xffffffffu, stdv, best) * no;
        float lp = -INFINITY;
        if (lane < K) {
          const float zz = (y - mean) / stdv;
          lp = -0.5f * (1.8378770664093453f + 2.0f * logf(stdv) + zz * zz) + logw;
        }
        const float m2 = warp_max(lp);
        const float s2 = warp_sum(lane < K ? expf(lp - m2) : 0.f);
        nx = warp_sum(nx) / (float)a.F;
        if (lane == 0) {
          ys[s] = y;
          xm[s] = xm[S + s];
          xm[S + s] = nx;
          if (rank == 0 && !*abort_flag) {
            const size_t o = (size_t)(stream0 + s) * a.Nt + t;
            a.samples[o] = y;
            if (a.comp) a.comp[o] = best;
            if (a.logdens) a.logdens[o] = m2 + logf(s2);
          }
        }
      }
      sync_compute();
      SEQ_TL(16 * L + 3);
    }
  }

  // Nobody leaves while another CTA could still write here.  Without an abort every store has been waited for; after
  // one the peers have issued their last when the barrier opens, and some may be in flight.
  __syncthreads();
  if (bars->abort_flag && warp == kWarps && lane == 0) {   // the copies in flight land first, too
#pragma unroll 1
    for (int i = 0; i < n_slots; ++i) {
      if (!((filled >> i) & 1)) continue;
      const uint32_t par = i < slot ? phase ^ 1 : phase;   // phase in which slot i was last filled
      const long long t0 = clock64();
      while (!mbar_try(smem_u32(&bars->full[i]), par) && clock64() - t0 < kDefaultWaitCycles) {
      }
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (bars->abort_flag) {
    if (tid == 0 && a.status) atomicExch(a.status, 4);
    zero_results(a);
    const long long t0 = clock64();
    while (clock64() - t0 < 100000) {
    }
  }
}

template <typename CT, int DH, int R, bool SHARED>
SmemConfig& smem_config() {
  static SmemConfig c;
  return c;
}

template <typename CT, int DH, int R, bool SHARED>
int launch_seq_variant(const SeqArgs& a, const SeqPlan& p, cudaStream_t s) {
  cudaError_t e = smem_config<CT, DH, R, SHARED>().ensure(seq_simt_kernel<CT, DH, R, SHARED>, p.smem);
  if (e == cudaSuccess)
    e = launch_dependent_cluster(seq_simt_kernel<CT, DH, R, SHARED>, dim3(p.grid), dim3(kT + 32), p.smem, s, (unsigned)p.C, a);
  ARTAB_REQUIRE(e == cudaSuccess, ARTAB_ELAUNCH, "seq_simt_kernel: launch refused: %s", cudaGetErrorString(e));
  return ARTAB_OK;
}

template <typename CT, int DH>
int launch_seq_dh(const SeqArgs& a, const SeqPlan& p, cudaStream_t s) {
  if (a.G == 1) {
    switch (p.rows) {
      case 2: return launch_seq_variant<CT, DH, 2, true>(a, p, s);
      case 4: return launch_seq_variant<CT, DH, 4, true>(a, p, s);
      case 8: return launch_seq_variant<CT, DH, 8, true>(a, p, s);
      default: return launch_seq_variant<CT, DH, 16, true>(a, p, s);
    }
  }
  switch (p.rows) {
    case 2: return launch_seq_variant<CT, DH, 2, false>(a, p, s);
    case 4: return launch_seq_variant<CT, DH, 4, false>(a, p, s);
    case 8: return launch_seq_variant<CT, DH, 8, false>(a, p, s);
    default: return launch_seq_variant<CT, DH, 16, false>(a, p, s);
  }
}

// clusters of C CTAs that fit the GPU at once (every variant takes a whole SM per CTA)
template <typename CT>
int seq_max_clusters(int C, size_t smem) {
  if (smem_config<CT, 32, 8, true>().ensure(seq_simt_kernel<CT, 32, 8, true>, smem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kT + 32);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, seq_simt_kernel<CT, 32, 8, true>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace
}  // namespace artab
