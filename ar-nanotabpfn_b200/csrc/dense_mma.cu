// Per-token layer chain in bf16 mode for few rows (a decode step, a short prefill): a cluster of four CTAs owns 32 rows.
//
// The tcgen05 chain takes 128 rows per CTA (pair), so a decode step of 512 streams (1024 rows) kept 16 of 148 SMs
// busy and its 30 us were the serial walk of one CTA through all matrices.  Here 32 such clusters fill the chip:
// every product is split by output columns over the four CTAs, each of which reads a quarter of the weights
// (0.24 MB per layer at d_model 192).  32 x 48 x 192 per CTA is far below a tcgen05 tile (M = 128, and 100 cycles
// per instruction whatever N), so the products are warp-level mma.m16n8k16: activations split hi + lo in shared
// memory, weights straight from L2 into registers in fragment order (_pack.py), fetched before the wait that
// precedes their use.  Full rows are put together through distributed shared memory: 32 x D floats after the
// out-projection, the MLP (reduce, then gather) and the folded feature attention, as st.async stores counted by an
// mbarrier of the receiver; each barrier completes once per launch.
//
// What bounds it: a chain of about twelve short phases; a product phase is bounded by the shared-memory reads of the
// activation operand (each warp reads all 32 rows for its 16 columns).  512 streams x 128 targets on 1024 context rows,
// 6 layers, d_model 192: 44.8 ms per sampling job with the tcgen05 chain, 32.4 ms with this one (40 K cycles from the
// end of the wait to the last store).  One rolled loop for all products, so that their instructions are fetched once,
// was slower (37.1 ms).
#include "cluster.cuh"
#include "dense.cuh"
#include "head.cuh"
#include "kv_scatter.cuh"

namespace artab {

namespace {

constexpr int kC = 4, kRows = 32, kWarps = 12, kThreads = kWarps * 32;

struct Bars {
  uint64_t x[4];   // arrivals: out-projection, MLP partial sums, MLP rows, fold (or head partial sums)
  int abort_flag;
};

extern __shared__ __align__(128) uint8_t g_mma_smem[];

// shared-memory plan (bytes)
struct Plan {
  int act, hid, res, xa, xb, part, red, vec, raw, total;
};
__host__ __device__ constexpr Plan plan_of(int D, int HS) {
  Plan p{};
  const int DS = D / kC, KS = D / 64;
  const int red_a = KS * kRows * (DS + 4), red_b = 8 * kRows * 20;
  p.act = 128;                                    // [hi, lo][32][D + 8] bf16
  p.hid = p.act + 2 * kRows * (D + 8) * 2;        // [hi, lo][32][HS + 8] bf16
  p.res = p.hid + 2 * kRows * (HS + 8) * 2;       // [32][D + 4] residual stream
  p.xa = p.res + kRows * (D + 4) * 4;             // [32][D + 4] rows that arrive: out-projection, fold, head
  p.xb = p.xa + kRows * (D + 4) * 4;              // [32][D + 4] rows that arrive: MLP
  p.part = p.xb + kRows * (D + 4) * 4;            // [4][32][DS] MLP partial sums of this CTA's columns
  p.red = p.part + kC * kRows * DS * 4;           // partial sums of the k splits
  p.vec = p.red + 4 * (red_a > red_b ? red_a : red_b);  // LayerNorm vectors and biases
  p.raw = p.vec + 4 * (9 * D + 2 * HS);           // [8][32] head outputs
  p.total = p.raw + 8 * 32 * 4;
  return p;
}

__device__ __noinline__ void wait_slow(uint32_t bar, volatile int* abort_flag) {
  const long long t0 = clock64();
  for (;;) {
    if (*abort_flag) return;
    if (mbar_try(bar, 0)) return;
    if (clock64() - t0 > kDefaultWaitCycles) {
      *abort_flag = 1;
      return;
    }
  }
}
// bounded wait for the one completion of an exchange barrier
__device__ __forceinline__ void wait_x(int i) {
  Bars* b = reinterpret_cast<Bars*>(g_mma_smem);
  const uint32_t bar = smem_u32(&b->x[i]);
  if (!mbar_test(bar, 0)) wait_slow(bar, &b->abort_flag);
}

__device__ __forceinline__ uint4 ldg_weights(const uint4* p) {  // volatile: stays where it is written, ahead of the waits
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack2(x, y);
  lo = pack2(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ float gelu_erf(float v) { return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f)); }

// An activation operand: hi part, then the lo part, rows pitch bytes apart (an odd number of 16-byte pieces).
struct Operand {
  uint32_t base;   // shared address of this lane's ldmatrix row
  int pitch, lo;
  __device__ __forceinline__ Operand(const uint8_t* p, int k) : pitch((k + 8) * 2), lo(kRows * (k + 8) * 2) {
    const int lane = threadIdx.x & 31;
    base = smem_u32(p) + (lane & 15) * pitch + (lane >> 4) * 16;
  }
};

// Weight fragments of 16 columns: two tiles of 8 columns, NU blocks of 32 k
template <int NU>
struct Frags {
  uint4 w[2][NU];
  // m: matrix slice in fragment order, k32 blocks per column tile; blocks u0 .. u0 + n - 1 of column pair `pair`
  __device__ __forceinline__ void load(const uint4* m, int pair, int k32, int u0, int n) {
    const uint4* p = m + (size_t)(2 * pair * k32 + u0) * 32 + (threadIdx.x & 31);
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int u = 0; u < NU; ++u)
        if (u < n) w[t][u] = ldg_weights(p + (t * k32 + u) * 32);
  }
};

// acc[m tile][n tile] += act . w over n blocks of 32 k; PARTS 2: hi and lo part of the activations, 1: the hi part
template <int PARTS, int NU>
__device__ __forceinline__ void multiply(float (&acc)[2][2][4], const Frags<NU>& f, const Operand& x, int u0, int n) {
  // the fragments of a k step are read while the MMAs of the step before it run
  uint32_t a[2][2][PARTS][4];
  auto read = [&](int step) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int part = 0; part < PARTS; ++part)
        ldmatrix4(a[step & 1][m][part], x.base + part * x.lo + m * 16 * x.pitch + u0 * 64 + step * 32);
  };
  read(0);
#pragma unroll
  for (int step = 0; step < 2 * NU; ++step) {
    const int u = step >> 1;
    if (u < n) {
      if (step + 1 < 2 * NU && (step + 1) >> 1 < n) read(step + 1);
#pragma unroll
      for (int part = 0; part < PARTS; ++part)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int t = 0; t < 2; ++t)
            mma(acc[m][t], a[step & 1][m][part], step & 1 ? f.w[t][u].z : f.w[t][u].x, step & 1 ? f.w[t][u].w : f.w[t][u].y);
    }
  }
}
__device__ __forceinline__ void zero(float (&acc)[2][2][4]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) (&acc[0][0][0])[i] = 0.f;
}

// f(row, column of the pair, v[4]): every lane's results as four neighbouring columns of one row
template <class F>
__device__ __forceinline__ void each_quad(const float (&acc)[2][2][4], F f) {
  const int lane = threadIdx.x & 31;
  const bool odd = lane & 1;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float* c = acc[m][t];
      const float r0 = __shfl_xor_sync(0xffffffffu, odd ? c[0] : c[2], 1);
      const float r1 = __shfl_xor_sync(0xffffffffu, odd ? c[1] : c[3], 1);
      const float v[4] = {odd ? r0 : c[0], odd ? r1 : c[1], odd ? c[2] : r0, odd ? c[3] : r1};
      f(16 * m + (lane >> 2) + (odd ? 8 : 0), 8 * t + 4 * ((lane & 3) >> 1), v);
    }
}

__device__ __forceinline__ void store_split(uint8_t* operand, int k, int row, int col, const float (&v)[4]) {
  uint2 hi, lo;
  split2(v[0], v[1], hi.x, lo.x);
  split2(v[2], v[3], hi.y, lo.y);
  uint8_t* p = operand + (row * (k + 8) + col) * 2;
  *reinterpret_cast<uint2*>(p) = hi;
  *reinterpret_cast<uint2*>(p + kRows * (k + 8) * 2) = lo;
}

// act <- LayerNorm(res + xg + bias) as hi and lo part; res <- the same unless it is the last use; optional copy of this
// CTA's eight rows to global memory.  Eight lanes per row.  `x`: the exchange that brings xg (-1: none).
template <int D>
__device__ __forceinline__ void layer_norm(float* res, const float* xg, const float* bias, const float* gamma, const float* beta,
                                        uint8_t* act, int x, float* copy, int rank, int n_valid) {
  constexpr int N = D / 32, P = D + 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 8) {
    const int row = warp * 4 + (lane >> 3), c0 = 4 * (lane & 7);
    float v[N][4];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float4 r = *reinterpret_cast<const float4*>(res + row * P + c0 + 32 * i);
      v[i][0] = r.x; v[i][1] = r.y; v[i][2] = r.z; v[i][3] = r.w;
      if (bias) {
        const float4 b = *reinterpret_cast<const float4*>(bias + c0 + 32 * i);
        v[i][0] += b.x; v[i][1] += b.y; v[i][2] += b.z; v[i][3] += b.w;
      }
    }
    if (x >= 0) wait_x(x);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (xg) {
        const float4 g = *reinterpret_cast<const float4*>(xg + row * P + c0 + 32 * i);
        v[i][0] += g.x; v[i][1] += g.y; v[i][2] += g.z; v[i][3] += g.w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) s += v[i][e];
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = s * (1.0f / D);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[i][e] -= mean;
        ss = fmaf(v[i][e], v[i][e], ss);
      }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rstd = 1.0f / sqrtf(ss * (1.0f / D) + 1e-5f);
    const bool mine = copy && (row >> 3) == rank && row < n_valid;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float4 g = *reinterpret_cast<const float4*>(gamma + c0 + 32 * i), b = *reinterpret_cast<const float4*>(beta + c0 + 32 * i);
      const float y[4] = {fmaf(v[i][0] * rstd, g.x, b.x), fmaf(v[i][1] * rstd, g.y, b.y), fmaf(v[i][2] * rstd, g.z, b.z),
                          fmaf(v[i][3] * rstd, g.w, b.w)};
      const float4 y4 = make_float4(y[0], y[1], y[2], y[3]);
      *reinterpret_cast<float4*>(res + row * P + c0 + 32 * i) = y4;
      store_split(act, D, row, c0 + 32 * i, y);
      if (mine) *reinterpret_cast<float4*>(copy + ((c0 + 32 * i) >> 2) * 128 + row * 4) = y4;   // lane-major tile
    }
  }
  __syncthreads();
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1) dense_mma_kernel(const __grid_constant__ DenseArgs a) {
  constexpr int DS = D / kC, P = D + 4, NU = D / 32, KS = D / 64, PAIRS = DS / 16;
  const int HS = a.Dff / kC, KU = HS / 32;
  const Plan p = plan_of(D, HS);
  Bars* bars = reinterpret_cast<Bars*>(g_mma_smem);
  uint8_t* act = g_mma_smem + p.act;
  uint8_t* hid = g_mma_smem + p.hid;
  float* res = reinterpret_cast<float*>(g_mma_smem + p.res);
  float* xa = reinterpret_cast<float*>(g_mma_smem + p.xa);
  float* xb = reinterpret_cast<float*>(g_mma_smem + p.xb);
  float* part = reinterpret_cast<float*>(g_mma_smem + p.part);
  float* red = reinterpret_cast<float*>(g_mma_smem + p.red);
  float* vec = reinterpret_cast<float*>(g_mma_smem + p.vec);
  float* raw = reinterpret_cast<float*>(g_mma_smem + p.raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t crank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const int rank = (int)crank;
  const long row0 = (long)(blockIdx.x / kC) * kRows;
  const int n_valid = (int)min((long)kRows, (long)a.rows - row0);

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars->x[i])) : "memory");
    bars->abort_flag = a.wait_cycles <= 1;   // one cycle: the limit has run out here (tests); any other is the built-in one,
                                              // which costs the waits no instruction: passing it on took 0.3 % of a job
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // what this CTA will receive: 32 rows of D floats each time, the last one of a head launch 4 x 8 x 16 floats
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bars->x[i])),
                   "r"(i == 3 && a.do_head ? kC * 8 * 16 * 4 : kRows * D * 4)
                   : "memory");
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // peers may send once all have passed

  // ---- what needs nothing from the preceding kernel: vectors, the first weights ----
  float* v_ln2g = vec, *v_ln2b = vec + D, *v_b2 = vec + 2 * D, *v_ln3g = vec + 3 * D, *v_ln3b = vec + 4 * D;
  float* v_ln1g = vec + 5 * D, *v_ln1b = vec + 6 * D, *v_lnfg = vec + 7 * D, *v_lnfb = vec + 8 * D;
  float* v_b1 = vec + 9 * D, *v_ba = v_b1 + HS;
  if (tid < D) {   // every load before the first store: one round trip
    const bool post = a.do_post, pre = a.do_pre, fin = a.do_final;
    const float* src[9] = {post ? a.post_w.ln2_g : nullptr, post ? a.post_w.ln2_b : nullptr, post ? a.post_w.b2 : nullptr,
                           post ? a.post_w.ln3_g : nullptr, post ? a.post_w.ln3_b : nullptr, pre ? a.pre_w.ln1_g : nullptr,
                           pre ? a.pre_w.ln1_b : nullptr,   fin ? a.lnf_g : nullptr,         fin ? a.lnf_b : nullptr};
    float v[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = src[i] ? __ldg(src[i] + tid) : 0.f;
#pragma unroll
    for (int i = 0; i < 9; ++i) vec[i * D + tid] = v[i];
  }
  for (int i = tid; i < HS; i += kThreads) {
    if (a.do_post) v_b1[i] = __ldg(a.post_w.b1 + rank * HS + i);
    if (a.do_head) v_ba[i] = __ldg(a.ba + rank * HS + i);
  }
  // slices of this rank: hi part, then lo part of every matrix (in uint4: eight weights)
  constexpr int WD = D * DS / 8;
  const int WH = D * HS / 8;
  const uint4* w_post = reinterpret_cast<const uint4*>(a.post_w.mma_post) + (size_t)rank * 2 * (WD + 2 * WH);
  const uint4* w_pre = reinterpret_cast<const uint4*>(a.pre_w.mma_pre) + (size_t)rank * 8 * WD;
  const uint4* w_head = reinterpret_cast<const uint4*>(a.mma_head) + (size_t)rank * 2 * (WH + 2 * HS);
  const int lo_post = a.post_w.tc_lo, lo_pre = a.pre_w.tc_lo;
  const Operand x_act(act, D), x_hid(hid, HS);
  float acc[2][2][4];
  const int sq_pair = warp % PAIRS, sq_ks = warp / PAIRS;   // D x D products: column pair and k split of this warp
  const bool sq_active = warp < PAIRS * KS;
  Frags<2> wsq;
  if (sq_active) wsq.load(a.do_post ? w_post : w_pre, sq_pair, NU, 2 * sq_ks, 2);

  dep_wait();
  dep_trigger();

  // ---- rows in ----
  {
    const float4* src = reinterpret_cast<const float4*>(a.do_post ? a.attn : a.x_in) + row0 * (D / 4);
    const float4* s1 = reinterpret_cast<const float4*>(a.do_post ? a.x1_in : a.x_in) + row0 * (D / 4);
    const bool lm = a.do_post || a.x_in_lane_major;
    constexpr int NI = (kRows * D / 4 + kThreads - 1) / kThreads;
    float4 v[NI], r[NI];
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int i = tid + j * kThreads;
      const bool ok = i < kRows * D / 4 && (lm || i / (D / 4) < n_valid);
      v[j] = ok ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      r[j] = ok ? s1[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const int i = tid + j * kThreads;
      if (i < kRows * D / 4) {
        const int row = lm ? i & 31 : i / (D / 4), c4 = lm ? i >> 5 : i - row * (D / 4);
        const float y[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        store_split(act, D, row, 4 * c4, y);
        *reinterpret_cast<float4*>(res + row * P + 4 * c4) = r[j];
      }
    }
  }
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

  // this warp's share of act . W for a [D][DS] slice, put together and sent to every CTA's xa
  auto square_send = [&](const uint4* m, bool lo, int x) {
    if (sq_active) {
      zero(acc);
      multiply<2>(acc, wsq, x_act, 2 * sq_ks, 2);
      if (lo) {
        wsq.load(m + WD, sq_pair, NU, 2 * sq_ks, 2);
        multiply<1>(acc, wsq, x_act, 2 * sq_ks, 2);
      }
      each_quad(acc, [&](int r, int c, const float (&v)[4]) {
        *reinterpret_cast<float4*>(red + (sq_ks * kRows + r) * (DS + 4) + 16 * sq_pair + c) = make_float4(v[0], v[1], v[2], v[3]);
      });
    }
    __syncthreads();
    for (int i = tid; i < kRows * DS / 4; i += kThreads) {
      const int r = i / (DS / 4), c = 4 * (i - r * (DS / 4));
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const float4 t = *reinterpret_cast<const float4*>(red + (k * kRows + r) * (DS + 4) + c);
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
      const uint32_t at = smem_u32(xa + r * P + rank * DS + c), bar = smem_u32(&bars->x[x]);
#pragma unroll
      for (int q = 0; q < kC; ++q) st_async<4>(map_to_rank(at, q), v, map_to_rank(bar, q));
    }
  };
  // hid <- gelu(act . W + b) for a [D][HS] slice; `w`: fragments of this warp's first column pair
  auto hidden = [&](Frags<NU>& w, const uint4* m, bool lo, const float* bias) {
#pragma unroll 1
    for (int pr = warp; pr < HS / 16; pr += kWarps) {
      if (pr != warp) w.load(m, pr, NU, 0, NU);
      zero(acc);
      multiply<2>(acc, w, x_act, 0, NU);
      if (lo) {
        w.load(m + WH, pr, NU, 0, NU);
        multiply<1>(acc, w, x_act, 0, NU);
      }
      each_quad(acc, [&](int r, int c, const float (&v)[4]) {
        const float4 b = *reinterpret_cast<const float4*>(bias + 16 * pr + c);
        const float y[4] = {gelu_erf(v[0] + b.x), gelu_erf(v[1] + b.y), gelu_erf(v[2] + b.z), gelu_erf(v[3] + b.w)};
        store_split(hid, HS, r, 16 * pr + c, y);
      });
    }
  };

  Frags<NU> wide;
  const bool hid_active = warp < HS / 16;
  if (a.do_post) {
    square_send(w_post, lo_post & 1, 0);
    const uint4* w1 = w_post + 2 * WD, *w2 = w1 + 2 * WH;
    if (hid_active) wide.load(w1, warp, NU, 0, NU);
    layer_norm<D>(res, xa, nullptr, v_ln2g, v_ln2b, act, 0, nullptr, rank, n_valid);
    hidden(wide, w1, lo_post & 2, v_b1);
    constexpr int ND = 6;   // blocks of 32 k held at once
    Frags<ND> deep;
    const bool w2_active = warp < D / 16;
    if (w2_active) deep.load(w2, warp, KU, 0, min(KU, ND));
    __syncthreads();
    if (w2_active) {
      zero(acc);
#pragma unroll 1
      for (int u = 0; u < KU; u += ND) {
        const int n = min(KU - u, ND);
        if (u) deep.load(w2, warp, KU, u, n);
        multiply<2>(acc, deep, x_hid, u, n);
        if (lo_post & 4) {
          deep.load(w2 + WH, warp, KU, u, n);
          multiply<1>(acc, deep, x_hid, u, n);
        }
      }
      const int owner = 16 * warp / DS;
      const uint32_t at = map_to_rank(smem_u32(part + rank * kRows * DS + 16 * warp - owner * DS), owner);
      const uint32_t bar = map_to_rank(smem_u32(&bars->x[1]), owner);
      each_quad(acc, [&](int r, int c, const float (&v)[4]) { st_async<4>(at + (r * DS + c) * 4, v, bar); });
    }
    if (a.do_pre && sq_active) wsq.load(w_pre, sq_pair, NU, 2 * sq_ks, 2);
    wait_x(1);
    for (int i = tid; i < kRows * DS / 4; i += kThreads) {
      const int r = i / (DS / 4), c = 4 * (i - r * (DS / 4));
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        const float4 t = *reinterpret_cast<const float4*>(part + (k * kRows + r) * DS + c);
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
      const uint32_t at = smem_u32(xb + r * P + rank * DS + c), bar = smem_u32(&bars->x[2]);
#pragma unroll
      for (int q = 0; q < kC; ++q) st_async<4>(map_to_rank(at, q), v, map_to_rank(bar, q));
    }
    layer_norm<D>(res, xb, v_b2, v_ln3g, v_ln3b, act, 2, nullptr, rank, n_valid);
  }

  if (a.do_head) {
    if (hid_active) wide.load(w_head, warp, NU, 0, NU);
    if (a.do_final) layer_norm<D>(res, nullptr, nullptr, v_lnfg, v_lnfb, act, -1, nullptr, rank, n_valid);
    hidden(wide, w_head, a.tc_head_lo & 1, v_ba);
    const uint4* wb = w_head + 2 * WH;   // [HS][16]: one column pair, a block of 32 k per warp
    Frags<1> last;
    if (warp < KU) last.load(wb, 0, KU, warp, 1);
    __syncthreads();
    if (warp < KU) {
      zero(acc);
      multiply<2>(acc, last, x_hid, warp, 1);
      if (a.tc_head_lo & 2) {
        last.load(wb + 2 * HS, 0, KU, warp, 1);
        multiply<1>(acc, last, x_hid, warp, 1);
      }
      each_quad(acc, [&](int r, int c, const float (&v)[4]) {
        *reinterpret_cast<float4*>(red + (warp * kRows + r) * 20 + c) = make_float4(v[0], v[1], v[2], v[3]);
      });
    }
    __syncthreads();
    if (tid < kRows * 4) {   // rows 8 c .. 8 c + 7 belong to CTA c
      const int r = tid >> 2, c = 4 * (tid & 3);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      for (int k = 0; k < KU; ++k) {
        const float4 t = *reinterpret_cast<const float4*>(red + (k * kRows + r) * 20 + c);
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
      st_async<4>(map_to_rank(smem_u32(xa + (rank * 8 + (r & 7)) * 16 + c), r >> 3), v, map_to_rank(smem_u32(&bars->x[3]), r >> 3));
    }
    if (warp < 8) {
      wait_x(3);
      const int r = rank * 8 + warp;
      if (lane < 16) {
        float v = lane < 3 * a.n_comp ? __ldg(a.bb + lane) : 0.f;
#pragma unroll
        for (int k = 0; k < kC; ++k) v += xa[(k * 8 + warp) * 16 + lane];
        raw[warp * 32 + lane] = v;
      }
      __syncwarp();
      if (r < n_valid && !*(volatile int*)&bars->abort_flag) head_row(a, raw + warp * 32, row0 + r);
    }
  } else if (a.do_pre) {
    square_send(w_pre, lo_pre & 8, 3);
    // Q | K | V columns of this rank: 3 * PAIRS column pairs
    const uint4* wq = w_pre + 2 * WD;
    const bool qkv_active = warp < 3 * PAIRS;
    if (qkv_active) wide.load(wq, warp, NU, 0, NU);
    layer_norm<D>(res, xa, nullptr, v_ln1g, v_ln1b, act, 3, a.x1_out + row0 * D, rank, n_valid);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // nobody sends any more
    if (qkv_active) {
      zero(acc);
      multiply<2>(acc, wide, x_act, 0, NU);
      if (lo_pre & 16) {
        wide.load(wq + 3 * WD, warp, NU, 0, NU);
        multiply<1>(acc, wide, x_act, 0, NU);
      }
      if (!*(volatile int*)&bars->abort_flag) {
        const int which = warp / PAIRS, col0 = rank * DS + 16 * (warp - which * PAIRS);
        each_quad(acc, [&](int r, int c, const float (&v)[4]) {
          if (r >= n_valid) return;
          if (which == 0)
            store4(reinterpret_cast<__nv_bfloat16*>(a.q_out) + (size_t)(row0 + r) * D + col0 + c, v);
          else if (a.kv.mode != KV_NONE)
            scatter4<__nv_bfloat16>(a.kv, which, (unsigned)(row0 + r), col0 + c, v);
        });
      }
    }
  }
  // nobody leaves while a peer could still write here
  __syncthreads();
  if (a.do_head) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (bars->abort_flag) {
    if (tid == 0 && a.status) atomicExch(a.status, 6);
    const long long t0 = clock64();
    while (clock64() - t0 < 100000) {   // after a wait that gave up, a peer's stores may be in flight
    }
  }
}

template <int D>
SmemConfig& smem_config() {
  static SmemConfig c;
  return c;
}

constexpr int kMaxDff = 1024;   // of the weight tiles this chain takes (dense_tc_applicable)

// rows of the clusters that fit the GPU at once
template <int D>
int rows_at_once(int d_ff) {
  static thread_local int cached[kMaxDevices][kMaxDff / 128 + 1];
  int dev = 0;
  if (d_ff > kMaxDff || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int& rows = cached[dev][d_ff / 128];
  if (rows) return rows;
  const size_t smem = plan_of(D, d_ff / kC).total;
  if (smem_config<D>().ensure(dense_mma_kernel<D>, smem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kC);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kC;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, dense_mma_kernel<D>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return rows = n * kRows;
}

template <int D>
int launch_d(const DenseArgs& args, cudaStream_t s) {
  DenseArgs a = args;
  a.wait_cycles = debug_wait_cycles() > 0 ? debug_wait_cycles() : kDefaultWaitCycles;
  const size_t smem = plan_of(D, a.Dff / kC).total;
  cudaError_t e = smem_config<D>().ensure(dense_mma_kernel<D>, smem);
  prof_begin(PROF_DENSE, s);
  if (e == cudaSuccess)
    e = launch_dependent_cluster(dense_mma_kernel<D>, dim3((a.rows + kRows - 1) / kRows * kC), dim3(kThreads), smem, s, kC, a);
  prof_end(s);
  ARTAB_REQUIRE(e == cudaSuccess, ARTAB_ELAUNCH, "dense_mma_kernel: launch refused: %s", cudaGetErrorString(e));
  count_launch();
  return check_launch("dense_mma_kernel");
}

}  // namespace

// One wave of clusters: beyond it the tcgen05 chain, whose time hardly grows up to 148 row tiles, is the faster one.
bool dense_mma_applicable(const DenseArgs& a) {
  if (!a.lane_major || !(a.do_pre || (a.do_post && a.do_head)) || a.x_out || a.z_out || !dense_tc_applicable(a)) return false;
  if ((a.do_post && !a.post_w.mma_post) || (a.do_pre && !a.pre_w.mma_pre) || (a.do_head && !a.mma_head)) return false;
  const int most = a.D == 64 ? rows_at_once<64>(a.Dff) : a.D == 128 ? rows_at_once<128>(a.Dff) : rows_at_once<192>(a.Dff);
  return a.rows <= most;
}

int launch_dense_mma(const DenseArgs& a, cudaStream_t s) {
  switch (a.D) {
    case 64: return launch_d<64>(a, s);
    case 128: return launch_d<128>(a, s);
    default: return launch_d<192>(a, s);
  }
}

}  // namespace artab
