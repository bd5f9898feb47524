// Per-token layer chain in fp32 FMA for many rows (prefill, teacher forcing, masked forward).
//
// The same chain as dense_chain_kernel, but a CTA owns 16 - 128 rows and every product is a register tile of
// TR rows x 4 columns per thread: 4 + TR 16-byte shared-memory reads for 16 TR FMAs.  The 8-row kernel reads
// an activation and a weight from shared memory for every 2 - 4 FMAs and walks all weights once per 8 rows,
// which kept it at 2 - 4 % of the FMA rate; a 16-byte read costs the SM four cycles, so at TR = 8 the FMA
// pipe and the shared-memory pipe are about equally busy.
//
// Every matrix is a sequence of D x D panels, stored panel after panel in the order of use (_pack.py): fold,
// Q, K, V | out-projection, then for every D-wide chunk of the hidden layer W1 and W2, whose products
// accumulate in registers, so the hidden layer never exists as a whole.  A producer warp streams 32-row slabs
// of the panels through a ring of bulk copies.
#include "cluster.cuh"
#include "dense.cuh"
#include "head.cuh"
#include "kv_scatter.cuh"

namespace artab {

namespace {

constexpr int kSlots = 4;

extern __shared__ __align__(128) uint8_t g_fma_smem[];

template <int D>
struct Shape {
  static constexpr int CG = D / 4;                       // column groups: threads across a row
  static constexpr int RG = D == 64 ? 16 : 8;            // row groups
  static constexpr int T = CG * RG;                      // compute threads: 256, 256, 384
  static constexpr int P = D + 4;                        // floats between activation rows
  static constexpr int SLAB = 32 * D;                    // floats of a slab: 32 rows of a panel
};

struct Bars {
  uint64_t full[kSlots], empty[kSlots];
  long long limit;
  int abort_flag;
};

__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, volatile Bars* b) {
  const long long t0 = clock64();
  for (;;) {
    if (b->abort_flag) return;   // first: after an abort no wait may block again
    if (clock64() - t0 > b->limit) {
      b->abort_flag = 1;
      return;
    }
    if (mbar_try(bar, parity)) return;
  }
}
// bounded; on return the phase is over or the CTA is aborting
__device__ __forceinline__ void mbar_wait(uint64_t* b, uint32_t parity, Bars* bars) {
  const uint32_t bar = smem_u32(b);
  if (!mbar_test(bar, parity)) wait_slow(bar, parity, bars);
}
template <int T>
__device__ __forceinline__ void sync_compute() { asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory"); }
__device__ __forceinline__ float gelu_erf(float v) { return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f)); }

template <int D, int TR>
struct Chain {
  using S = Shape<D>;
  Bars* bars;
  float* ring;
  int used;                 // slabs consumed
  int cg, rg;

  // acc += act[R][D] . panel[D][D], this thread's TR rows and 4 columns
  __device__ __forceinline__ void panel(const float* act, float (&acc)[TR][4]) {
    const float* x = act + rg * TR * S::P;
#pragma unroll 1
    for (int s = 0; s < D / 32; ++s, x += 32) {
      const int slot = used % kSlots;
      mbar_wait(&bars->full[slot], (used / kSlots) & 1, bars);
      const float4* w = reinterpret_cast<const float4*>(ring + slot * S::SLAB) + cg;
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {
        float4 ww[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) ww[i] = w[(4 * k + i) * (D / 4)];
#pragma unroll
        for (int r = 0; r < TR; ++r) {
          const float4 a = *reinterpret_cast<const float4*>(x + r * S::P + 4 * k);
          acc[r][0] = fmaf(a.w, ww[3].x, fmaf(a.z, ww[2].x, fmaf(a.y, ww[1].x, fmaf(a.x, ww[0].x, acc[r][0]))));
          acc[r][1] = fmaf(a.w, ww[3].y, fmaf(a.z, ww[2].y, fmaf(a.y, ww[1].y, fmaf(a.x, ww[0].y, acc[r][1]))));
          acc[r][2] = fmaf(a.w, ww[3].z, fmaf(a.z, ww[2].z, fmaf(a.y, ww[1].z, fmaf(a.x, ww[0].z, acc[r][2]))));
          acc[r][3] = fmaf(a.w, ww[3].w, fmaf(a.z, ww[2].w, fmaf(a.y, ww[1].w, fmaf(a.x, ww[0].w, acc[r][3]))));
        }
      }
      ++used;
      __syncwarp();
      if ((threadIdx.x & 31) == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bars->empty[slot])) : "memory");
    }
  }
  __device__ __forceinline__ void store(float* dst, const float (&acc)[TR][4]) {
#pragma unroll
    for (int r = 0; r < TR; ++r)
      *reinterpret_cast<float4*>(dst + (rg * TR + r) * S::P + 4 * cg) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
  }
};

template <int TR>
__device__ __forceinline__ void zero(float (&acc)[TR][4]) {
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
}

// dst[r] = LayerNorm(a[r] (+ h[r]) (+ bias) (+ g[r] from global memory)), one warp per row; optional copy to global
template <int D>
__device__ __noinline__ void ln_rows(float* dst, const float* a, const float* h, const float* bias, const float* g,
                                     const float* gamma, const float* beta, float* copy, int rows, int n_valid) {
  using S = Shape<D>;
  constexpr int N = D / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float gm[N], bt[N], bs[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    gm[i] = __ldg(gamma + lane + 32 * i);
    bt[i] = __ldg(beta + lane + 32 * i);
    bs[i] = bias ? __ldg(bias + lane + 32 * i) : 0.f;
  }
#pragma unroll 2
  for (int r = warp; r < rows; r += S::T / 32) {
    float v[N], s = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int d = lane + 32 * i;
      v[i] = bs[i];
      if (a) v[i] += a[r * S::P + d];
      if (h) v[i] += h[r * S::P + d];
      if (g && r < n_valid) v[i] += g[(size_t)r * D + d];
      s += v[i];
    }
    const float mean = warp_sum(s) * (1.0f / D);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      v[i] -= mean;
      ss = fmaf(v[i], v[i], ss);
    }
    const float rstd = 1.0f / sqrtf(warp_sum(ss) * (1.0f / D) + 1e-5f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int d = lane + 32 * i;
      const float y = v[i] * rstd * gm[i] + bt[i];
      dst[r * S::P + d] = y;
      if (copy && r < n_valid) copy[(size_t)r * D + d] = y;
    }
  }
  sync_compute<S::T>();
}

template <typename T, int D, int TR>
__global__ void __launch_bounds__(Shape<D>::T + 32, D == 64 ? 2 : 1) dense_fma_kernel(const DenseArgs a) {
  using S = Shape<D>;
  constexpr int R = S::RG * TR;
  float* ring = reinterpret_cast<float*>(g_fma_smem);
  float* x = ring + kSlots * S::SLAB;   // [R][P] residual stream
  float* h = x + R * S::P;              // [R][P] attention rows, hidden chunk, product to be normalised
  Bars* bars = reinterpret_cast<Bars*>(h + R * S::P);
  const int tid = threadIdx.x;
  const long row0 = (long)blockIdx.x * R;
  const int n_valid = (int)min((long)R, (long)a.rows - row0);
  const int n_hidden = a.Dff / D;

  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars->full[i])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&bars->empty[i])), "r"(S::T / 32) : "memory");
    }
    bars->abort_flag = 0;
    bars->limit = a.wait_cycles;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (tid >= S::T) {
    // ------------------------------ producer warp ------------------------------
    int issued = 0;
    if (tid == S::T) {
      auto stream = [&](const float* w, int panels) {
#pragma unroll 1
        for (int i = 0; i < panels * (D / 32); ++i, w += S::SLAB) {
          const int slot = issued % kSlots;
          if (issued >= kSlots) mbar_wait(&bars->empty[slot], ((issued / kSlots) + 1) & 1, bars);
          if (*(volatile int*)&bars->abort_flag) return;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bars->full[slot])),
                       "r"(S::SLAB * 4)
                       : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           smem_u32(ring + slot * S::SLAB)),
                       "l"(w), "r"(S::SLAB * 4), "r"(smem_u32(&bars->full[slot]))
                       : "memory");
          ++issued;
        }
      };
      if (a.do_post) stream(a.post_w.fma_post, 1 + 2 * n_hidden);
      if (a.do_head) stream(a.fma_head, 2 * n_hidden);
      else if (a.do_pre) stream(a.pre_w.fma_pre, 4);
    }
    __syncthreads();   // the compute threads are done, or have given up: then the copies in flight land before the CTA may exit
    if (tid == S::T && bars->abort_flag) {
      for (int i = max(0, issued - kSlots); i < issued; ++i) {
        const long long t0 = clock64();
        while (!mbar_try(smem_u32(&bars->full[i % kSlots]), (i / kSlots) & 1) && clock64() - t0 < kDefaultWaitCycles) {
        }
      }
    }
    return;
  }

  Chain<D, TR> ch{bars, ring, 0, tid % S::CG, tid / S::CG};
  float acc[TR][4];
  auto load_rows = [&](float* dst, const float* src) {
    for (int i = tid; i < R * (D / 4); i += S::T) {
      const int r = i / (D / 4), c = i - r * (D / 4);
      *reinterpret_cast<float4*>(dst + r * S::P + 4 * c) =
          r < n_valid ? __ldg(reinterpret_cast<const float4*>(src + (size_t)(row0 + r) * D) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    sync_compute<S::T>();
  };
  // h <- the product in acc, once every thread is done reading h
  auto to_h = [&]() {
    sync_compute<S::T>();
    ch.store(h, acc);
    sync_compute<S::T>();
  };
  // MLP or head: acc <- act(x . W1 + b) . W2 chunk by chunk; the result is left in h
  auto mlp = [&](const float* bias) {
    float out[TR][4];
    zero<TR>(out);
#pragma unroll 1
    for (int j = 0; j < n_hidden; ++j) {
      const float4 b = __ldg(reinterpret_cast<const float4*>(bias + j * D) + ch.cg);
      zero<TR>(acc);
      ch.panel(x, acc);
#pragma unroll
      for (int r = 0; r < TR; ++r) {
        acc[r][0] = gelu_erf(acc[r][0] + b.x);
        acc[r][1] = gelu_erf(acc[r][1] + b.y);
        acc[r][2] = gelu_erf(acc[r][2] + b.z);
        acc[r][3] = gelu_erf(acc[r][3] + b.w);
      }
      to_h();
      ch.panel(h, out);
    }
#pragma unroll
    for (int r = 0; r < TR; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = out[r][c];
    to_h();
  };

  if (a.do_post) {
    load_rows(h, a.attn);
    zero<TR>(acc);
    ch.panel(h, acc);
    to_h();
    ln_rows<D>(x, nullptr, h, nullptr, a.x1_in + (size_t)row0 * D, a.post_w.ln2_g, a.post_w.ln2_b, nullptr, R, n_valid);
    mlp(a.post_w.b1);
    ln_rows<D>(x, x, h, a.post_w.b2, nullptr, a.post_w.ln3_g, a.post_w.ln3_b, a.x_out ? a.x_out + (size_t)row0 * D : nullptr, R, n_valid);
  } else {
    load_rows(x, a.x_in);
  }
  if (a.do_final)
    ln_rows<D>(x, x, nullptr, nullptr, nullptr, a.lnf_g, a.lnf_b, a.z_out ? a.z_out + (size_t)row0 * D : nullptr, R, n_valid);
  if (a.do_head) {
    mlp(a.ba);
    if (!bars->abort_flag) {
      const int warp = tid >> 5, lane = tid & 31;
      for (int r = warp; r < n_valid; r += S::T / 32) {
        float* raw = h + r * S::P;
        for (int i = lane; i < 3 * a.n_comp; i += 32) raw[i] += __ldg(a.bb + i);
        __syncwarp();
        head_row(a, raw, row0 + r);
      }
    }
  } else if (a.do_pre) {
    zero<TR>(acc);
    ch.panel(x, acc);
    to_h();
    ln_rows<D>(x, x, h, nullptr, nullptr, a.pre_w.ln1_g, a.pre_w.ln1_b, a.x1_out + (size_t)row0 * D, R, n_valid);
#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
      zero<TR>(acc);
      ch.panel(x, acc);
#pragma unroll
      for (int r = 0; r < TR; ++r) {
        const int rr = ch.rg * TR + r;
        if (rr >= n_valid) continue;
        if (p == 0)
          store4<T>(reinterpret_cast<T*>(a.q_out) + (size_t)(row0 + rr) * D + 4 * ch.cg, acc[r]);
        else if (a.kv.mode != KV_NONE)
          scatter4<T>(a.kv, p, (unsigned)(row0 + rr), 4 * ch.cg, acc[r]);
      }
    }
  }
  __syncthreads();
  if (tid == 0 && bars->abort_flag && a.status) atomicExch(a.status, 5);
}

template <typename T, int D, int TR>
int launch_variant(const DenseArgs& args, cudaStream_t s) {
  DenseArgs a = args;
  a.wait_cycles = debug_wait_cycles() > 0 ? debug_wait_cycles() : kDefaultWaitCycles;
  using S = Shape<D>;
  constexpr int R = S::RG * TR;
  const size_t smem = (size_t)(kSlots * S::SLAB + 2 * R * S::P) * sizeof(float) + sizeof(Bars);
  static SmemConfig configured;
  const cudaError_t e = configured.ensure(dense_fma_kernel<T, D, TR>, smem, D == 64);
  ARTAB_REQUIRE(e == cudaSuccess, ARTAB_ELAUNCH, "dense_fma_kernel: %zu bytes of shared memory refused: %s", smem,
                cudaGetErrorString(e));
  prof_begin(PROF_DENSE, s);
  dense_fma_kernel<T, D, TR><<<(a.rows + R - 1) / R, S::T + 32, smem, s>>>(a);
  prof_end(s);
  count_launch();
  return check_launch("dense_fma_kernel");
}

// Rows per thread: the fewest waves x (time of a wave).  A wave takes about TR units of FMAs plus two of
// LayerNorms, weight streaming and barriers that do not shrink with TR.
int pick_tr(int rows, int row_groups, int per_sm) {
  int best = 1;
  double best_cost = 1e30;
  for (int tr = 1; tr <= 8; tr *= 2) {
    const long ctas = (rows + (long)row_groups * tr - 1) / ((long)row_groups * tr), slots = 148L * per_sm;
    const double cost = (double)((ctas + slots - 1) / slots) * (tr + 2.0);
    if (cost < best_cost) {
      best_cost = cost;
      best = tr;
    }
  }
  return best;
}

template <typename T, int D>
int launch_d(const DenseArgs& a, cudaStream_t s) {
  switch (pick_tr(a.rows, Shape<D>::RG, D == 64 ? 2 : 1)) {
    case 1: return launch_variant<T, D, 1>(a, s);
    case 2: return launch_variant<T, D, 2>(a, s);
    case 4: return launch_variant<T, D, 4>(a, s);
    default: return launch_variant<T, D, 8>(a, s);
  }
}

template <typename T>
int launch_t(const DenseArgs& a, cudaStream_t s) {
  switch (a.D) {
    case 64: return launch_d<T, 64>(a, s);
    case 128: return launch_d<T, 128>(a, s);
    default: return launch_d<T, 192>(a, s);
  }
}

}  // namespace

bool dense_fma_applicable(const DenseArgs& a) {
  if (!(a.D == 64 || a.D == 128 || a.D == 192) || a.Dff % a.D || a.Dff > 1024 || a.lane_major) return false;
  if (3 * a.n_comp > a.D || a.n_comp > 32) return false;
  if (a.do_post && !a.post_w.fma_post) return false;
  if (a.do_head && !a.fma_head) return false;
  if (a.do_pre && !a.do_head && !a.pre_w.fma_pre) return false;
  return a.do_post || a.do_pre || a.do_head;
}

int launch_dense_fma(const DenseArgs& a, cudaStream_t s) {
  if (a.rows <= 0) return ARTAB_OK;
  return a.kv.dtype == ARTAB_BF16 ? launch_t<__nv_bfloat16>(a, s) : launch_t<float>(a, s);
}

}  // namespace artab
