// Host side of the whole-sequence decode: applicability, shared-memory plan, context re-tiling, launch.
#include <cstring>

#include "attn.cuh"
#include "dense.cuh"
#include "seq.cuh"

namespace artab {

namespace {

constexpr size_t kSmemMax = 227 * 1024;
constexpr int kMaxRowsPerCluster = 16;
constexpr size_t kWorkspaceMax = (size_t)4 << 30;

inline int largest_divisor(int n, int most) {
  for (int c = most; c > 1; --c)
    if (n % c == 0) return c;
  return 1;
}

struct Areas {
  int red, area;  // floats
  bool direct;
};

// shared-memory floats of the kernel variant that holds R rows
Areas areas_of(const artab_model* m, int C, int R) {
  const int D = m->d_model, DH = m->head_dim, S = R / 2, DS = D / C, NB = (3 * m->n_comp + 15) & ~15;
  Areas a;
  // partial sums of the MLP: to every CTA at once while that is a few KB, else reduced first
  a.direct = C * R * D * 4 <= 12 * 1024;
  const int parts = kSeqWarps + kSeqBufferParts;
  const int attn = parts * R * (DH + 2) + kSeqWarps * 32 * R, prod = kSeqThreads * (R >= 2 ? R / 2 : 1);
  a.red = attn > prod ? attn : prod;
  a.area = R * kSeqPitch * (a.direct ? 6 : 7) + S * kSeqPitch + (a.direct ? C * R * kSeqPitch : C * R * DS) + C * S * NB +
           6 * 32 + 3 * S;
  a.area = (a.area + 3) & ~3;
  return a;
}

SeqMat mat_of(int K, int N) {
  SeqMat m;
  m.tiles = N / 16;
  m.octs = K / 32;
  const int most = kSeqWarps / m.tiles, per = (m.octs + most - 1) / most;  // k blocks per warp
  m.kw = (m.octs + per - 1) / per;
  return m;
}

// context in the order the kernel reads it: per (layer, group, head) tiles of 32 keys, fp32, the K rows in the
// lane order of the score loop ([Dh / 16][4 keys of a lane][32 lanes][4]), then the V rows in that of the P.V loop
// ([DH / 4 keys of a slice][128 / DH slices][DH]); bf16 V is hi + lo, which fp32 holds exactly
template <typename T>
__global__ void __launch_bounds__(256) retile_kernel(const T* __restrict__ k, const T* __restrict__ v, float4* __restrict__ out,
                                                     int DH, int n_ctx, int n_ctx_pad, int v_transposed) {
  const int tile = blockIdx.x, n_tiles = gridDim.x;
  const size_t head = (size_t)blockIdx.z * gridDim.y + blockIdx.y;  // (layer * group) * heads + head
  const T* kh = k + head * n_ctx_pad * DH;
  const T* vh = v + head * n_ctx_pad * DH * (v_transposed ? 2 : 1);
  float4* o = out + (head * n_tiles + tile) * (16 * DH);
  dep_wait();
  dep_trigger();
  const int d4 = DH / 4, ni = DH / 4;  // ni: keys of a slice of the P.V loop
  for (int i = threadIdx.x; i < 32 * d4; i += blockDim.x) {
    const int key = i / d4, d = i - key * d4, kk = tile * 32 + key;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
    if (kk < n_ctx) {
      const T* p = kh + (size_t)kk * DH + 4 * d;
      x = make_float4(to_f32<T>(p[0]), to_f32<T>(p[1]), to_f32<T>(p[2]), to_f32<T>(p[3]));
      if (!v_transposed) {
        p = vh + (size_t)kk * DH + 4 * d;
        y = make_float4(to_f32<T>(p[0]), to_f32<T>(p[1]), to_f32<T>(p[2]), to_f32<T>(p[3]));
      }
    }
    // dims 4d .. 4d + 3: block j = d / 4 of slice ds = d % 4; key 4 kg + (key % 4)
    o[((d >> 2) * 4 + (key & 3)) * 32 + (d & 3) * 8 + (key >> 2)] = x;
    if (!v_transposed) o[8 * DH + (key & (ni - 1)) * 32 + key / ni * d4 + d] = y;
  }
  if (v_transposed) {
    float* ov = reinterpret_cast<float*>(o + 8 * DH);
    for (int i = threadIdx.x; i < 32 * DH; i += blockDim.x) {
      const int d = i >> 5, key = i & 31, kk = tile * 32 + key;
      ov[(key & (ni - 1)) * 128 + key / ni * DH + d] = kk < n_ctx ? to_f32<T>(vh[(size_t)d * n_ctx_pad + kk]) + to_f32<T>(vh[(size_t)(DH + d) * n_ctx_pad + kk]) : 0.f;
    }
  }
}

size_t context_bytes(const artab_model* m, const artab_state* st) {
  return (size_t)m->n_layers * st->n_groups * m->n_heads * ((st->n_ctx + 31) / 32) * (64 * (size_t)m->head_dim * 4);
}

// Which path is faster, from a cost of each: microseconds per layer and target.
//
// One launch: a serial chain of phases per layer that grows with d_model and with the rows of the kernel variant, the
// walk of the head's context keys by one CTA, the context laid out again once per job, the head and the sampler per
// target.  A launch per layer: a chain that hardly notices the rows, and a contraction whose keys are split over the
// chip, bounded by the walk of a split (at most 16), by FMAs or by the bytes of the streams' own contexts.
//
// The constants are fitted to 856 points where both ran: d_model 64 - 192, 2 - 12 heads, 2 - 12 layers, fp32 and bf16,
// 1 - 400 streams on one context of 128 - 16384 rows or 4 - 250 own ones of 100 - 6000, 8 - 64 targets.  Of these the
// path picked is never more than 12 % slower than the other one and 0.1 % on average.  One launch against one per
// layer, us: d_model 128, fp32, 8 streams, 128 rows 12.6 : 45, 1000 rows 15.8 : 48, 4000 rows 29 : 52, 16384 rows
// 88 : 73; 200 streams, 1000 rows 51 : 58, 4000 rows 121 : 86; d_model 192, bf16, 32 streams, 1000 rows 22 : 30, 4000
// rows 38 : 33; 64 datasets of 500 rows 37 : 48, of 2000 rows 64 : 77.
bool faster_in_one_launch(const artab_model* m, const artab_state* st, int C, int spc) {
  const double D = m->d_model, L = m->n_layers, H = m->n_heads, head = m->head_dim / 32.0;
  const double B = st->n_streams, keys = st->n_ctx, targets = st->max_buf > 1 ? st->max_buf : 1;
  const bool shared = st->n_groups == 1, bf = st->dtype == ARTAB_BF16;

  const int variant = spc <= 1 ? 0 : spc <= 2 ? 1 : spc <= 4 ? 2 : 3;   // 2, 4, 8, 16 rows
  static const double kChain[4] = {1, 1.2, 2.0, 2.6}, kKeys[4] = {4.4e-3, 5.2e-3, 8.3e-3, 28e-3};
  double one = (5.7 + 0.036 * D) * (variant == 3 && !shared ? 3.5 : kChain[variant]) + 5 / L;
  one += H / C * head * keys * (shared ? kKeys[variant] : 4.8e-3 * spc);
  one += (shared ? 1 : B) * D * keys * 8 / 1.3e6 / targets;

  double each = (chain_on_tc(m, st) ? 7 + 0.099 * D : 8 + 0.35 * D) + 21 / L;
  const double bytes = B * D * keys * (bf ? 6 : 8);                     // own contexts
  if (ctx_attn_tc_supported(st->dtype, m->head_dim)) {
    each += shared ? 0.86e-3 * keys : 0.012 * B * H + bytes / 3.6e6;
  } else {
    const int rows = 2 * st->n_streams, tiles = (st->n_ctx + 63) / 64;
    const double walk = keys / (tiles < 16 ? tiles : 16) * head * (rows <= 16 ? 0.022 : rows <= 32 ? 0.027 : 0.054);
    const double work = shared ? rows * keys * D * 4 / 22e6 : bytes / 1.1e6;
    each += shared && walk > work ? walk : work;
    if (bf) each += (shared ? walk : 0.012 * B * H) + 8.9 * (keys < 1000 ? keys / 1000 : 1);
  }
  return one < each;
}

bool seq_plan(const artab_model* m, const artab_state* st, SeqPlan& p, SeqArgs& a) {
  const int D = m->d_model, DH = m->head_dim, H = m->n_heads;
  if (m->seq_ranks <= 0 || m->n_layers > kSeqMaxLayers || m->n_comp > 32) return false;
  const int C = largest_divisor(H, 8);
  // a CTA of its own has no cluster to st.async into: the one launch of this kernel without a cluster
  // dimension (one head) ended in an illegal instruction
  if (C < 2) return false;
  if (C != m->seq_ranks || !(D == 64 || D == 128 || D == 192) || !(DH == 16 || DH == 32 || DH == 64)) return false;
  const int DS = D / C, HS = m->d_ff / C, NB = (3 * m->n_comp + 15) & ~15;
  if (D % C || m->d_ff % C || DS % 16 || HS % 32 || HS > 192 || 3 * DS > 192) return false;
  // streams per cluster: as few as one wave of clusters needs, at most what the variants hold
  const int most = kMaxRowsPerCluster / 2;
  static thread_local int clusters[9][kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  int& fit = clusters[C][dev];
  if (!fit) fit = seq_simt_max_clusters(C, kSmemMax);
  if (fit <= 0) return false;
  // One wave: a second one doubles the time, while the launch-per-layer path hardly notices (fp32, 512 context
  // rows, 8 targets, d_model 128, 6 layers: 2.3 against 3.4 ms at 128 streams, 4.9 against 3.7 at 512, 16.5 against
  // 6.6 at 2048).
  if (st->n_streams > fit * most) return false;
  // the re-tiled copy of the context is as large as its fp32 cache: not where that is a good part of the memory
  if (context_bytes(m, st) > kWorkspaceMax) return false;
  const int spc = (st->n_streams + fit - 1) / fit;
  if (!faster_in_one_launch(m, st, C, spc)) return false;
  const int R = spc <= 1 ? 2 : spc <= 2 ? 4 : spc <= 4 ? 8 : kMaxRowsPerCluster;
  const Areas ar = areas_of(m, C, R);
  const size_t fixed = kSeqBarBytes + 4 * ((size_t)ar.red + ar.area);
  if (fixed + 4 * kSeqSlotBytes > kSmemMax) return false;
  size_t vec = 4 * ((size_t)m->n_layers * (7 * D + HS) + 2 * D + HS);
  if (fixed + vec + 6 * kSeqSlotBytes > kSmemMax) vec = 0;   // a deep ring matters more
  int slots = (int)((kSmemMax - fixed - vec) / kSeqSlotBytes);
  if (slots > kSeqMaxSlots) slots = kSeqMaxSlots;
  p.C = C;
  p.spc = spc;
  p.rows = R;
  p.n_slots = slots;
  p.smem = fixed + vec + (size_t)slots * kSeqSlotBytes;
  p.grid = (st->n_streams + spc - 1) / spc * C;
  a.mat[SEQ_DS] = mat_of(D, DS);
  a.mat[SEQ_QKV] = mat_of(D, 3 * DS);
  a.mat[SEQ_W1] = mat_of(D, HS);
  a.mat[SEQ_W2] = mat_of(HS, D);
  a.mat[SEQ_WB] = mat_of(HS, NB);
  a.hc = H / C;
  a.DS = DS;
  a.HS = HS;
  a.NB = NB;
  a.C = C;
  a.spc = spc;
  a.n_slots = slots;
  a.off_red = kSeqBarBytes + slots * kSeqSlotBytes;
  a.off_areas = a.off_red + 4 * ar.red;
  a.vec_smem = vec ? a.off_areas + 4 * ar.area : 0;
  a.mlp_direct = ar.direct;
  a.n_ctx_tiles = (st->n_ctx + 31) / 32;
  const int fits = kSeqSlotBytes / (64 * DH * 4);
  const int want = (a.n_ctx_tiles + kSeqWarps - 1) / kSeqWarps;  // every warp a slab while there are tiles enough
  a.tiles_per_slab = want < 1 ? 1 : want > fits ? fits : want;
  return true;
}

}  // namespace

bool seq_applicable(const artab_model* m, const artab_state* st) {
  SeqPlan p;
  SeqArgs a;
  return seq_plan(m, st, p, a);
}
size_t seq_workspace_bytes(const artab_model* m, const artab_state* st) { return context_bytes(m, st); }

int launch_seq(const artab_model* m, const artab_state* st, const SeqCall& c, cudaStream_t s) {
  SeqPlan p;
  SeqArgs a;
  memset(&a, 0, sizeof(a));
  ARTAB_REQUIRE(seq_plan(m, st, p, a), ARTAB_EINVAL, "decode_sequence: not available for this model");
  ARTAB_REQUIRE(m->seq_w, ARTAB_EINVAL, "decode_sequence: the weight streams (seq_w) are missing");
  ARTAB_REQUIRE(c.workspace_bytes >= context_bytes(m, st), ARTAB_ECAPACITY, "decode_sequence: workspace too small");
  const bool bf = st->dtype == ARTAB_BF16;
  if (c.t0 == 0) {  // first part of a sequence: the context is new
    const dim3 grid(a.n_ctx_tiles, m->n_heads, m->n_layers * st->n_groups);
    prof_begin(PROF_APPEND, s);
    cudaError_t e;
    if (bf)
      e = launch_dependent(retile_kernel<__nv_bfloat16>, grid, dim3(256), 0, s, (const __nv_bfloat16*)st->k_ctx,
                           (const __nv_bfloat16*)st->v_ctx, (float4*)c.workspace, m->head_dim, st->n_ctx, st->n_ctx_pad, 1);
    else
      e = launch_dependent(retile_kernel<float>, grid, dim3(256), 0, s, (const float*)st->k_ctx, (const float*)st->v_ctx,
                           (float4*)c.workspace, m->head_dim, st->n_ctx, st->n_ctx_pad, 0);
    prof_end(s);
    ARTAB_REQUIRE(e == cudaSuccess, ARTAB_ELAUNCH, "retile_kernel: %s", cudaGetErrorString(e));
    count_launch();
  }
  a.D = m->d_model;
  a.L = m->n_layers;
  a.H = m->n_heads;
  a.n_comp = m->n_comp;
  a.S_ar = m->n_ar_tokens;
  a.B = st->n_streams;
  a.G = st->n_groups;
  a.n_ctx = st->n_ctx;
  a.max_buf = st->max_buf;
  a.wx = m->wx;
  a.bx = m->bx;
  a.wy = m->wy;
  a.by = m->by;
  a.marker = m->marker;
  a.ar_tokens = m->ar_tokens;
  a.bb = m->bb;
  a.mean_bias = m->mean_bias;
  a.std_bias = m->std_bias;
  a.weight_bias = m->weight_bias;
  a.weights = reinterpret_cast<const uint8_t*>(m->seq_w);
  a.rank_bytes = (size_t)m->seq_rank_bytes;
  a.vec_off = (size_t)m->seq_vec_off;
  a.ctx = c.workspace;
  a.kv_buf = st->kv_buf;
  a.xt = c.xt;
  a.xt_stride = c.xt_stride;
  a.F = c.n_feat;
  a.Nt = c.n_targets;
  a.t0 = c.t0;
  a.t1 = c.t1;
  a.samples = c.samples;
  a.expo = c.expo;
  a.normal = c.normal;
  a.logdens = c.logdens;
  a.comp = c.comp;
  a.status = st->status;
  a.wait_cycles = debug_wait_cycles() > 0 ? debug_wait_cycles() : kDefaultWaitCycles;
  a.scale_log2e = kLog2e / sqrtf((float)m->head_dim);
  prof_begin(PROF_DENSE, s);
  int rc;
  switch (m->head_dim) {
    case 16: rc = bf ? launch_seq_bf16_16(a, p, s) : launch_seq_f32_16(a, p, s); break;
    case 32: rc = bf ? launch_seq_bf16_32(a, p, s) : launch_seq_f32_32(a, p, s); break;
    default: rc = bf ? launch_seq_bf16_64(a, p, s) : launch_seq_f32_64(a, p, s); break;
  }
  prof_end(s);
  if (rc) return rc;
  count_launch();
  return check_launch("seq_simt_kernel");
}

}  // namespace artab
