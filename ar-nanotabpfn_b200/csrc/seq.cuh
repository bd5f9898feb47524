// Whole-sequence decode: one launch walks every target of a sampling job.
//
// Sample streams are independent given the context, so nothing in the decode loop needs a grid-wide
// step: a thread-block cluster owns a few streams and takes them through every layer of every target
// on its own.  One CTA of the cluster per attention head (or per group of heads): the projections are
// split by columns, attention stays inside a CTA, and what the next matrix needs of the other CTAs
// crosses through distributed shared memory.
#pragma once
#include "common.cuh"

namespace artab {

constexpr int kSeqMaxLayers = 24;
// compute warps; one more streams weights.  13 warps are four per scheduler: 128 registers per thread
constexpr int kSeqWarps = 12, kSeqThreads = kSeqWarps * 32;
constexpr int kSeqSlotBytes = 16384;                         // ring slot of the weight / context stream
constexpr int kSeqMaxSlots = 12;
constexpr int kSeqBarBytes = 1024;                           // barriers and the abort flag, at offset 0; then the ring

constexpr int kSeqSlabUnits = 8;      // weight units (32 k x 16 columns of fp32, 2 KB) in one ring slot
constexpr int kSeqPitch = 196;         // floats between the rows of an activation array: d_model, slices <= 192
constexpr int kSeqBufferParts = 4;     // partial results of the private keys of a stream

// A matrix slice [K][N] as the GEMM walks it: N / 16 column tiles, K / 32 k blocks, kw warps per column tile.
struct SeqMat {
  int tiles, octs, kw;
};
enum SeqMatKind : int { SEQ_DS = 0, SEQ_QKV = 1, SEQ_W1 = 2, SEQ_W2 = 3, SEQ_WB = 4, SEQ_MATS = 5 };

struct SeqArgs {
  SeqMat mat[SEQ_MATS];                   // fold / out-projection, Q|K|V, W1 (and head.0), W2, head.2
  int D, L, H, C, n_comp, S_ar;           // C: CTAs per cluster, a divisor of H
  int hc, DS, HS, NB;                     // per CTA: heads, columns of D, columns of Dff; head outputs padded to 16
  int B, G, n_ctx, n_ctx_tiles, max_buf;  // G: 1 (shared context) or B
  int spc;                                // streams per cluster
  const float *wx, *bx, *wy, *by, *marker, *ar_tokens;
  const float *bb, *mean_bias, *std_bias, *weight_bias;
  const uint8_t* weights;   // [C] weight streams, see _pack.py
  size_t rank_bytes, vec_off;  // bytes of one of them; offset of its LayerNorm / bias vectors
  const void* ctx;          // re-tiled context, see the re-tiling kernels
  void* kv_buf;             // [L][B][H][T][2][Dh]
  const float* xt;          // target features: stream b at xt + b * xt_stride, [Nt][F]
  size_t xt_stride;
  int F, Nt, t0, t1;        // targets [t0, t1) of Nt are decoded by this launch
  float* samples;           // [B][Nt]
  const float *expo, *normal;  // [Nt][B][K], [Nt][B]
  float* logdens;           // [B][Nt] or null
  int32_t* comp;            // [B][Nt] or null
  int32_t* status;
  long long wait_cycles;
  float scale_log2e;
  // shared-memory plan (bytes from the start of dynamic shared memory)
  int n_slots, off_red, off_areas, vec_smem;  // vec_smem: 0 when the vectors stay in global memory
  int mlp_direct;           // second MLP matrix: partial sums to every CTA at once instead of reduce, then gather
  int tiles_per_slab;
};

struct SeqPlan {
  int C, spc, rows, n_slots;   // rows: the kernel variant (template R)
  size_t smem;
  int grid;
};

int launch_seq_f32_16(const SeqArgs& a, const SeqPlan& p, cudaStream_t s);  // cache type, head size
int launch_seq_f32_32(const SeqArgs& a, const SeqPlan& p, cudaStream_t s);
int launch_seq_f32_64(const SeqArgs& a, const SeqPlan& p, cudaStream_t s);
int launch_seq_bf16_16(const SeqArgs& a, const SeqPlan& p, cudaStream_t s);
int launch_seq_bf16_32(const SeqArgs& a, const SeqPlan& p, cudaStream_t s);
int launch_seq_bf16_64(const SeqArgs& a, const SeqPlan& p, cudaStream_t s);
int seq_simt_max_clusters(int C, size_t smem);

// one decode_sequence call
struct SeqCall {
  const float* xt;
  size_t xt_stride;
  int n_feat, n_targets, t0, t1;
  float* samples;
  const float *expo, *normal;
  float* logdens;
  int32_t* comp;
  void* workspace;
  size_t workspace_bytes;
};
bool seq_applicable(const artab_model* m, const artab_state* st);
size_t seq_workspace_bytes(const artab_model* m, const artab_state* st);
int launch_seq(const artab_model* m, const artab_state* st, const SeqCall& c, cudaStream_t s);

}  // namespace artab
