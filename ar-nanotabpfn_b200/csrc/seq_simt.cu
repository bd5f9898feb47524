// One translation unit per (cache type, head size): the build compiles this file once for each pair with
// ARTAB_SEQ_BF16 = 0 | 1 and ARTAB_SEQ_DH = 16 | 32 | 64.
#include "seq_simt.cuh"

#define ARTAB_CAT_(a, b) a##b
#define ARTAB_CAT(a, b) ARTAB_CAT_(a, b)

namespace artab {
#if ARTAB_SEQ_BF16
int ARTAB_CAT(launch_seq_bf16_, ARTAB_SEQ_DH)(const SeqArgs& a, const SeqPlan& p, cudaStream_t s) {
  return launch_seq_dh<__nv_bfloat16, ARTAB_SEQ_DH>(a, p, s);
}
#else
int ARTAB_CAT(launch_seq_f32_, ARTAB_SEQ_DH)(const SeqArgs& a, const SeqPlan& p, cudaStream_t s) {
  return launch_seq_dh<float, ARTAB_SEQ_DH>(a, p, s);
}
#if ARTAB_SEQ_DH == 32
int seq_simt_max_clusters(int C, size_t smem) { return seq_max_clusters<float>(C, smem); }
#endif
#endif
}  // namespace artab

#ifdef ARTAB_TIMELINE
extern "C" __attribute__((visibility("default"))) int ARTAB_CAT(ARTAB_CAT(artab_debug_seq_, ARTAB_SEQ_BF16), ARTAB_CAT(_, ARTAB_SEQ_DH))(long long* dst) {
  return (int)cudaMemcpyFromSymbol(dst, artab::g_seq_tl, sizeof(artab::g_seq_tl));
}
#endif
