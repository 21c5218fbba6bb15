// ops.cuh - internal launch helpers shared between the op-level entry points and the token schedule.
#pragma once
#include <algorithm>
#include "common.cuh"

#include <type_traits>

// All helpers enqueue on `st` and return cudaGetLastError() state through bn_launch_check by the caller.
namespace bnk {

// Programmatic dependent launch for every kernel of the token schedule: a kernel may be scheduled while its predecessor
// drains, which hides the launch latency, and blocks in its dependency wait (griddepcontrol.wait) until the predecessor is
// complete and its memory visible. Most kernels release their successor before that wait, so a chain of unfinished kernels may
// stand in front of one that has just started. What a kernel may read before its wait is therefore
//   * constants (weights, signs, norm weights), and
//   * words that no kernel of the same pass writes in front of it: the position, and the layer's recurrent state and conv taps,
//     which one kernel of a pass updates, behind its own wait. They were written in an earlier pass, or by the kernel that sets
//     token and position (k_set_cols, k_set_tok_pos), and every pass begins behind a plain launch, a copy or a graph launch,
//     which waits for all that was enqueued before it. Those must stay plain: with this attribute they would be part of the chain.
//     (In a pass whose first launch follows k_set_cols directly that launch is embed_rotate, which waits before it releases.)
//   * the residual, in gdn_step alone: the projection in front of it releases it late (Q2Args::late);
//   * the residual and its norm factor, in k_gdn_core of several sequences: the projections of several columns release their dependents
//     behind their own wait, and the kernel that wrote the factor stands in front of them.
extern bool g_pdl;
template <class... KArgs, class... Args>
inline void launch_as(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
    BN_COUNT(1);
}
template <class... KArgs, class... Args>
inline void launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    launch_as(g_pdl, kernel, grid, block, smem, st, args...);
}
// The same for a grid of at most a few CTAs per SM: as much unused shared memory as keeps them evenly spread. Launched while the
// kernel in front is finishing, small CTAs would otherwise crowd on the first SMs that become free while others stay idle.
// MOST: CTAs per SM up to which it is done.
template <auto K, int MOST = 4, typename... Args>
inline void launch_spread(dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    constexpr int SM = 233472, RESERVED = 1024, MAX_CTA = 232448;         // shared memory of an SM, of it per CTA, a CTA's most
    static const int fixed = [] {                                          // the kernel's static shared memory
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, K) != cudaSuccess) return MAX_CTA;
        cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_CTA - int(fa.sharedSizeBytes));
        return int(fa.sharedSizeBytes);
    }();
    const int per = int((size_t(grid.x) * grid.y * grid.z + 147) / 148), apart = SM / (per + 1) - RESERVED - fixed + 256;
    if (per <= MOST && apart > int(smem)) smem = size_t(apart);
    launch(K, grid, block, smem, st, args...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_sync() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// Several sequences ("columns") in one launch: blockIdx.z is the column; its activations live at the column-0
// pointer + col * arena bytes, its recurrent state, conv taps and KV cache at + col * the respective stream strides.
// The default (no columns) leaves every pointer as it is.
struct Cols {
    int n = 0;
    size_t arena = 0, gdn = 0, conv = 0, kv = 0;
    unsigned z() const { return n > 0 ? unsigned(n) : 1u; }
};
#ifdef __CUDACC__
template <class T> __device__ __forceinline__ T *colp(T *p, size_t bytes) {
    return p ? reinterpret_cast<T *>(reinterpret_cast<char *>(const_cast<typename std::remove_const<T>::type *>(p)) + bytes) : p;
}
#endif

constexpr int Q81_DWORDS = 36;
constexpr int BF_WORDS = 512;
inline size_t act_pack_bytes(int K) { return size_t(K / 128) * (Q81_DWORDS + BF_WORDS) * 4; }

// PTQ1_0 x q8_1 GEMV. out[M] final fp32. scratch: >= ceil(K/512) * M floats.
void gemv_q81(cudaStream_t st, int sm_count, const uint32_t *W, int M, int K, const uint32_t *pack, float *out,
              float *scratch, int32_t *dots);
void act_quant_q81(cudaStream_t st, const float *x, int K, uint32_t *pack);
// the same projection streamed from the native rows without scratch (ptq_stream.cu); W 4-byte aligned
bool ptq_stream_supported(int K);
cudaError_t ptq_stream(cudaStream_t st, int sm_count, const void *W, int M, int K, const uint32_t *pack, float *out);

// y = H(s . x) per `block`-wide chunk, then q8_1 + operand table into pack (pack may be null: rotate only,
// y may be null when only the pack is wanted). n % block == 0, block = power of two in [128, 4096].
void rotate_quant(cudaStream_t st, const float *x, const int32_t *signs, int n, int block, float *y, uint32_t *pack);
// embedding side: y = s . H(x)
// PTQ1_0 row gather: out[K] = dequantised row `tok` (tok read from tok_ptr[0])
// y = signs . H(row tok_ptr[0] of the embedding), Hadamard blocks of `block` values
void embed_rotate(cudaStream_t st, const uint32_t *W, int K, const int *tok_ptr, const int32_t *signs, int block, float *y, Cols cols = {});

void rms_norm(cudaStream_t st, const float *x, const float *w, int rows, int cols, float eps, float *y);
void add_inplace(cudaStream_t st, float *res, const float *d, int n);       // res = d + res
void swiglu(cudaStream_t st, const float *a, const float *b, int n, float *y, Cols cols = {});
void gemv_f32_small(cudaStream_t st, const float *W, int M, int K, const float *x, float *out);

struct GdnDims { int heads, qk_heads, dim; };
void gdn_gates(cudaStream_t st, const float *alpha, const float *beta_raw, const float *dt_bias, const float *ssm_a,
               int n, float *gate, float *beta);
void conv_silu(cudaStream_t st, const float *x, const float *w, float *hist, int channels, float *y);
void l2_norm_rows(cudaStream_t st, const float *x, int rows, float eps, float *y);   // 128-wide rows
void gdn_delta(cudaStream_t st, GdnDims d, const float *q, const float *k, const float *v, const float *gate,
               const float *beta, float *state, float *o);
// fused layer mixer: alpha/beta projections of the normed residual + gates, conv + silu, L2 norms, delta rule,
// per-head RMS * ssm_norm, swiglu(z, .), v-grouped permutation -> y. hist0 / hist1: the two conv-history
// buffers; position parity picks which is read and which is written. hidden <= 16384.
void gdn_core_fused(cudaStream_t st, GdnDims d, int hidden, const float *qkv, const float *conv_w, float *hist0,
                    float *hist1, const int *pos_ptr, const float *x, const float *inv_ptr, const float *norm_w, const float *alpha_w,
                    const float *beta_w, const float *dt_bias, const float *ssm_a, float *state, const float *z,
                    const float *ssm_norm, float eps, float *y, Cols cols = {}, bool alone = false);
// the same fused mixer for one token of one sequence on heads x 4 CTAs (gdn_step.cu). The kernel reads the residual before its
// dependency wait: the launch in front of it must be one that releases its dependents behind its own wait (Q2Args::late).
// alone (both): a plain launch, for a sweep of cores without the projections between them - a core reads the layer's state before
// its wait, and the core in front may be the one that writes it.
struct GdnStep {
    int heads, qk_heads, hidden;
    const float *qkv, *z, *conv_w;
    float *hist0, *hist1;
    const int *pos;
    const float *x, *norm_w, *alpha_w, *beta_w, *dt_bias, *ssm_a;
    float *state;
    const float *ssm_norm;
    float eps, scale;
    float *y;
    int *err;                              // device error word (a bounded wait)
};
void gdn_step(cudaStream_t st, const GdnStep &a, bool alone = false);
cudaError_t launch_wait_selftest_step(cudaStream_t st, int *err);
// the mixer for n <= 32 consecutive positions of one sequence (gdn_seq.cu): column c's activations at + c * stride bytes
struct GdnSeq {
    int heads, qk_heads, hidden;
    const float *qkv, *conv_w;
    float *hist0, *hist1;                  // conv taps by position parity
    const int *pos;                        // position of the first column
    const float *x, *inv, *norm_w, *alpha_w, *beta_w, *dt_bias, *ssm_a;
    float *state;
    float *qk, *v, *eg, *bt, *o;           // working memory per column: normed q and k heads, v, decay, beta, delta-rule output
    float scale;
    size_t stride;
};
void gdn_sequence(cudaStream_t st, const GdnSeq &a, int n, const float *z, const float *ssm_norm, float eps, float *y);
// per-head RMS (no weight) * ssm_norm, swiglu(z, .), v-grouped permutation -> y[heads*dim]
void gdn_out(cudaStream_t st, GdnDims d, const float *o, const float *z, const float *ssm_norm, float eps, float *y);

struct AttnDims { int n_head, n_kv, head_dim, n_rot, cap; float eps, rope_base; int k_mode, v_mode; };
struct KvLayer { void *k_data; uint16_t *k_scale; void *v_data; uint16_t *v_scale; };   // scales null in fp16 mode
// where a query token stands: at ptr[0] (a device word; one per column) or, with ptr null, at `imm`
struct AttnPos {
    const int *ptr;
    int imm;
#ifdef __CUDACC__
    __device__ __forceinline__ int get() const { return ptr ? ptr[0] : imm; }
#endif
};
// norm + rope + fp16 rounding of q, gate split, K/V quantise + insert at the position; tokens > 1 (no columns): that many
// consecutive K / V rows from there, the query at the last of them
void attn_prep(cudaStream_t st, AttnDims a, const float *qg, const float *kin, const float *vin, const float *qn_w,
               const float *kn_w, AttnPos where, KvLayer kv, float *q16f, float *gate, float *esum, Cols cols = {}, int tokens = 1);
// scores -> softmax (fp16-rounded probabilities) -> PV -> sigmoid gate. Scratch buffers sized by cap.
void attn_decode(cudaStream_t st, AttnDims a, const float *q16f, const float *gate, AttnPos where, KvLayer kv,
                 float *score /*[nh][cap]*/, float *p16f /*[nh][cap]*/, float *esum /*[nh][128] partial softmax sums + [nh] row maxima*/,
                 float *pv_part /*[splits][nh][hd]*/, int splits,
                 float *pregate /*[nh][hd] or null*/, float *gated, int *err, Cols cols = {});
// the same in one launch (attn_cluster.cu), without scratch; false: this capacity, or this device, is not for it
bool attn_cluster(cudaStream_t st, AttnDims a, const float *q16f, const float *gate, AttnPos where, KvLayer kv, int splits, float *pregate,
                  float *gated, Cols cols, int *err);
cudaError_t launch_wait_selftest_exchange(cudaStream_t st, int *err);
// cand (optional): per column (value, row0 + index) of the maximum, for an output head whose rows are sharded
void argmax_first(cudaStream_t st, const float *x, int n, int *out_idx, float *scratch_val, int *scratch_idx, Cols cols = {},
                  float *cand = nullptr, int row0 = 0);
// first maximum over n_shards x ncol candidates (value, row), shards in ascending row order
void pick_shards(cudaStream_t st, const float *cands, int n_shards, int ncol, int *out);

// fp32-activation projection (the reference engine's own arithmetic, gemv_ternary.comp): scratch holds
// gemv_f32act_scratch_floats(M, K, n_splits) floats
size_t gemv_f32act_scratch_floats(int M, int K, int n_splits);
void gemv_f32act(cudaStream_t st, const uint8_t *W, int M, int K, const float *x, int n_splits, float *out, float *scratch);

}  // namespace bnk
