// Internal launcher interface between the C ABI (capi.cu) and the kernel translation units.
#pragma once
#include <cuda.h>
#include <utility>
#include "wkv7_common.cuh"

namespace wkv7 {

// Launches a kernel that calls stream_wait(): it may start while the one ahead of it in the stream drains.  For kernels that follow others
// closely.  Without / with this alone, us: B32 T1024 C768, ddlerp forward and backward 307 / 288, expand_loras 277 / 269, time mixer 2104 /
// 2073; layer of 515 rows, C = 2048, forward 149 / 134; attn forward and backward, B3 T1003 H16 170 / 163, fp32 B8 T512 H12 289 / 285.  (Not so
// launched, since it did not pay: the fp32 forward, B8 T512 H12 287 -> 293 us, and the sums between the two walks of time_split, 497 -> 521.)
template <typename... P, typename... A> inline bool launch(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid; c.blockDim = dim3(threads); c.dynamicSmemBytes = smem; c.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &attr; c.numAttrs = 1;
    if (cudaLaunchKernelEx(&c, kern, std::forward<A>(args)...) == cudaSuccess) return true;
    cudaGetLastError();  // (reported by the status; not left for the caller's next check)
    return false;
}

struct FwdParams {
    const void *r, *w, *k, *v, *a, *b;  // [B,T,H,N], io dtype
    const void* g;                      // attn_ln only
    const float* params;                // attn_ln only: [3, H*N] = ln_weight, ln_bias, bonus
    const float* s0;                    // [B,H,N,N] or null (zeros)
    void* y;                            // [B,T,H,N]
    float* sT;                          // [B,H,N,N] or null
    float* ckpt;                        // [B,H,T/16,CK_FLOATS] checkpoint records (chunk-start state + 4 matrices), or null
    long long B, T, H;
    Strides st;
    float eps;
    int* status;                        // device status word
    unsigned* flags;                    // scratch for cut chains (WorkSplit), or null: every chain is worked by one CTA
    // tcgen05 forward: the chains as affine maps S -> S M + R, R to sT [B,H,N,N] and M to sM, no y.  The batch entries are segments of
    // sequences, nseg of each; R of a sequence's first one starts from s0 [B/nseg,H,N,N] (or null: zeros).  Null: the ordinary forward
    float* sM;
    int nseg;
};

struct BwdParams {
    const void *r, *w, *k, *v, *a, *b, *dy;  // dy: gradient of y (attn) or of the fused output (attn_ln)
    const void* g;           // attn_ln only
    const float* params;     // attn_ln only
    void* dg;                // attn_ln only
    float* dparams;          // attn_ln only: [3, H*N]
    float* dparams_ws;       // attn_ln only: [B, 3, H*N] per-(batch, head) partials
    float eps;
    const float* ckpt;   // written by the forward
    const float* dsT;    // [B,H,N,N] or null (zeros)
    const float* sT;     // final state of the forward; needed only when dsT is given
    void *dr, *dw, *dk, *dv, *da, *db;
    float* ds0;          // or null
    long long B, T, H;
    Strides st;
    int* status;
    unsigned* flags;     // scratch for cut chains (WorkSplit), or null
};

struct StepParams {
    const void *r, *w, *k, *v, *a, *b;  // [B,T,H,N], io dtype
    const float* s0;                    // [B,H,N,N] or null (zeros); may be the same buffer as sT
    void* y;                            // [B,T,H,N]
    float* sT;                          // [B,H,N,N] or null
    long long B, T, H;
    Strides st;
    int* status;                        // device status word
};

// Work split for `chains` chains of `per_chain` chunks with `per_sm` resident CTAs per SM.  Chains are cut only when there are
// more of them than resident CTAs (below that every chain has a CTA to itself and cutting gains nothing).
WorkSplit plan_work(long long chains, long long per_chain, int per_sm, unsigned* flags);
int sm_count();
constexpr size_t WORK_FLAG_BYTES = 4096;  // room for the flags of 1024 CTAs

// tensor map of a bf16 [B,T,H,N] tensor, box = 16 time steps of one head, 128-byte swizzle
bool encode_bthn_map(CUtensorMap* m, void* base, long long B, long long T, long long H, const Strides& st);

int launch_fwd(const FwdParams& p, int io_dtype, bool ln, cudaStream_t stream);
// the recurrence step by step on fp32 FMAs (decode); io_dtype 0 = bf16, otherwise fp32 tensors
int launch_step(const StepParams& p, int io_dtype, cudaStream_t stream);
// tensor maps over the checkpoint records' states and matrices, for the backward kernels' loads (see wkv7_bwd.cu)
bool encode_ckpt_state_map(CUtensorMap* m, const float* ckpt, long long records);
bool encode_ckpt_mats_map(CUtensorMap* m, const float* ckpt, long long records);
int launch_bwd_bf16(const BwdParams& p, bool ln, cudaStream_t stream);
size_t bwd_workspace_bytes(long long B, long long T, long long H, bool ln);  // what launch_bwd wants at p.flags for bf16 tensors
size_t bwd32_workspace_bytes(long long B, long long T, long long H);         // and for fp32 ones, attn
int launch_reduce_dparams(const BwdParams& p, cudaStream_t stream);  // dparams = sum over the batch of dparams_ws
int launch_bwd(const BwdParams& p, int io_dtype, bool ln, cudaStream_t stream);
// tcgen05 forward (bf16 IO; attn, or attn_ln with ln = true).  impl 2, 3, 4: a CTA has 3, 4 or 5 slots, i.e. chunks in flight (attn_ln: always 4); negative:
// the same with operands not rounded to TF32 by their producer (the tensor core truncates them)
int launch_fwd_tc(const FwdParams& p, int impl, bool ln, cudaStream_t stream);
// bf16 forward with the sequences cut into nseg segments each (wkv7_time_split.cu)
size_t time_split_workspace_bytes(long long B, long long H, int nseg);
int launch_fwd_time_split(const FwdParams& p, int nseg, int impl, cudaStream_t stream);
// for each of `count` products C[M,N] = act(A[M,K] W[N,K]^T), bf16, A's rows lda apart, tanh on columns [tanh_from, tanh_to); tcgen05 + TMA (proj_gemm.cu)
constexpr int PROJ_MAX = 6;
int launch_proj_gemm(int count, const void* const* A, const void* const* W, void* const* C, const int64_t* N, const int64_t* K, const int64_t* lda,
                     const int64_t* tanh_from, const int64_t* tanh_to, long long M, int* status, cudaStream_t stream);
// one small CTA running the tcgen05 forward's bounded mbarrier wait on barriers nothing arrives on
int launch_bounded_wait_selftest(long long limit_cycles, int* status, long long* cycles, cudaStream_t stream);

}  // namespace wkv7
