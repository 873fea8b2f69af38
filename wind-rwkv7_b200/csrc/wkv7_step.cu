// WKV7 decode step: the recurrence itself, one time step at a time, for generation after a prefill.
//
//     S <- S diag(exp(-exp(w_t))) + (S a_t) b_t^T + v_t k_t^T ,   y_t = S r_t
//
// (the loop body of the reference's naive recurrence, wind_rwkv/rwkv7/time_mixer.py:13-15; the
// reference has no kernel for it: its chunked kernels need T % 16 == 0, rwkv7_attn.py:22).  The
// state uses the fp32 [B,H,N,N] format of wkv7_fwd's s0 / sT, so a prefill's final state is this
// kernel's input.  Meant for T of one to a few steps: no chunking, no tensor cores, no checkpoints;
// plain fp32 FMAs, exact to fp32 rounding.
//
// One CTA of 256 threads per (batch, head) chain.  Thread (i, q) = (tid / 4, tid % 4) keeps 16 elements of state row i in
// registers for all T steps: columns 4q..4q+3 of each 16, so that the row's four threads read and write whole 64-byte pieces and
// fetch their share of a, b, k, r and the decays from shared memory without bank conflicts.  The two row contractions (S a and
// S r) are 16 FMAs per thread and two shuffles.  The step's vectors are loaded, converted and (the decays) exponentiated once per
// CTA, not by each of the 64 rows (8192 exponentials per chain).
// What is left is the state traffic: 2 * 16 KB per chain and call, all loads of it in flight before the first barrier, six CTAs an
// SM (40 registers; at 76 registers and three CTAs 54 us): 6400 chains 54 -> 44.6 us; the same kernel without the arithmetic 36 us.
#include "wkv7_kernels.h"

namespace wkv7 {

template <typename IoT>
__global__ void __launch_bounds__(256, 6) wkv7_step_kernel(StepParams p) {
    __shared__ __align__(16) float vec[2][6][N];  // decay, a, b, k, r, v of one step; two buffers: one barrier per step
    const int tid = threadIdx.x, i = tid >> 2, q = tid & 3;
    const long long bh = blockIdx.x;
    const long long bi = bh / p.H, hi = bh % p.H;
    const long long base = bi * p.st.b + hi * p.st.h + (tid & 63);
    // this thread's elements of the step's vectors: one of w, a, b, k and (tid < 128) one of r, v
    const int part = tid >> 6;
    const IoT* src0 = (const IoT*)(part == 0 ? p.w : part == 1 ? p.a : part == 2 ? p.b : p.k) + base;
    const IoT* src1 = (const IoT*)(part == 0 ? p.r : p.v) + base;
    IoT x0 = src0[0], x1 = src0[0];
    if (part < 2) x1 = src1[0];
    float S[16];
    const long long at = bh * N * N + i * N + 4 * q;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.s0) s = *reinterpret_cast<const float4*>(p.s0 + at + 16 * j);
        S[4 * j] = s.x; S[4 * j + 1] = s.y; S[4 * j + 2] = s.z; S[4 * j + 3] = s.w;
    }
    for (long long t = 0; t < p.T; ++t) {
        float (*u)[N] = vec[t & 1];
        const float f0 = to_f32<IoT>(x0);
        u[part][tid & 63] = part == 0 ? expf(-expf(f0)) : f0;
        if (part < 2) u[4 + part][tid & 63] = to_f32<IoT>(x1);
        __syncthreads();
        if (t + 1 < p.T) {
            x0 = src0[(t + 1) * p.st.t];
            if (part < 2) x1 = src1[(t + 1) * p.st.t];
        }
        float sa = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 a = *reinterpret_cast<const float4*>(&u[1][16 * j + 4 * q]);
            sa = fmaf(S[4 * j], a.x, sa); sa = fmaf(S[4 * j + 1], a.y, sa);
            sa = fmaf(S[4 * j + 2], a.z, sa); sa = fmaf(S[4 * j + 3], a.w, sa);
        }
        sa += __shfl_xor_sync(0xffffffffu, sa, 1);
        sa += __shfl_xor_sync(0xffffffffu, sa, 2);
        const float v = u[5][i];
        float y = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 d = *reinterpret_cast<const float4*>(&u[0][16 * j + 4 * q]), b = *reinterpret_cast<const float4*>(&u[2][16 * j + 4 * q]);
            const float4 k = *reinterpret_cast<const float4*>(&u[3][16 * j + 4 * q]), r = *reinterpret_cast<const float4*>(&u[4][16 * j + 4 * q]);
            S[4 * j] = fmaf(S[4 * j], d.x, fmaf(sa, b.x, v * k.x)); y = fmaf(S[4 * j], r.x, y);
            S[4 * j + 1] = fmaf(S[4 * j + 1], d.y, fmaf(sa, b.y, v * k.y)); y = fmaf(S[4 * j + 1], r.y, y);
            S[4 * j + 2] = fmaf(S[4 * j + 2], d.z, fmaf(sa, b.z, v * k.z)); y = fmaf(S[4 * j + 2], r.z, y);
            S[4 * j + 3] = fmaf(S[4 * j + 3], d.w, fmaf(sa, b.w, v * k.w)); y = fmaf(S[4 * j + 3], r.w, y);
        }
        y += __shfl_xor_sync(0xffffffffu, y, 1);
        y += __shfl_xor_sync(0xffffffffu, y, 2);
        if (q == 0) ((IoT*)p.y)[base - (tid & 63) + t * p.st.t + i] = from_f32<IoT>(y);
    }
    if (p.sT) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(p.sT + at + 16 * j) = make_float4(S[4 * j], S[4 * j + 1], S[4 * j + 2], S[4 * j + 3]);
    }
}

int launch_step(const StepParams& p, int io_dtype, cudaStream_t stream) {
    if (io_dtype == 0) wkv7_step_kernel<__nv_bfloat16><<<(unsigned)(p.B * p.H), 256, 0, stream>>>(p);
    else wkv7_step_kernel<float><<<(unsigned)(p.B * p.H), 256, 0, stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

}  // namespace wkv7
