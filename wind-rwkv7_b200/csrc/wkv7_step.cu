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
// SM (40 registers; at 76 registers and three CTAs 1.2 times as long).  Many chains, up to eight steps: wkv7_step_ring_kernel below.
// Both start while the kernel ahead of them drains (stream_order): steps in a row, T = 1, 6400 chains 37.0 -> 35.8 us, 3200 20.5 -> 18.0, 1280 10.3 ->
// 8.9, 768 8.2 -> 6.4, and the smallest calls, whose time is the host's, 6.1 -> 5.6.  (The next but one state on its way, too: 10240 chains 56.3 -> 59.4.)
#include "wkv7_kernels.h"

namespace wkv7 {

// One step: thread (i, q)'s 16 elements of state row i, the step's vectors u.  Returns y_i (in all of the row's threads).
__device__ __forceinline__ float step_row(float (&S)[16], const float (*u)[N], int i, int q) {
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
    return y + __shfl_xor_sync(0xffffffffu, y, 2);
}

template <typename IoT>
__global__ void __launch_bounds__(256, 6) wkv7_step_kernel(StepParams p) {
    stream_order();
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
        const float y = step_row(S, u, i, q);
        if (q == 0) ((IoT*)p.y)[base - (tid & 63) + t * p.st.t + i] = from_f32<IoT>(y);
    }
    if (p.sT) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(p.sT + at + 16 * j) = make_float4(S[4 * j], S[4 * j + 1], S[4 * j + 2], S[4 * j + 3]);
    }
}

// More chains than resident CTAs: each CTA walks several, and the next one's state comes by a bulk copy while this one is worked and stored
// (a CTA per chain leaves the memory idle between its last store and its successor's first load).  Four CTAs an SM (five or six spill: 39 us): 6400
// chains 44.0 -> 38.5 us, 10240 65.6 -> 57.8, 3200 25.1 -> 21.0, 1280 11.4 -> 10.8, 768 9.5 -> 9.9, hence the line at two chains a CTA.
// More steps a call: what counts is more and more the steps' latency, which six CTAs an SM hide better than four, and how full the last round of
// CTAs is.  A CTA per chain / here, us, at T = 4: 1280 chains 25.8 / 22.7, 1600 28.9 / 28.7, 3200 51.2 / 47.3, 6400 92.8 / 90.2; T = 8: 1280
// 41.1 / 37.0, 1600 45.3 / 47.3, 2688 73.9 / 69.9, 6400 161.2 / 162.1; T = 12: 1280 56.1 / 51.4, 1600 61.6 / 67.6, 3200 118.9 / 120.4, 6400
// 230.8 / 233.9; T = 16: 10240 473 / 479; hence the line at eight steps.
constexpr int RING_PER_SM = 4, RING_STEPS = 8;
template <typename IoT>
__global__ void __launch_bounds__(256, RING_PER_SM) wkv7_step_ring_kernel(StepParams p, int chains) {
    __shared__ __align__(128) float st[N * N];
    __shared__ __align__(16) float vec[2][6][N];
    __shared__ uint64_t full;
    __shared__ volatile int abort, zero;
    const int tid = threadIdx.x, i = tid >> 2, q = tid & 3, part = tid >> 6, H = (int)p.H;
    const IoT* const in0 = (const IoT*)(part == 0 ? p.w : part == 1 ? p.a : part == 2 ? p.b : p.k) + (tid & 63);
    const IoT* const in1 = (const IoT*)(part == 0 ? p.r : p.v) + (tid & 63);
    auto offset = [&](int bh) { const int b = (int)((unsigned)bh / (unsigned)H); return b * p.st.b + (bh - b * H) * p.st.h; };
    auto load = [&](int bh) {  // one thread
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full)), "n"(N * N * 4) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(st)), "l"(p.s0 + (long long)bh * N * N), "n"(N * N * 4), "r"(smem_u32(&full)) : "memory");
    };
    int bh = blockIdx.x, loads = 0;
    if (tid == 0) {
        mbar_init(&full, 1);
        abort = zero = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    stream_order();
    if (tid == 0 && p.s0) { load(bh); ++loads; }
    long long base = offset(bh);
    IoT x0 = in0[base], x1 = x0;
    if (part < 2) x1 = in1[base];
    __syncthreads();
    unsigned step = 0;
    for (int n = 0; bh < chains; ++n) {
        const int next = bh + (int)gridDim.x;
        const long long next_base = next < chains ? offset(next) : 0;
        float S[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) S[j] = 0.f;
        if (p.s0) {
            mbar_wait_bounded<false>(&full, n & 1, &abort, p.status);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 s = *reinterpret_cast<const float4*>(st + i * N + 16 * j + 4 * q);
                S[4 * j] = s.x; S[4 * j + 1] = s.y; S[4 * j + 2] = s.z; S[4 * j + 3] = s.w;
            }
        }
        IoT* const y = (IoT*)p.y + base + i;
        for (long long t = 0; t < p.T; ++t, ++step) {
            float (*u)[N] = vec[step & 1];
            const float f0 = to_f32<IoT>(x0);
            u[part][tid & 63] = part == 0 ? expf(-expf(f0)) : f0;
            if (part < 2) u[4 + part][tid & 63] = to_f32<IoT>(x1);
            __syncthreads();
            if (t == 0 && tid == 0 && p.s0 && next < chains && !abort) {  // everyone has read the state
                fence_async_smem();
                load(next);
                ++loads;
            }
            const bool same = t + 1 < p.T;
            if (same || next < chains) {
                const long long at = same ? base + (t + 1) * p.st.t : next_base;
                x0 = in0[at];
                if (part < 2) x1 = in1[at];
            }
            const float yt = step_row(S, u, i, q);
            if (q == 0) y[t * p.st.t] = from_f32<IoT>(yt);
        }
        if (p.sT) {
            float* out = p.sT + (long long)bh * N * N + i * N + 4 * q;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(out + 16 * j) = make_float4(S[4 * j], S[4 * j + 1], S[4 * j + 2], S[4 * j + 3]);
        }
        bh = next;
        base = next_base;
    }
    if (tid == 0) mbar_landed(&full, loads, &zero, p.status);  // shared memory must outlive the loads, also where a wait has given up
}

template <typename IoT> static int launch_step_t(const StepParams& p, cudaStream_t stream) {
    const long long chains = p.B * p.H;
    // (the smallest calls, whose time is the host's, do not ask for the number of SMs)
    const long long resident = chains > 512 ? (long long)RING_PER_SM * sm_count() : chains;
    if (chains > 2 * resident && chains <= 0x3fffffff && p.T <= RING_STEPS && p.status) return launch(wkv7_step_ring_kernel<IoT>, dim3((unsigned)resident), 256, 0, stream, p, (int)chains) ? kOk : kLaunchFailed;
    return launch(wkv7_step_kernel<IoT>, dim3((unsigned)chains), 256, 0, stream, p) ? kOk : kLaunchFailed;
}
int launch_step(const StepParams& p, int io_dtype, cudaStream_t stream) {
    return io_dtype == 0 ? launch_step_t<__nv_bfloat16>(p, stream) : launch_step_t<float>(p, stream);
}

}  // namespace wkv7
