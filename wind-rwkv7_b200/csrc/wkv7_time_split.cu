// Forward of few long chains with the sequence cut into segments that run in parallel (bf16, tcgen05 forward).
//
// Over a segment the state goes S -> S M + R with M and R independent of where it starts.  Pass 1 runs the segments from the zero
// state (end state R) and from the identity with v = 0 (end state M); the start states follow by S_{j+1} = S_j M_j + R_j; pass 2 is the
// ordinary forward of the segments from there.  With one sequence, segment 0 starts from the given state in pass 1 and is finished
// then, and the last segment's R and M are not needed: 3 n - 4 segments are walked, not 3 n.
// Bound by the forward kernel; what lies between the passes is two small kernels.  65536 steps of 12 heads, n = 16: 1120 -> 900 us
// (before: fills and copies of zeros and identities, 2 (n - 1) launches for the start states at 9 us a step).
#include <cuda_runtime.h>

#include "wkv7_kernels.h"

namespace wkv7 {
namespace {

constexpr int NN = N * N;

// init[b][j][h]: s0 (or zeros) for j = 0, zeros for the rest; eye: identities.  One float4 per thread and buffer.
__global__ void __launch_bounds__(256) split_init_kernel(const float* s0, float* init, float* eye, int nseg, long long H, long long total4) {
    const long long i = blockIdx.x * 256LL + threadIdx.x;
    if (i >= total4) return;
    const long long chain = i / (NN / 4), b = chain / (nseg * H), j = chain / H % nseg, h = chain % H;
    const int e = (int)(i % (NN / 4)) * 4, row = e / N, col = e % N;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j == 0 && s0) v = reinterpret_cast<const float4*>(s0)[(b * H + h) * (NN / 4) + i % (NN / 4)];
    reinterpret_cast<float4*>(init)[i] = v;
    reinterpret_cast<float4*>(eye)[i] = make_float4(row == col, row == col + 1, row == col + 2, row == col + 3);
}

// start[b][j+1][h] = start[b][j][h] M[b][j][h] + R[b][j][h] from start[b][1] = R[b][0] on.  A CTA carries 16 rows of one chain's state
// (rows are independent), a thread one row's 4 adjacent columns; M comes through shared memory, the next one requested while this one
// is used.  Plain fp32 products.  Bound by the latency of its steps, 1.8 us each.
__global__ void __launch_bounds__(256) split_starts_kernel(const float* R, const float* M, float* start, int nseg, long long H) {
    __shared__ __align__(16) float m[2][NN], s[2][16][N];
    const int tid = threadIdx.x, r = tid >> 4, c = (tid & 15) * 4;
    const long long b = blockIdx.x / H, h = blockIdx.x % H;
    auto at = [&](int j) { return ((b * nseg + j) * H + h) * NN; };
    const long long mine = (16 * blockIdx.y + r) * N + c;
    auto fetch = [&](int j) {
        if (j < nseg - 1)
            for (int i = tid; i < NN / 4; i += 256) cp_async16(&m[j & 1][4 * i], M + at(j) + 4 * i);
        cp_async_commit();
    };
    fetch(1);
    float4 S = *reinterpret_cast<const float4*>(R + at(0) + mine);
    for (int j = 1; j < nseg; ++j) {
        *reinterpret_cast<float4*>(start + at(j) + mine) = S;
        if (j == nseg - 1) break;
        float4 o = *reinterpret_cast<const float4*>(R + at(j) + mine);
        *reinterpret_cast<float4*>(&s[j & 1][r][c]) = S;
        cp_async_wait<0>();
        __syncthreads();  // everyone is past the other buffers, too
        fetch(j + 1);
        const float *row = s[j & 1][r], *mat = m[j & 1] + c;
#pragma unroll 16
        for (int k = 0; k < N; ++k) {
            const float x = row[k];
            const float4 y = *reinterpret_cast<const float4*>(mat + k * N);
            o.x = fmaf(x, y.x, o.x); o.y = fmaf(x, y.y, o.y); o.z = fmaf(x, y.z, o.z); o.w = fmaf(x, y.w, o.w);
        }
        S = o;
    }
    cp_async_wait<0>();
}

}  // namespace

size_t time_split_workspace_bytes(long long B, long long H, int nseg) { return WORK_FLAG_BYTES + 4 * (size_t)(B * nseg * H) * NN * sizeof(float); }

// p: the whole sequences, p.st.b == p.T * p.st.t, p.T % nseg == 0, p.flags: the workspace
int launch_fwd_time_split(const FwdParams& p, int nseg, int groups, cudaStream_t stream) {
    const long long chains = p.B * nseg * p.H, Ts = p.T / nseg;
    float* init = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p.flags) + WORK_FLAG_BYTES);
    float *R = init + chains * NN, *eye = R + chains * NN, *M = eye + chains * NN;
    const long long total4 = chains * (NN / 4);
    split_init_kernel<<<(unsigned)((total4 + 255) / 256), 256, 0, stream>>>(p.s0, init, eye, nseg, p.H, total4);
    if (cudaGetLastError() != cudaSuccess) return kLaunchFailed;
    // segments [from, to) as batch entries
    auto run = [&](int from, long long to, bool zero_v, const float* s0, float* sT) {
        if (from >= to) return (int)kOk;
        FwdParams q = p;
        const long long off = from * Ts * p.st.t * 2, st = from * p.H * NN;
        auto shift = [&](const void* x) { return reinterpret_cast<const unsigned char*>(x) + off; };
        q.r = shift(p.r); q.w = shift(p.w); q.k = shift(p.k); q.a = shift(p.a); q.b = shift(p.b);
        q.v = zero_v ? nullptr : shift(p.v);
        q.y = const_cast<unsigned char*>(shift(p.y));
        q.s0 = s0 + st; q.sT = sT + st;
        q.B = to - from; q.T = Ts; q.st.b = Ts * p.st.t;
        return launch_fwd_tc(q, groups, false, stream);
    };
    const bool one = p.B == 1;
    const int first = one ? 1 : 0;
    const long long last = one ? nseg - 1 : p.B * nseg;
    int rc;
    if ((rc = run(0, last, false, init, R)) != kOk) return rc;      // (y of a later segment is overwritten in pass 2)
    if ((rc = run(first, last, true, eye, M)) != kOk) return rc;
    split_starts_kernel<<<dim3((unsigned)(p.B * p.H), 4), 256, 0, stream>>>(R, M, init, nseg, p.H);
    if (cudaGetLastError() != cudaSuccess) return kLaunchFailed;
    if ((rc = run(first, p.B * nseg, false, init, R)) != kOk) return rc;
    for (long long b = 0; b < p.B; ++b)
        if (p.sT && cudaMemcpyAsync(p.sT + b * p.H * NN, R + (b * nseg + nseg - 1) * p.H * NN, p.H * NN * sizeof(float), cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
            return kLaunchFailed;
    return kOk;
}

}  // namespace wkv7
