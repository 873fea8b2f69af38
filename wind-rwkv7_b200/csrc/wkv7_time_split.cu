// Forward of few long chains with the sequence cut into segments that run in parallel (bf16, tcgen05 forward).
//
// Over a segment the state goes S -> S M + R with M and R independent of where it starts.  Pass 1 walks the segments as such maps
// (wkv7_fwd_tc_kernel, AFF: both in one state of 128 rows); the start states follow by S_{j+1} = S_j M_j + R_j; pass 2 is the
// ordinary forward of the segments from there.  With one sequence the last segment's map is not needed: 2 n - 1 segments are walked
// (before, R and M in passes of their own with an output nobody reads: 3 n - 4).
// Bound by the forward kernel; what lies between the passes is one small kernel.   65536 steps of 12 heads, n = 16: 830 -> 545 us.
#include <cuda_runtime.h>

#include "wkv7_kernels.h"

namespace wkv7 {
namespace {

constexpr int NN = N * N;

// start[b][j+1][h] = start[b][j][h] M[b][j][h] + R[b][j][h] from start[b][0] = s0 (or zeros), start[b][1] = R[b][0] on.  A CTA carries
// ROWS rows of one chain's state (rows are independent); of a step's products its four warps take 16 of the 64 terms each, all rows and two
// columns a lane, so that M is read from shared memory once, and add their parts up.  Plain fp32 products.  Bound by the latency of its
// nseg - 2 steps, 1.1 us each (16 rows, whole sums in a thread, M read by every warp: 1.8).
constexpr int ROWS = 8;
__global__ void __launch_bounds__(128) split_starts_kernel(const float* s0, const float* R, const float* M, float* start, int nseg, long long H) {
    __shared__ __align__(16) float m[2][NN], s[N][ROWS], part[4][ROWS][N];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, r = tid >> 4, c = (tid & 15) * 4;  // this thread's entries of the state: row r, columns c ..
    const long long b = blockIdx.x / H, h = blockIdx.x % H;
    auto at = [&](int j) { return ((b * nseg + j) * H + h) * NN; };
    const long long mine = (ROWS * blockIdx.y + r) * N + c;
    auto fetch = [&](int j) {
        if (j < nseg - 1)
            for (int i = tid; i < NN / 4; i += 128) cp_async16(&m[j & 1][4 * i], M + at(j) + 4 * i);
        cp_async_commit();
    };
    fetch(1);
    *reinterpret_cast<float4*>(start + at(0) + mine) = s0 ? *reinterpret_cast<const float4*>(s0 + (long long)blockIdx.x * NN + mine) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 S = *reinterpret_cast<const float4*>(R + at(0) + mine), next = nseg > 2 ? *reinterpret_cast<const float4*>(R + at(1) + mine) : S;
    for (int j = 1; j < nseg; ++j) {
        *reinterpret_cast<float4*>(start + at(j) + mine) = S;
        if (j == nseg - 1) break;
        s[c][r] = S.x; s[c + 1][r] = S.y; s[c + 2][r] = S.z; s[c + 3][r] = S.w;
        S = next;
        cp_async_wait<0>();
        __syncthreads();  // everyone is past the other buffers, too
        fetch(j + 1);
        if (j + 2 < nseg) next = *reinterpret_cast<const float4*>(R + at(j + 1) + mine);
        F2 acc[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) acc[i] = f2(0.f, 0.f);
#pragma unroll
        for (int kk = 0; kk < N / 4; ++kk) {
            const int k = N / 4 * w + kk;
            const float2 y = *reinterpret_cast<const float2*>(&m[j & 1][k * N + 2 * lane]);
            float x[ROWS];
            *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(&s[k][0]);
            *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(&s[k][4]);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) acc[i] = fma2(f2(x[i], x[i]), f2(y.x, y.y), acc[i]);
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i) *reinterpret_cast<float2*>(&part[w][i][2 * lane]) = make_float2(acc[i].x, acc[i].y);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 v = *reinterpret_cast<const float4*>(&part[q][r][c]);
            S.x += v.x; S.y += v.y; S.z += v.z; S.w += v.w;
        }
    }
    cp_async_wait<0>();
}
static_assert(ROWS == 8 && N == 64, "thread mapping");

}  // namespace

size_t time_split_workspace_bytes(long long B, long long H, int nseg) { return WORK_FLAG_BYTES + 3 * (size_t)(B * nseg * H) * NN * sizeof(float); }

// p: the whole sequences, p.st.b == p.T * p.st.t, p.T % nseg == 0, p.flags: the workspace
int launch_fwd_time_split(const FwdParams& p, int nseg, int impl, cudaStream_t stream) {
    const long long chains = p.B * nseg * p.H;
    float* start = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p.flags) + WORK_FLAG_BYTES);
    float *R = start + chains * NN, *M = R + chains * NN;
    FwdParams q = p;  // segments as batch entries
    q.T = p.T / nseg; q.st.b = q.T * p.st.t;
    q.B = p.B == 1 ? nseg - 1 : p.B * nseg;
    q.sT = R; q.sM = M; q.nseg = nseg;
    int rc = launch_fwd_tc(q, impl, false, stream);
    if (rc != kOk) return rc;
    split_starts_kernel<<<dim3((unsigned)(p.B * p.H), N / ROWS), 128, 0, stream>>>(p.s0, R, M, start, nseg, p.H);
    if (cudaGetLastError() != cudaSuccess) return kLaunchFailed;
    q.B = p.B * nseg;
    q.s0 = start; q.sM = nullptr;
    if ((rc = launch_fwd_tc(q, impl, false, stream)) != kOk) return rc;
    for (long long b = 0; b < p.B; ++b)
        if (p.sT && cudaMemcpyAsync(p.sT + b * p.H * NN, R + (b * nseg + nseg - 1) * p.H * NN, p.H * NN * sizeof(float), cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
            return kLaunchFailed;
    return kOk;
}

}  // namespace wkv7
