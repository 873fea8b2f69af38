// expand_loras for sm_100a: second-stage LoRA expansion producing (w, k, kk, b) for the WKV7 mixer.
// Replaces fw_triton_ / bw_triton_ of the reference (wind_rwkv/rwkv7/rwkv7_expand_loras.py:32-79, 91-211):
//     w  = -softplus(-(w_bias + w_in)) - 0.5
//     z  = tanh(z_in) @ Wz^T + k_in ;   kk = z / sqrt(max(sum_head z^2, 1e-12))
//     a  = sigmoid(a_in @ Wa^T + a_bias)   ma, mk likewise
//     k  = k_in * (ma + a - ma*a) * exp(w * mk) ;   b = -kk * a
// A warp (backward: two) handles 16 tokens x one head (64 channels): the rank-D products are bf16 m16n8k16 MMAs
// with the head's weight slices staged in shared memory, the per-head L2 norm is a 4-lane shuffle.
// Forward: grid (H, rows/64).  Backward: grid (H, segments), each walking its rows in 64-token tiles so the
// weight gradients stay in registers (half a LoRA per warp; bias gradients ride along as an extra
// all-ones input column) and are flushed once with fp32 atomics; the input gradients, which
// contract over all heads, are written as per-head partials and summed by a small kernel.
#include "expand_loras.h"
#include "mma_bf16.cuh"
#include "wkv7_kernels.h"

namespace wkv7 {

constexpr int HC = 64;  // channels per head

// The gates of two adjacent channels:  a, ma, mk = sigmoid(xa, xm, xk);  w = -softplus(-v) - 0.5;  E = exp(w * mk).
// Seven special-function instructions an element (three tanh for the sigmoids, ex2 + lg2 for the softplus, ex2 for E), everything
// else two elements an instruction: the op is bound by issue slots.
struct Gates { F2 a, ma, mk, w, E; };
__device__ __forceinline__ float lg2_approx(float x) {  // of 1 + e^.., at least 1; with __log2f B32 T1024 C768, forward and backward, took 276 us, with this 271
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ F2 sigmoid2(F2 x) {
    x = mul2(x, f2(0.5f, 0.5f));
    return fma2(f2(tanh_f(x.x), tanh_f(x.y)), f2(0.5f, 0.5f), f2(0.5f, 0.5f));
}
__device__ __forceinline__ F2 neg2(F2 x) { return f2(-x.x, -x.y); }
__device__ __forceinline__ F2 bf2(const void* p) {  // two bf16 values
    const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p));
    return f2(v.x, v.y);
}
// SIG = false: xa is a already.
template <bool SIG = true> __device__ __forceinline__ Gates lora_gates(F2 xa, F2 xm, F2 xk, F2 v) {
    constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
    Gates o;
    o.a = SIG ? sigmoid2(xa) : xa;
    o.ma = sigmoid2(xm);
    o.mk = sigmoid2(xk);
    const F2 n = mul2(v, f2(-LOG2E, -LOG2E));
    const F2 e = add2(f2(ex2_approx(fminf(n.x, 115.f)), ex2_approx(fminf(n.y, 115.f))), f2(1.f, 1.f));
    o.w = fma2(f2(lg2_approx(e.x), lg2_approx(e.y)), f2(-LN2, -LN2), f2(-0.5f, -0.5f));
    const F2 x = mul2(mul2(o.w, o.mk), f2(LOG2E, LOG2E));
    o.E = f2(ex2_approx(x.x), ex2_approx(x.y));
    return o;
}

constexpr int GLD = HC + 8;  // row stride (bf16) of the [token][channel] tiles: 4-byte accesses in the MMA fragment pattern
                             // (rows g, columns 2 * t4) and 16-byte row accesses are both free of bank conflicts
template <int D> struct LorasFwdSmem {
    bf16 W[4][HC][D + 8];  // [channel][rank]
    // [token][channel] tiles of one head: w_in, k_in on the way in (16-byte cp.async, whole 128-byte rows), the four
    // outputs on the way out (at rank 16 two by two through two tiles, which makes room for six CTAs an SM: 97 -> 86 us for 32768 rows of
    // 768 channels; at higher ranks the registers that the other two wait in cost more than that) (written in the fragment pattern, stored as whole rows).  Global accesses in the
    // fragment pattern itself would touch 16 bytes per row and instruction.
    static constexpr int TILES = D == 16 ? 2 : 4;
    bf16 io[TILES][64][GLD];
};

// B fragments (rows 8 j .., k block k0) of LoRAs l and l + 1 / of LoRA l alone
template <int D> __device__ __forceinline__ void ldW2(uint32_t (&b0)[2], uint32_t (&b1)[2], const bf16 (*W)[HC][D + 8], int l, int n0, int k0, int lane) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(b0[0]), "=r"(b0[1]), "=r"(b1[0]), "=r"(b1[1])
                 : "r"(smem_addr(&W[l + (lane >> 4)][n0 + (lane & 7)][k0 + (lane & 8)])));
}
template <int D> __device__ __forceinline__ void ldW1(uint32_t (&b)[2], const bf16 (*W)[HC][D + 8], int l, int n0, int k0, int lane) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(b[0]), "=r"(b[1])
                 : "r"(smem_addr(&W[l][n0 + (lane & 7)][k0 + (lane & 8)])));
}

// A fragments of a [16, D] input block straight from global memory (rows r0+g, r0+g+8).
template <int D, bool TANH>
__device__ __forceinline__ void load_in_frags(uint32_t (&a)[D / 16][4], const bf16* base, long long ld, long long r0, long long rows, int g, int t4) {
    const bf16* p0 = base + min(r0 + g, rows - 1) * ld + 2 * t4;      // (rows past the end: any values, nothing of them is stored)
    const bf16* p1 = base + min(r0 + g + 8, rows - 1) * ld + 2 * t4;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t v[4] = {*reinterpret_cast<const uint32_t*>(p0 + 16 * ks), *reinterpret_cast<const uint32_t*>(p1 + 16 * ks),
                         *reinterpret_cast<const uint32_t*>(p0 + 16 * ks + 8), *reinterpret_cast<const uint32_t*>(p1 + 16 * ks + 8)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (TANH) {
                float2 f = unpack_bf16x2(v[i]);
                v[i] = pack_bf16x2(tanh_f(f.x), tanh_f(f.y));
            }
            a[ks][i] = v[i];
        }
    }
}

template <int D>
__global__ void __launch_bounds__(128, D == 16 ? 6 : 1) loras_fwd_kernel(LorasParams p) {
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<LorasFwdSmem<D>*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int h = blockIdx.x, C = (int)p.C;
    const long long t0 = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * 64, r0 = t0 + 16 * warp;
    for (int i = tid; i < 4 * HC * (D / 8); i += 128) {
        const int l = i / (HC * (D / 8)), r = (i / (D / 8)) % HC, ch = i % (D / 8);
        cp_async16(&sm.W[l][r][ch * 8], (const bf16*)p.W[l] + (long long)(h * HC + r) * D + ch * 8);
    }
    {   // this CTA's 64 tokens of w_in and k_in; rows past the end are filled with zeros
        for (int i = tid; i < 2 * 64 * 8; i += 128) {
            const int ten = i / 512, r = (i / 8) % 64, ch = i % 8;
            const bool live = t0 + r < p.rows;
            const bf16* src = (const bf16*)(ten ? p.k_in : p.w_in) + (live ? t0 + r : 0) * C + h * HC + ch * 8;
            cp_async16_zfill(&sm.io[ten][r][ch * 8], src, live);
        }
    }
    cp_async_commit();
    // the LoRA inputs come straight from global memory into MMA fragments: requested before the wait for the asynchronous
    // copies, so that the two latencies overlap
    uint32_t az[D / 16][4], aa[D / 16][4], am[D / 16][4], ak[D / 16][4];
    if (r0 < p.rows) {
        load_in_frags<D, true>(az, (const bf16*)p.lin[0], p.ld[0], r0, p.rows, g, t4);
        load_in_frags<D, false>(aa, (const bf16*)p.lin[1], p.ld[1], r0, p.rows, g, t4);
        load_in_frags<D, false>(am, (const bf16*)p.lin[2], p.ld[2], r0, p.rows, g, t4);
        load_in_frags<D, false>(ak, (const bf16*)p.lin[3], p.ld[3], r0, p.rows, g, t4);
    }
    cp_async_wait<0>();
    __syncthreads();
    if (r0 >= p.rows) return;
    const int lr = 16 * warp;  // this warp's first tile row

    float z[8][4];
    float ss0 = 0.f, ss1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        z[j][0] = z[j][1] = z[j][2] = z[j][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t b[2];
            ldW1<D>(b, sm.W, 0, 8 * j, 16 * ks, lane);
            mma_bf16(z[j], az[ks], b);
        }
        const float2 k0 = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&sm.io[1][lr + g][8 * j + 2 * t4]));
        const float2 k1 = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&sm.io[1][lr + g + 8][8 * j + 2 * t4]));
        z[j][0] += k0.x; z[j][1] += k0.y; z[j][2] += k1.x; z[j][3] += k1.y;
        ss0 += z[j][0] * z[j][0] + z[j][1] * z[j][1];
        ss1 += z[j][2] * z[j][2] + z[j][3] * z[j][3];
    }
    ss0 += __shfl_xor_sync(0xffffffffu, ss0, 1); ss0 += __shfl_xor_sync(0xffffffffu, ss0, 2);
    ss1 += __shfl_xor_sync(0xffffffffu, ss1, 1); ss1 += __shfl_xor_sync(0xffffffffu, ss1, 2);
    const float in0 = rsqrtf(fmaxf(ss0, 1e-12f)), in1 = rsqrtf(fmaxf(ss1, 1e-12f));

    constexpr int TILES = LorasFwdSmem<D>::TILES;
    uint32_t kb2[TILES == 2 ? 8 : 1][2][2];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = h * HC + 8 * j + 2 * t4;
        const F2 wb = bf2((const bf16*)p.w_bias + c), ab = bf2((const bf16*)p.bias[0] + c), mb = bf2((const bf16*)p.bias[1] + c), kb = bf2((const bf16*)p.bias[2] + c);
        float fa[4] = {ab.x, ab.y, ab.x, ab.y}, fm[4] = {mb.x, mb.y, mb.x, mb.y}, fk[4] = {kb.x, kb.y, kb.x, kb.y};
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t ba[2], bm[2], bk[2];
            ldW2<D>(ba, bm, sm.W, 1, 8 * j, 16 * ks, lane);
            ldW1<D>(bk, sm.W, 3, 8 * j, 16 * ks, lane);
            mma_bf16(fa, aa[ks], ba);
            mma_bf16(fm, am[ks], bm);
            mma_bf16(fk, ak[ks], bk);
        }
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
            const int tr = lr + g + 8 * hrow, tc = 8 * j + 2 * t4;
            const F2 ki = bf2(&sm.io[1][tr][tc]);
            const float in = hrow ? in1 : in0;
            const Gates gt = lora_gates(f2(fa[2 * hrow], fa[2 * hrow + 1]), f2(fm[2 * hrow], fm[2 * hrow + 1]), f2(fk[2 * hrow], fk[2 * hrow + 1]),
                                        add2(wb, bf2(&sm.io[0][tr][tc])));
            const F2 kk = mul2(f2(z[j][2 * hrow], z[j][2 * hrow + 1]), f2(in, in)), nkk = neg2(kk);
            const F2 ok = mul2(mul2(ki, fma2(neg2(gt.ma), gt.a, add2(gt.ma, gt.a))), gt.E), ob = mul2(nkk, gt.a);
            // w and k replace w_in and k_in in their tiles (this thread's element, already read); kk and b wait in registers
            *reinterpret_cast<uint32_t*>(&sm.io[0][tr][tc]) = pack_bf16x2(gt.w.x, gt.w.y);
            *reinterpret_cast<uint32_t*>(&sm.io[1][tr][tc]) = pack_bf16x2(ok.x, ok.y);
            if (TILES == 2) {
                kb2[TILES == 2 ? j : 0][hrow][0] = pack_bf16x2(kk.x, kk.y);
                kb2[TILES == 2 ? j : 0][hrow][1] = pack_bf16x2(ob.x, ob.y);
            } else {
                *reinterpret_cast<uint32_t*>(&sm.io[TILES - 2][tr][tc]) = pack_bf16x2(kk.x, kk.y);
                *reinterpret_cast<uint32_t*>(&sm.io[TILES - 1][tr][tc]) = pack_bf16x2(ob.x, ob.y);
            }
        }
    }
    // the warp's 16 rows of two outputs at a time leave as whole 128-byte rows (live rows only)
#pragma unroll
    for (int pair = 0; pair < 2; ++pair) {
        __syncwarp();
        if (pair && TILES == 2) {
#pragma unroll
            for (int j = 0; j < (TILES == 2 ? 8 : 0); ++j)
#pragma unroll
                for (int hrow = 0; hrow < 2; ++hrow) {
                    const int tr = lr + g + 8 * hrow, tc = 8 * j + 2 * t4;
                    *reinterpret_cast<uint32_t*>(&sm.io[0][tr][tc]) = kb2[j][hrow][0];
                    *reinterpret_cast<uint32_t*>(&sm.io[1][tr][tc]) = kb2[j][hrow][1];
                }
            __syncwarp();
        }
#pragma unroll
        for (int ten = 0; ten < 2; ++ten) {
            bf16* out = (bf16*)(pair ? (ten ? p.b_out : p.kk_out) : (ten ? p.k_out : p.w_out));
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int r = lr + 4 * it + (lane >> 3), ch = lane & 7;
                const long long row = t0 + r;
                if (row < p.rows) *reinterpret_cast<uint4*>(out + row * C + h * HC + ch * 8) = *reinterpret_cast<const uint4*>(&sm.io[TILES == 2 ? ten : 2 * pair + ten][r][ch * 8]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------

template <int D> struct LorasBwdSmem {
    bf16 W[4][HC][D + 8];        // [channel][rank]: B operand of the forward, [k][n] operand of d(input)
    bf16 in[4][64][D + 8];       // tanh(z_in), a_in, ma_in, mk_in; column D is all ones (bias gradient)
    // [token][channel] tiles of one head.  On the way in (16-byte cp.async, whole 128-byte rows) tiles 0..5 hold
    // w_in, k_in, dw_out, dk_out, db_out, dkk_out.  Each thread replaces, element by element, what it has read: tiles
    // 0..4 become the pre-activation gradients of z, a, ma, mk and dw_in (the gradient of w_in), tile 5 becomes dk_in.
    bf16 gr[6][64][GLD];
    float rs[2][64][2];          // row sums of the two channel halves
};

// Eight warps: warps rg and rg + 4 share the 16 tokens rg of a tile, 32 channels each (the row sums meet in shared memory), so that
// the per-thread state fits 128 registers and 16 warps are resident (four warps of all channels: 212 registers and 8 warps
// an SM).  Bound by instruction latency (0.46 instructions a cycle and scheduler) at 188 us for 32768 rows x 12 heads of rank 16, 254 us
// with four warps, unpacked arithmetic and conflicting row pitches.
constexpr int BWD_THREADS = 256;
template <int D>
__global__ void __launch_bounds__(BWD_THREADS, D <= 32 ? 2 : 1) loras_bwd_kernel(LorasParams p) {
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<LorasBwdSmem<D>*>(smem_raw);
    const int tid = threadIdx.x, warp = (tid >> 5) & 3, half = tid >> 7, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + warp) : "memory"); };
    const int h = blockIdx.x, C = (int)p.C, H = C / HC;
    const long long T = p.rows;

    for (int i = tid; i < 4 * HC * (D / 8); i += BWD_THREADS) {
        const int l = i / (HC * (D / 8)), r = (i / (D / 8)) % HC, ch = i % (D / 8);
        cp_async16(&sm.W[l][r][ch * 8], (const bf16*)p.W[l] + (long long)(h * HC + r) * D + ch * 8);
    }
    cp_async_commit();
    for (int i = tid; i < 4 * 64 * 8; i += BWD_THREADS) {  // ones column and padding
        const int l = i / (64 * 8), r = (i / 8) % 64, c = i % 8;
        sm.in[l][r][D + c] = __float2bfloat16(c == 0 ? 1.f : 0.f);
    }

    // weight-gradient accumulators: warps w, w + 4 own LoRA w: 32 channels each x [D ranks + ones column], plus channel
    // m-tile w of the dw_bias column, two of the four token blocks each
    constexpr int NT = D / 8 + 1;
    float dWacc[2][NT][4] = {};
    float dwb[4] = {};

    // gridDim.y CTAs share a head's rows: each walks a contiguous range of 64-token tiles (more resident
    // CTAs per SM; the price is one more flush of the weight-gradient accumulators per extra CTA)
    const long long tiles = (T + 63) / 64, per = (tiles + gridDim.y - 1) / gridDim.y;
    const long long tbeg = blockIdx.y * per * 64, tend = min(T, tbeg + per * 64);
    for (long long t0 = tbeg; t0 < tend; t0 += 64) {
        const long long r0 = t0 + 16 * warp;
        const bool valid = t0 + 16 * warp < T;
        // ---- the six [token][channel] tiles first (asynchronous copies), then this tile's LoRA inputs under them ------------
        {
            const bf16* src6[6] = {(const bf16*)p.w_in, (const bf16*)p.k_in, (const bf16*)p.dw_out, (const bf16*)p.dk_out,
                                   (const bf16*)p.db_out, (const bf16*)p.dkk_out};
            for (int i = tid; i < 6 * 64 * 8; i += BWD_THREADS) {
                const int ten = i / 512, r = (i / 8) % 64, ch = i % 8;
                const bool live = t0 + r < T;
                cp_async16_zfill(&sm.gr[ten][r][ch * 8], src6[ten] + (live ? t0 + r : 0) * C + h * HC + ch * 8, live);
            }
            cp_async_commit();
        }
        // LoRA inputs (tanh applied to z_in): the loads of a group of four are issued together, so that their latencies overlap
        {
            constexpr int ITEMS = 4 * 64 * (D / 8) / BWD_THREADS, G = ITEMS < 4 ? ITEMS : 4;  // per thread
            static_assert(ITEMS % G == 0, "whole groups of loads per thread");
#pragma unroll
            for (int i0 = 0; i0 < ITEMS; i0 += G) {
                uint4 v[G];
#pragma unroll
                for (int u = 0; u < G; ++u) {
                    const int i = tid + BWD_THREADS * (i0 + u);
                    const int l = i / (64 * (D / 8)), r = (i / (D / 8)) % 64, ch = i % (D / 8);
                    v[u] = make_uint4(0, 0, 0, 0);
                    if (t0 + r < T) v[u] = *reinterpret_cast<const uint4*>((const bf16*)p.lin[l] + (t0 + r) * p.ld[l] + ch * 8);
                }
#pragma unroll
                for (int u = 0; u < G; ++u) {
                    const int i = tid + BWD_THREADS * (i0 + u);
                    const int l = i / (64 * (D / 8)), r = (i / (D / 8)) % 64, ch = i % (D / 8);
                    if (l == 0) {
                        float f[8];
                        unpack8(v[u], f);
#pragma unroll
                        for (int q = 0; q < 8; ++q) f[q] = tanh_f(f[q]);
                        v[u] = pack8(f);
                    }
                    *reinterpret_cast<uint4*>(&sm.in[l][r][ch * 8]) = v[u];
                }
            }
        }
        cp_async_wait<0>();
        __syncthreads();

        if (valid) {
            const int lr = 16 * warp;  // first tile row of this warp
            uint32_t az[D / 16][4], aa[D / 16][4], am[D / 16][4], ak[D / 16][4];
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                ldA_mk(az[ks], &sm.in[0][0][0], D + 8, lr, 16 * ks, g, t4);
                ldA_mk(aa[ks], &sm.in[1][0][0], D + 8, lr, 16 * ks, g, t4);
                ldA_mk(am[ks], &sm.in[2][0][0], D + 8, lr, 16 * ks, g, t4);
                ldA_mk(ak[ks], &sm.in[3][0][0], D + 8, lr, 16 * ks, g, t4);
            }
            // ---- pass A: z, a; row sums for the norm and its gradient -----------------------------------
            float z[4][4], dzo[4][4];
            F2 av[4][2];  // (kept for pass B: formed again, product and sigmoid, 292 us where this is 285, forward and backward of 32768 rows of 768)
            F2 ss2[2] = {}, dn2[2] = {};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const F2 ab = bf2((const bf16*)p.bias[0] + h * HC + 32 * half + 8 * j + 2 * t4);
                float fa[4] = {ab.x, ab.y, ab.x, ab.y};
                z[j][0] = z[j][1] = z[j][2] = z[j][3] = 0.f;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    uint32_t bz[2], ba[2];
                    ldW2<D>(bz, ba, sm.W, 0, 8 * j + 32 * half, 16 * ks, lane);
                    mma_bf16(z[j], az[ks], bz);
                    mma_bf16(fa, aa[ks], ba);
                }
#pragma unroll
                for (int hrow = 0; hrow < 2; ++hrow) {
                    const int tr = lr + g + 8 * hrow, tc = 32 * half + 8 * j + 2 * t4;
                    const F2 zz = add2(f2(z[j][2 * hrow], z[j][2 * hrow + 1]), bf2(&sm.gr[1][tr][tc]));
                    const F2 a = sigmoid2(f2(fa[2 * hrow], fa[2 * hrow + 1]));
                    av[j][hrow] = a;
                    const F2 dz = fma2(neg2(bf2(&sm.gr[4][tr][tc])), a, bf2(&sm.gr[5][tr][tc]));  // gradient of kk
                    ss2[hrow] = fma2(zz, zz, ss2[hrow]);
                    dn2[hrow] = fma2(dz, zz, dn2[hrow]);
                    z[j][2 * hrow] = zz.x; z[j][2 * hrow + 1] = zz.y;
                    dzo[j][2 * hrow] = dz.x; dzo[j][2 * hrow + 1] = dz.y;
                }
            }
            float ss[2] = {ss2[0].x + ss2[0].y, ss2[1].x + ss2[1].y}, dn[2] = {dn2[0].x + dn2[0].y, dn2[1].x + dn2[1].y};
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                ss[hrow] += __shfl_xor_sync(0xffffffffu, ss[hrow], 1); ss[hrow] += __shfl_xor_sync(0xffffffffu, ss[hrow], 2);
                dn[hrow] += __shfl_xor_sync(0xffffffffu, dn[hrow], 1); dn[hrow] += __shfl_xor_sync(0xffffffffu, dn[hrow], 2);
            }
            if (t4 == 0) {
#pragma unroll
                for (int hrow = 0; hrow < 2; ++hrow)
                    *reinterpret_cast<float2*>(sm.rs[half][lr + g + 8 * hrow]) = make_float2(ss[hrow], dn[hrow]);
            }
            pair_sync();
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                const float2 o = *reinterpret_cast<const float2*>(sm.rs[half ^ 1][lr + g + 8 * hrow]);
                ss[hrow] += o.x;
                dn[hrow] += o.y;
            }
            const float inorm[2] = {rsqrtf(fmaxf(ss[0], 1e-12f)), rsqrtf(fmaxf(ss[1], 1e-12f))};
            const float ncorr[2] = {-dn[0] * inorm[0] * inorm[0] * inorm[0], -dn[1] * inorm[1] * inorm[1] * inorm[1]};
            // ---- pass B: everything elementwise, gradients into the shared tiles ----------------------------
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = h * HC + 32 * half + 8 * j + 2 * t4;
                const F2 wb = bf2((const bf16*)p.w_bias + c), mb = bf2((const bf16*)p.bias[1] + c), kb = bf2((const bf16*)p.bias[2] + c);
                float fm[4] = {mb.x, mb.y, mb.x, mb.y}, fk[4] = {kb.x, kb.y, kb.x, kb.y};
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    uint32_t bm[2], bk[2];
                    ldW2<D>(bm, bk, sm.W, 2, 8 * j + 32 * half, 16 * ks, lane);
                    mma_bf16(fm, am[ks], bm);
                    mma_bf16(fk, ak[ks], bk);
                }
#pragma unroll
                for (int hrow = 0; hrow < 2; ++hrow) {
                    const int tr = lr + g + 8 * hrow, tc = 32 * half + 8 * j + 2 * t4;
                    const F2 ki = bf2(&sm.gr[1][tr][tc]), v = add2(wb, bf2(&sm.gr[0][tr][tc]));
                    const Gates gt = lora_gates<false>(av[j][hrow], f2(fm[2 * hrow], fm[2 * hrow + 1]), f2(fk[2 * hrow], fk[2 * hrow + 1]), v);
                    const F2 kmix = fma2(neg2(gt.ma), gt.a, add2(gt.ma, gt.a));
                    const F2 zz = f2(z[j][2 * hrow], z[j][2 * hrow + 1]), in = f2(inorm[hrow], inorm[hrow]);
                    const F2 dkE = mul2(bf2(&sm.gr[3][tr][tc]), gt.E), dkin = mul2(dkE, ki);
                    const F2 de = mul2(dkin, kmix);                                      // gradient of w * mk
                    const F2 dwt = fma2(de, gt.mk, bf2(&sm.gr[2][tr][tc])), dmk = mul2(de, gt.w);
                    const F2 dma = fma2(neg2(dkin), gt.a, dkin);
                    const F2 da = fma2(neg2(bf2(&sm.gr[4][tr][tc])), mul2(zz, in), fma2(neg2(dkin), gt.ma, dkin));
                    const F2 o_z = fma2(f2(dzo[j][2 * hrow], dzo[j][2 * hrow + 1]), in, mul2(zz, f2(ncorr[hrow], ncorr[hrow])));
                    const F2 o_dw = mul2(dwt, sigmoid2(neg2(v))), o_dk = fma2(dkE, kmix, o_z);
                    const F2 o_a = mul2(da, fma2(neg2(gt.a), gt.a, gt.a)), o_m = mul2(dma, fma2(neg2(gt.ma), gt.ma, gt.ma));
                    const F2 o_k = mul2(dmk, fma2(neg2(gt.mk), gt.mk, gt.mk));
                    *reinterpret_cast<uint32_t*>(&sm.gr[5][tr][tc]) = pack_bf16x2(o_dk.x, o_dk.y);
                    *reinterpret_cast<uint32_t*>(&sm.gr[0][tr][tc]) = pack_bf16x2(o_z.x, o_z.y);
                    *reinterpret_cast<uint32_t*>(&sm.gr[1][tr][tc]) = pack_bf16x2(o_a.x, o_a.y);
                    *reinterpret_cast<uint32_t*>(&sm.gr[2][tr][tc]) = pack_bf16x2(o_m.x, o_m.y);
                    *reinterpret_cast<uint32_t*>(&sm.gr[3][tr][tc]) = pack_bf16x2(o_k.x, o_k.y);
                    *reinterpret_cast<uint32_t*>(&sm.gr[4][tr][tc]) = pack_bf16x2(o_dw.x, o_dw.y);
                }
            }
            pair_sync();
            {   // dw_in (tile 4, one warp) and dk_in (tile 5, the other) leave as whole 128-byte rows (live rows only)
                const int ten = 4 + half;
#pragma unroll
                    for (int it = 0; it < 4; ++it) {
                        const int r = lr + 4 * it + (lane >> 3), ch = lane & 7;
                        if (t0 + r < T)
                            *reinterpret_cast<uint4*>((bf16*)(ten == 4 ? p.dw_in : p.dk_in) + (t0 + r) * C + h * HC + ch * 8) =
                                *reinterpret_cast<const uint4*>(&sm.gr[ten][r][ch * 8]);
                    }
            }
            // ---- d(input) partial of this head: [16, D] = grad[16, 64] @ W[64, D] ----------------------------
#pragma unroll
            for (int l2 = 0; l2 < 2; ++l2) {
                const int l = 2 * half + l2;
                float acc[D / 8][4] = {};
#pragma unroll
                for (int ks = 0; ks < HC / 16; ++ks) {
                    uint32_t a[4];
                    ldA_mk(a, &sm.gr[l][0][0], GLD, lr, 16 * ks, g, t4);
#pragma unroll
                    for (int j = 0; j < D / 8; ++j) {
                        uint32_t b[2];
                        ldB_kn_trans(b, &sm.W[l][0][0], D + 8, 8 * j, 16 * ks, lane);
                        mma_bf16(acc[j], a, b);
                    }
                }
                bf16* po = (bf16*)p.partial + (((long long)l * p.rows + r0 + g) * H + h) * D + 2 * t4;
#pragma unroll
                for (int j = 0; j < D / 8; ++j) {
                    float v0 = acc[j][0], v1 = acc[j][1], v2 = acc[j][2], v3 = acc[j][3];
                    if (l == 0) {  // through the tanh of z_in
                        const float2 t0v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&sm.in[0][lr + g][8 * j + 2 * t4]));
                        const float2 t1v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&sm.in[0][lr + g + 8][8 * j + 2 * t4]));
                        v0 *= 1.f - t0v.x * t0v.x; v1 *= 1.f - t0v.y * t0v.y;
                        v2 *= 1.f - t1v.x * t1v.x; v3 *= 1.f - t1v.y * t1v.y;
                    }
                    if (r0 + g < T) *reinterpret_cast<uint32_t*>(po + 8 * j) = pack_bf16x2(v0, v1);
                    if (r0 + g + 8 < T) *reinterpret_cast<uint32_t*>(po + 8LL * H * D + 8 * j) = pack_bf16x2(v2, v3);
                }
            }
        } else {
            // rows past the end of the sequence contribute nothing to the weight gradients
            for (int i = lane + 32 * half; i < 5 * 16 * (HC / 8); i += 64) {
                const int l = i / (16 * (HC / 8)), r = (i / (HC / 8)) % 16, ch = i % (HC / 8);
                *reinterpret_cast<uint4*>(&sm.gr[l][16 * warp + r][ch * 8]) = make_uint4(0, 0, 0, 0);
            }
        }
        __syncthreads();
        // ---- weight gradients: dW_l[64, D+ones] += grad_l^T[64, tokens] @ in_l[tokens, D+ones] ---------------
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            uint32_t b[NT][2];
#pragma unroll
            for (int j = 0; j < NT; ++j) ldB_kn_trans(b[j], &sm.in[warp][0][0], D + 8, 8 * j, 16 * ks, lane);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                uint32_t a[4];
                ldA_km_trans(a, &sm.gr[warp][0][0], GLD, 32 * half + 16 * mt, 16 * ks, lane);
#pragma unroll
                for (int j = 0; j < NT; ++j) mma_bf16(dWacc[mt][j], a, b[j]);
            }
            if ((ks & 1) == half) {
                uint32_t a[4];
                ldA_km_trans(a, &sm.gr[4][0][0], GLD, 16 * warp, 16 * ks, lane);
                mma_bf16(dwb, a, b[NT - 1]);
            }
        }
        __syncthreads();
    }

    // ---- flush ------------------------------------------------------------------------------------------
    float* dWo = p.dW[warp];
    float* dbo = warp == 0 ? nullptr : p.dbias[warp - 1];  // LoRA 0 (z) has no bias
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
            const int ch = h * HC + 32 * half + 16 * mt + g + 8 * hrow;
#pragma unroll
            for (int j = 0; j < D / 8; ++j) {
                atomicAdd(dWo + (long long)ch * D + 8 * j + 2 * t4, dWacc[mt][j][2 * hrow]);
                atomicAdd(dWo + (long long)ch * D + 8 * j + 2 * t4 + 1, dWacc[mt][j][2 * hrow + 1]);
            }
            if (dbo && t4 == 0) atomicAdd(dbo + ch, dWacc[mt][NT - 1][2 * hrow]);
        }
    if (t4 == 0) {
        atomicAdd(p.dw_bias + h * HC + 16 * warp + g, dwb[0]);
        atomicAdd(p.dw_bias + h * HC + 16 * warp + g + 8, dwb[2]);
    }
}

// sums the per-head partials: out[l][row][d] = sum_h partial[l][row][h][d]; 8 values (16 bytes) per thread
__global__ void loras_reduce_heads_kernel(LorasParams p, int H, int D) {
    stream_order();
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;  // index over [rows, D / 8]
    const int l = blockIdx.y, per = D / 8;
    const long long row = i / per;
    if (row >= p.rows) return;
    const int d = (int)(i - row * per) * 8;
    const bf16* src = (const bf16*)p.partial + ((long long)l * p.rows + row) * H * D + d;
    float acc[8] = {};
#pragma unroll 4
    for (int hh = 0; hh < H; ++hh) {
        float f[8];
        unpack8(*reinterpret_cast<const uint4*>(src + (long long)hh * D), f);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] += f[q];
    }
    *reinterpret_cast<uint4*>((bf16*)p.dlin[l] + row * p.ldg[l] + d) = pack8(acc);
}

template <int D> static int launch_loras_fwd_t(const LorasParams& p, cudaStream_t stream) {
    auto kern = loras_fwd_kernel<D>;
    const int smem = (int)sizeof(LorasFwdSmem<D>);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return kLaunchFailed;
    const long long tiles = (p.rows + 63) / 64, ny = tiles < 32768 ? tiles : 32768;  // y and z end at 65535
    return launch(kern, dim3((unsigned)(p.C / HC), (unsigned)ny, (unsigned)((tiles + ny - 1) / ny)), 128, smem, stream, p) ? kOk : kLaunchFailed;
}

template <int D> static int launch_loras_bwd_t(const LorasParams& p, cudaStream_t stream) {
    const int C = (int)p.C, H = C / HC;
    // the accumulated outputs start from zero; one call where they lie back to back
    struct { float* p; size_t n; } z[8] = {{p.dW[0], (size_t)C * D}, {p.dW[1], (size_t)C * D}, {p.dW[2], (size_t)C * D}, {p.dW[3], (size_t)C * D},
                                           {p.dw_bias, (size_t)C}, {p.dbias[0], (size_t)C}, {p.dbias[1], (size_t)C}, {p.dbias[2], (size_t)C}};
    for (int i = 0; i < 8;) {
        size_t n = z[i].n;
        int j = i + 1;
        while (j < 8 && z[j].p == z[i].p + n) n += z[j++].n;
        if (cudaMemsetAsync(z[i].p, 0, sizeof(float) * n, stream) != cudaSuccess) return kLaunchFailed;
        i = j;
    }
    if (p.rows == 0) return kOk;
    auto kern = loras_bwd_kernel<D>;
    const int smem = (int)sizeof(LorasBwdSmem<D>);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return kLaunchFailed;
    // one round of resident CTAs, at most one per 64-token tile: each flushes its weight-gradient sums once, and a second round
    // would rarely be full (32768 rows x 12 heads, 1188 CTAs on 296 places: 5 % slower)
    static const int resident = [&] {
        int n = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, BWD_THREADS, smem) == cudaSuccess && n > 0 ? n : 1;
    }();
    const long long tiles = (p.rows + 63) / 64;
    long long nseg = (long long)resident * sm_count() / H;
    if (nseg > tiles) nseg = tiles;
    if (nseg < 1) nseg = 1;
    if (!launch(kern, dim3((unsigned)H, (unsigned)nseg), BWD_THREADS, smem, stream, p)) return kLaunchFailed;
    const long long n = p.rows * (D / 8);
    return launch(loras_reduce_heads_kernel, dim3((unsigned)((n + 255) / 256), 4), 256, 0, stream, p, H, D) ? kOk : kLaunchFailed;
}

int launch_loras_fwd(const LorasParams& p, cudaStream_t stream) {
    switch (p.D) {
        case 16: return launch_loras_fwd_t<16>(p, stream);
        case 32: return launch_loras_fwd_t<32>(p, stream);
        case 64: return launch_loras_fwd_t<64>(p, stream);
        case 128: return launch_loras_fwd_t<128>(p, stream);
        default: return kBadShape;
    }
}
int launch_loras_bwd(const LorasParams& p, cudaStream_t stream) {
    switch (p.D) {
        case 16: return launch_loras_bwd_t<16>(p, stream);
        case 32: return launch_loras_bwd_t<32>(p, stream);
        case 64: return launch_loras_bwd_t<64>(p, stream);
        case 128: return launch_loras_bwd_t<128>(p, stream);
        default: return kBadShape;
    }
}

}  // namespace wkv7
