// Shared device helpers for the sm_100a WKV7 kernels: TF32 warp-MMA fragments, the chunk
// preparation (decay scan, triangular inverse), MUFU-free exp / reciprocal, cp.async copies, and
// the status codes of the C ABI.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace wkv7 {

constexpr int N = 64;        // head size (value and key width of the state)
constexpr int L = 16;        // chunk length in time steps
constexpr int WARPS = 4;     // one warp per 16 value rows of the state
constexpr int THREADS = 32 * WARPS;
constexpr int OPS = N + 8;   // row stride (floats) of the [time][key] operand buffers
constexpr int SCS = L + 8;   // row stride (floats) of the [time][time] score buffers
// One checkpoint record per 16-step chunk, written by the forward for the backward: the fp32 state at
// the start of the chunk [N][N], then the chunk's four state-independent 16x16 matrices QK, QB (lower
// triangular), AK (strictly lower), AI = (I - AB)^-1 (stored transposed: it is an operand in that form).  The backward loads them instead of rebuilding
// them (two score products per warp and the 16-step inverse).  The matrices are kept in the layout of
// the tcgen05 forward's operand tiles, so that that kernel can copy them out with one bulk copy:
// three K-major tiles of 16-byte chunks, element (row, col) at float (row/8)*128 + (col/4)*32 + (row%8)*4
// + col%4; the first tile has 32 rows (AK in rows 0-15, QK in rows 16-31), then AI^T, then QB.
constexpr int CK_STATE = 0, CK_MATS = N * N;
constexpr int CK_SC = CK_MATS, CK_AI = CK_SC + 2 * L * L, CK_QB = CK_AI + L * L;
__host__ __device__ constexpr int ck_tile_at(int row, int chunk) { return (row >> 3) * 128 + chunk * 32 + (row & 7) * 4; }
constexpr int CK_FLOATS = CK_QB + L * L;  // 5120 floats = 20 KB
// Range of the decay within a chunk.  The kernels factor the decay between two steps of a chunk as P_t * (1 / P_s), with
// P_t the running decay product since the chunk start: over 16 steps of strong decay P_t leaves what fp32 holds.  Two
// measures keep every chunk inside, without a data-dependent branch:
//  * the products are kept as P~_t = 2^64 P_t and 1 / P~_t, so that both use the exponent range on either side of 1
//    (P~ from 2^64 down to e^-80, its reciprocal from 2^-64 up to e^80); every formula of the chunked algorithm is invariant
//    under P -> 2^64 P when the state is carried as S~ = 2^-64 S and its gradient as 2^64 dS (power-of-two scalings,
//    exact): initial states are scaled on the way in, final states and state gradients on the way out, and the
//    checkpoints hold S~;
//  * the per-step log-decay -exp(w) has a floor of -7.75 (16 * 7.75 = 124 = 80 + 64 ln 2): a step that would multiply the
//    state by less than e^-7.75 = 4.3e-4 (w > 2.05) multiplies it by e^-7.75.  RWKV-7 parameterises w <= -0.5 (per-step
//    log-decay >= -0.61) and never comes near it; N(-0.6, 0.5^2) inputs reach it at 5.3 sigma.
constexpr float ANCHOR_LN = 44.361419555836498f;      // 64 ln 2
constexpr float ANCHOR_LOG2 = 64.f;
constexpr float STATE_SCALE = 5.421010862427522e-20f;  // 2^-64
constexpr float STATE_UNSCALE = 18446744073709551616.f;  // 2^64
constexpr float MIN_CUM_LOG_DECAY = -(80.f + ANCHOR_LN);
constexpr float MIN_STEP_LOG_DECAY = -7.75f;

// ---- status codes (mirrored in include/wkv7_sm100.h) -------------------------------------
enum Status : int {
    kOk = 0,
    kBadShape = -1,        // negative or inconsistent dimensions
    kBadHeadSize = -2,     // only N == 64 is built
    kBadChunk = -3,        // ddlerp, expand_loras: C is not a multiple of 64
    kBadAlign = -4,        // pointer or stride not 16-byte aligned
    kBadDtype = -5,
    kNullPointer = -6,
    kLaunchFailed = -7,    // cudaGetLastError() after launch was not cudaSuccess
    kTooLarge = -8,
    kDeviceTimeout = -9,   // a bounded device-side wait (mbar_wait_bounded) gave up
};

// ---- IO element access ----------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// ---- TF32 operands ---------------------------------------------------------------------------
// PREC == 1: one TF32 MMA per product (operands rounded to 10 mantissa bits, fp32 accumulate).
// PREC == 3: hi/lo split, three MMAs per product (error ~2^-21: the fp32 path).
// Round to nearest (ties away from zero) to 10 mantissa bits with two integer instructions.  The
// conversion instruction (cvt.rna.tf32.f32) and MUFU share the XU pipe, which profiling showed
// ~90% busy in these kernels; integer adds run on a pipe with headroom.  Finite inputs only.
__device__ __forceinline__ uint32_t tf32_rna(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }

// Value as it is kept in shared memory for later use as an MMA operand: in the single-TF32 class
// it is rounded once by its producer, so that the (many) consumers need no conversion.
template <int PREC> __device__ __forceinline__ float pre(float x) { return PREC == 1 ? __uint_as_float(tf32_rna(x)) : x; }

template <int PREC> struct Op {  // one scalar operand
    uint32_t h, l;
    __device__ __forceinline__ void set(float x) {
        h = tf32_rna(x);
        if (PREC == 3) l = __float_as_uint(x - __uint_as_float(h)) + 0x1000u;  // rounded by the product, which does not look at the 13 bits below
        else l = 0;
    }
    // x was stored through pre<PREC>() or is exactly representable in TF32 (a bf16 value)
    __device__ __forceinline__ void setr(float x) {
        if (PREC == 1) { h = __float_as_uint(x); l = 0; }
        else set(x);
    }
    template <bool R> __device__ __forceinline__ void put(float x) { if (R) setr(x); else set(x); }
};

template <int PREC> struct FragA { Op<PREC> x[4]; };  // 16x8, (g,t) (g+8,t) (g,t+4) (g+8,t+4)
template <int PREC> struct FragB { Op<PREC> x[2]; };  // 8x8,  (k=t,n=g) (k=t+4,n=g)

__device__ __forceinline__ void mma_tf32_raw(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int PREC>
__device__ __forceinline__ void mma(float (&d)[4], const FragA<PREC>& a, const FragB<PREC>& b) {
    if (PREC == 3) {
        mma_tf32_raw(d, a.x[0].l, a.x[1].l, a.x[2].l, a.x[3].l, b.x[0].h, b.x[1].h);
        mma_tf32_raw(d, a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].l, b.x[1].l);
    }
    mma_tf32_raw(d, a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].h, b.x[1].h);
}

// Every contraction here sums over an index block of 8; the two k-slots a thread feeds
// (slot t and slot t+4) are mapped to the ADJACENT actual indices 2t and 2t+1 of the block,
// consistently for A and B.  That makes an accumulator tile (thread holds columns 2t, 2t+1)
// directly usable as the A operand of the next product, and turns every shared-memory
// operand fetch along the contraction index into one 8-byte load.

// A operand from an accumulator tile whose 8 columns are the contraction block.
template <int PREC> __device__ __forceinline__ FragA<PREC> fragA_from_acc(const float (&c)[4]) {
    FragA<PREC> f;
    f.x[0].set(c[0]);  // (g,   2t)
    f.x[1].set(c[2]);  // (g+8, 2t)
    f.x[2].set(c[1]);  // (g,   2t+1)
    f.x[3].set(c[3]);  // (g+8, 2t+1)
    return f;
}

// Column swizzle of the fp32 tiles of the backward kernels.  A tile is read in two ways: along the
// contraction index (lanes = rows g, 8-byte loads at columns 2t) and across it (lanes = columns g,
// rows 2t and 2t+1).
// X = 1, for row strides of 8 or 24 mod 32 words (the padded operand and score tiles): the first
//   pattern is conflict-free by the padding, in the second rows 2t and 2t+4 fall on the same banks;
//   XOR-ing the column with 8 for rows 4..7 of every block of 8 rows separates them.
// Groups of 8 floats stay contiguous under it.  X = 0: plain layout.
template <int X> __device__ __forceinline__ int xcol(int row, int col) {
    return X == 1 ? (col ^ ((row & 4) << 1)) : col;
}

// A operand from memory laid out [m][k] (row stride ld floats), rows m0+g, m0+g+8, block k0.
// The loaders' template argument R says the source was stored through pre<PREC>(), X that the
// tile carries the column swizzle above.
template <int PREC, bool R = false, int X = 0>
__device__ __forceinline__ FragA<PREC> fragA_mk(const float* p, int ld, int m0, int k0, int g, int t) {
    FragA<PREC> f;
    float2 lo = *reinterpret_cast<const float2*>(p + (m0 + g) * ld + xcol<X>(m0 + g, k0 + 2 * t));
    float2 hi = *reinterpret_cast<const float2*>(p + (m0 + g + 8) * ld + xcol<X>(m0 + g + 8, k0 + 2 * t));
    f.x[0].template put<R>(lo.x); f.x[1].template put<R>(hi.x); f.x[2].template put<R>(lo.y); f.x[3].template put<R>(hi.y);
    return f;
}

// A operand from memory laid out [k][m] (the transpose), rows k0+2t, k0+2t+1, columns m0+g, m0+g+8.
template <int PREC, bool R = false, int X = 0>
__device__ __forceinline__ FragA<PREC> fragA_km(const float* p, int ld, int m0, int k0, int g, int t) {
    FragA<PREC> f;
    const int k = k0 + 2 * t;
    const float *r0 = p + k * ld, *r1 = r0 + ld;
    f.x[0].template put<R>(r0[xcol<X>(k, m0 + g)]); f.x[1].template put<R>(r0[xcol<X>(k, m0 + g + 8)]);
    f.x[2].template put<R>(r1[xcol<X>(k + 1, m0 + g)]); f.x[3].template put<R>(r1[xcol<X>(k + 1, m0 + g + 8)]);
    return f;
}

// B operand from memory laid out [n][k]: row n0+g, block k0 (one 8-byte load).
template <int PREC, bool R = false, int X = 0>
__device__ __forceinline__ FragB<PREC> fragB_nk(const float* p, int ld, int n0, int k0, int g, int t) {
    FragB<PREC> f;
    float2 v = *reinterpret_cast<const float2*>(p + (n0 + g) * ld + xcol<X>(n0 + g, k0 + 2 * t));
    f.x[0].template put<R>(v.x); f.x[1].template put<R>(v.y);
    return f;
}

// B operand from memory laid out [k][n]: rows k0+2t, k0+2t+1, column n0+g.
template <int PREC, bool R = false, int X = 0>
__device__ __forceinline__ FragB<PREC> fragB_kn(const float* p, int ld, int n0, int k0, int g, int t) {
    FragB<PREC> f;
    const int k = k0 + 2 * t;
    f.x[0].template put<R>(p[k * ld + xcol<X>(k, n0 + g)]); f.x[1].template put<R>(p[(k + 1) * ld + xcol<X>(k + 1, n0 + g)]);
    return f;
}

// exp and reciprocal on the special-function unit (one MUFU instruction each, relative error about 2^-22) for the
// WKV7 kernels, whose XU pipe is otherwise idle (TF32 rounding is done with integer instructions).
__device__ __forceinline__ float exp_mufu(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fminf(fmaxf(x, -80.f), 80.f) * 1.4426950408889634f));
    return y;
}
__device__ __forceinline__ float rcp_mufu(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// exp() and 1/x by precision class: MUFU for the single-TF32 class, libdevice for the fp32 class.
template <int PREC> __device__ __forceinline__ float exp_p(float x) { return PREC == 3 ? expf(x) : exp_mufu(x); }
template <int PREC> __device__ __forceinline__ float rcp_p(float x) { return PREC == 3 ? 1.f / x : rcp_mufu(x); }
// P~ = 2^64 exp(c) for a running log-decay c <= 0 (clamped at MIN_CUM_LOG_DECAY).  fp32 class: exact power-of-two scaling
// of expf(c) wherever that has not underflowed.
template <int PREC> __device__ __forceinline__ float decay_up(float c) {
    if (PREC == 3) return expf(c >= -80.f ? c : fmaxf(c, MIN_CUM_LOG_DECAY) + ANCHOR_LN) * (c >= -80.f ? STATE_UNSCALE : 1.f);
    return exp_mufu(c + ANCHOR_LN);  // exp_mufu clamps its argument at -80
}

// ---- decay scan (state-independent chunk preparation, shared by forward and backward) ----------
// 8 consecutive IO elements (16 or 32 bytes) -> floats
template <typename T> __device__ __forceinline__ void load8(const unsigned char* p, float (&f)[8]);
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const unsigned char* p, float (&f)[8]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <> __device__ __forceinline__ void load8<float>(const unsigned char* p, float (&f)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 16);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// Eight floats of a row in two 16-byte stores.  With the 72-float row pitch rows r and r + 4 start on the same banks
// (also under the column swizzle, which moves both by the same 8 floats), and the eight lanes of a quarter-warp are
// rows r..r+7: `flip` (set for rows 4..7 of every eight) makes those lanes store their second half first, so that
// each of the two instructions touches eight different 16-byte bank groups.
__device__ __forceinline__ void store8(float* p, const float (&f)[8], bool flip = false) {
    float x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = flip ? f[4 + i] : f[i];  // goes out first
        y[i] = flip ? f[i] : f[4 + i];
    }
    const int off = flip ? 4 : 0;
    *reinterpret_cast<float4*>(p + off) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(p + (4 - off)) = make_float4(y[0], y[1], y[2], y[3]);
}

// One thread = one time step x 8 adjacent key channels (lane = row + 16 * channel-half, warp =
// 16-channel group).  The running log-decay along the 16 time rows is a 4-step warp-shuffle scan,
// eight independent channels per thread keep the pipes busy, and all shared-memory traffic is 16
// bytes wide.  Writes wq = q*P_t, wa = a*P_{t-1}, kwi = k/P_t, bwi = b/P_t (row stride OPS), the
// chunk decay fw = P_L, and optionally the running log-decay (fp32 class: P~_t itself) and the per-step log-decay.
// tq/tw/tk/ta/tb: staging tiles with row stride `rowb` bytes.
// live: number of time steps of this chunk that exist (16 except in the last chunk of a sequence whose length
// is not a multiple of 16); rows beyond it carry zero inputs and a per-step log-decay of zero, so that the state
// passes through them unchanged.
template <typename IoT, int PREC, int X = 0>
__device__ __forceinline__ void decay_scan(const unsigned char* tq, const unsigned char* tw, const unsigned char* tk,
                                           const unsigned char* ta, const unsigned char* tb, int rowb, float* wq, float* wa,
                                           float* kwi, float* bwi, float* fw, float* cum_out, float* lw_out, int warp, int lane,
                                           int live = L) {
    const int row = lane & 15, j0 = 16 * warp + 8 * (lane >> 4);
    const int off = row * rowb + j0 * (int)sizeof(IoT);
    float lw[8], cum[8], q[8], k[8], a[8], b[8];
    load8<IoT>(tw + off, lw);
    load8<IoT>(tq + off, q);
    load8<IoT>(tk + off, k);
    load8<IoT>(ta + off, a);
    load8<IoT>(tb + off, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) lw[i] = row < live ? fmaxf(-exp_p<PREC>(lw[i]), MIN_STEP_LOG_DECAY) : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) cum[i] = lw[i];
#pragma unroll
    for (int d = 1; d < 16; d <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float up = __shfl_up_sync(0xffffffffu, cum[i], d, 16);
            if (row >= d) cum[i] += up;
        }
    // P_t from one exp (argument clamped so that P_t and 1/P_t stay finite), 1/P_t from a reciprocal.
    float o[4][8], pt[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float incl = pt[i] = decay_up<PREC>(cum[i]);   // P~_t
        const float inv = rcp_p<PREC>(incl);
        // P_{t-1} = exp(cum_t - lw_t) (row 0: exp(0) = 1): one more exponential on the idle special-function unit is
        // cheaper here than fetching the row above with a shuffle
        const float non = decay_up<PREC>(cum[i] - lw[i]);
        o[0][i] = pre<PREC>(q[i] * incl);
        o[1][i] = pre<PREC>(a[i] * non);
        o[2][i] = pre<PREC>(k[i] * inv);
        o[3][i] = pre<PREC>(b[i] * inv);
        if (row == 15) fw[j0 + i] = incl;  // P~_16 = 2^64 P_16: users multiply by it first and by 2^-64 afterwards
    }
    const int at = row * OPS + xcol<X>(row, j0);
    const bool flip = (row >> 2) & 1;
    store8(wq + at, o[0], flip);
    store8(wa + at, o[1], flip);
    store8(kwi + at, o[2], flip);
    store8(bwi + at, o[3], flip);
    if (cum_out) store8(cum_out + at, PREC == 3 ? pt : cum, flip);
    if (lw_out) store8(lw_out + at, lw, flip);
}

// Two fp32 operations in one instruction (sm_100 packed arithmetic).
struct F2 { float x, y; };
__device__ __forceinline__ unsigned long long f2_bits(F2 a) { unsigned long long r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y)); return r; }
__device__ __forceinline__ F2 f2_from(unsigned long long r) { F2 a; asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r)); return a; }
__device__ __forceinline__ F2 f2(float x, float y) { return F2{x, y}; }
__device__ __forceinline__ F2 mul2(F2 a, F2 b) { unsigned long long r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b))); return f2_from(r); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) { unsigned long long r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b))); return f2_from(r); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { unsigned long long r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c))); return f2_from(r); }
// 8 bf16 values of a staging tile as four pairs
__device__ __forceinline__ void load8f2(const unsigned char* p, F2 (&f)[4]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = f2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}
__device__ __forceinline__ void load4f2(const unsigned char* p, F2 (&f)[2]) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    f[0] = f2(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u));
    f[1] = f2(__uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Column `col` of AI = (I - AB)^-1 for a strictly lower-triangular 16x16 AB, one lane per column.
// ABt holds AB TRANSPOSED (ABt[s][tq] = AB[tq][s], row stride SCS), so that everything step s needs
// is one contiguous row.  Right-looking substitution: as soon as entry s is final it is pushed
// into all later rows, so the dependent chain is 16 steps long rather than 120.
template <int S_> __device__ __forceinline__ void tri_fetch_row(float (&dst)[L], const float* ABt) {
    // entries tq > S_ of row S_ of ABt, in 16-byte pieces
#pragma unroll
    for (int v = (S_ + 1) / 4; v < L / 4; ++v) {
        const float4 x = *reinterpret_cast<const float4*>(ABt + S_ * SCS + 4 * v);
        dst[4 * v] = x.x; dst[4 * v + 1] = x.y; dst[4 * v + 2] = x.z; dst[4 * v + 3] = x.w;
    }
}
template <int PREC, int S_, int X>
__device__ __forceinline__ void tri_step(float (&r)[L], const float (&c)[L], float (&cn)[L], const float* ABt, float* AI, int col) {
    if (S_ + 1 < L) tri_fetch_row<(S_ + 1 < L ? S_ + 1 : 0)>(cn, ABt);  // one step ahead of its use
    const float ms = r[S_];
    AI[S_ * SCS + xcol<X>(S_, col)] = pre<PREC>(ms);
#pragma unroll
    for (int tq = S_ + 1; tq < L; ++tq) r[tq] = fmaf(c[tq], ms, r[tq]);
}
template <int PREC, int X = 0> __device__ __forceinline__ void tri_inverse_column(const float* ABt, float* AI, int col) {
    float r[L], ca[L], cb[L];
#pragma unroll
    for (int tq = 0; tq < L; ++tq) r[tq] = (tq == col) ? 1.f : 0.f;
    tri_fetch_row<0>(ca, ABt);
    tri_step<PREC, 0, X>(r, ca, cb, ABt, AI, col);   tri_step<PREC, 1, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 2, X>(r, ca, cb, ABt, AI, col);   tri_step<PREC, 3, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 4, X>(r, ca, cb, ABt, AI, col);   tri_step<PREC, 5, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 6, X>(r, ca, cb, ABt, AI, col);   tri_step<PREC, 7, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 8, X>(r, ca, cb, ABt, AI, col);   tri_step<PREC, 9, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 10, X>(r, ca, cb, ABt, AI, col);  tri_step<PREC, 11, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 12, X>(r, ca, cb, ABt, AI, col);  tri_step<PREC, 13, X>(r, cb, ca, ABt, AI, col);
    tri_step<PREC, 14, X>(r, ca, cb, ABt, AI, col);  tri_step<PREC, 15, X>(r, cb, ca, ABt, AI, col);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait for the phase of an mbarrier with the given parity, of all kernels but the tcgen05 forward, which has one of its own
// (mbar_wait in wkv7_fwd_tc.cu: the same limits, a poll interval of 40 ns, the status word written when the CTA ends).
// Returns at once, false, when the CTA has aborted.  When `limit` clocks pass without the phase completing it raises the
// CTA's abort flag (every later wait then falls through), records kDeviceTimeout in the device status word and
// returns: a lost copy or a missing arrival ends with an error code, never with a hung GPU.
// SLEEP: 100 ns between polls, for warps that wait for long beside others that work.
constexpr long long MBAR_WAIT_LIMIT = 1LL << 28;  // clocks (~0.14 s): far beyond any legitimate wait within a CTA
// The wait for another CTA's half of a cut chain (wait_handoff below) may legitimately take longer: the CTAs of one launch run at
// different speeds when other work shares the GPU with them, and a range of work can be 0.1 s long.  The waits of the same CTA that
// stand still meanwhile are given more again, so that the one that gives up is the one whose condition is missing.
constexpr long long HANDOFF_WAIT_LIMIT = 4 * MBAR_WAIT_LIMIT;         // 0.55 s
constexpr long long ACROSS_HANDOFF_LIMIT = 2 * HANDOFF_WAIT_LIMIT;    // 1.1 s
static_assert(MBAR_WAIT_LIMIT < HANDOFF_WAIT_LIMIT && HANDOFF_WAIT_LIMIT < ACROSS_HANDOFF_LIMIT, "see above");
static_assert(ACROSS_HANDOFF_LIMIT <= 1LL << 31, "mbar_wait_bounded counts in 32 bits");
__device__ __forceinline__ void give_up(volatile int* abort, int* status) {
    *abort = 1;
    *reinterpret_cast<volatile int*>(status) = (int)kDeviceTimeout;  // the launchers always pass the status word (host-visible)
    __threadfence_system();
}
template <bool SLEEP>
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort, int* status, long long limit = MBAR_WAIT_LIMIT) {
    const uint32_t addr = smem_u32(bar);
    const uint32_t start = clock(), most = (uint32_t)limit;
    uint32_t spin = 0;
    // (The loop is kept as small as it can be: it is inlined at many places of kernels whose loops fill the instruction cache; with
    // 64-bit clocks it was 1 KB a place.)
    for (;;) {
        uint32_t ok;
        asm volatile("{\n.reg .pred P;\nmbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\nselp.u32 %0, 1, 0, P;\n}\n"
                     : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
        if (*abort) return false;
        if (SLEEP) __nanosleep(100);
        if ((SLEEP || (++spin & 63) == 0) && (uint32_t)clock() - start > most) break;
    }
    give_up(abort, status);
    return false;
}

// Every thread that issues bulk loads ends with one of these: shared memory must outlive the loads also where a wait has given up and
// nobody waits for them any more (otherwise they landed long ago).  They rely on no load being issued on a barrier whose last phase is
// still open, so a thread whose wait returned false issues no more.  `never_set` takes the place of the abort flag.
// The `issued` loads that went to `bar`, a phase each:
__device__ __forceinline__ void mbar_landed(uint64_t* bar, int issued, volatile int* never_set, int* status) {
    if (issued > 0) mbar_wait_bounded<true>(bar, (issued - 1) & 1, never_set, status);
}
// the same for a ring of S barriers that take the loads in turn:
template <int S> __device__ __forceinline__ void ring_landed(uint64_t* ring, int issued, volatile int* never_set, int* status) {
#pragma unroll 1
    for (int s = 0; s < S; ++s) mbar_landed(ring + s, (issued + S - 1 - s) / S, never_set, status);
}
// and where nobody has counted, in a CTA that has aborted: the open phase, if there is one, has one of the two parities; the wait
// for the other one returns at once before it and runs out after it.
__device__ __forceinline__ void mbar_landed_uncounted(uint64_t* bar, volatile int* never_set, int* status) {
    mbar_wait_bounded<true>(bar, 0, never_set, status);
    mbar_wait_bounded<true>(bar, 1, never_set, status);
}

// Kernels are launched such that they may start before the one ahead of them in the stream has ended (launch() in wkv7_kernels.h), and
// call stream_wait() before they touch global memory: what stands before it - barriers, tensor memory - and the launch itself then overlap
// the other kernel's end.  From stream_release() on, called by at least one thread of each CTA or left to the CTA's end, the next kernel
// may start, which will in turn wait until this one has ended (a kernel that is not launched so waits by itself).  All CTAs of this kernel
// are then running or have ended, so that none of them has to wait for a place that a CTA of the next one holds; for the same reason
// tensor memory is allocated before stream_wait().
// A kernel releases the next one only when it has waited itself, so that no more than one of a stream waits; and kernels whose CTAs walk many
// chunks release it with their last ones, a few us before they end.  Otherwise the next one's CTAs hold the shared memory of all SMs that
// a few chains leave idle for as long as those take, and other streams stand still: beside the backward of 12 chains of 1024 chunks
// (990 us) a forward of 64 chains on another stream is done after 180 to 200 us, with the release at the kernels' start it was after 990;
// beside twelve forwards of 37 chains of 512 chunks (360 us each) after 195 us instead of 750.  One stream alone: no case slower.
__device__ __forceinline__ void stream_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void stream_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void stream_order() {  // of a kernel with little to do in each CTA
    stream_wait();
    stream_release();
}
// A __restrict__ pointer of a kernel that waits: without this the compiler may move loads through it ahead of the wait, which it takes not to
// touch what such a pointer alone leads to.  (Pointers that are not __restrict__ need nothing, and what is written is not.)
template <typename T> __device__ __forceinline__ T* after_stream_order(T* p) {
    asm volatile("" : "+l"(p) :: "memory");
    return p;
}

__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred P;\nelect.sync _|P, 0xffffffff;\nselp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
    return p;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16-byte asynchronous copy global -> shared through the load/store unit (no TMA request)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
// The same copy for a row that may lie beyond the end of the sequence: when `live` is false nothing is read and the
// 16 bytes are filled with zeros (the source address must still be a valid one).
__device__ __forceinline__ void cp_async16_zfill(void* smem, const void* gmem, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }


// ---- how chains are spread over the CTAs ---------------------------------------------------------
// A chain is serial in time, but nothing ties a whole chain to one CTA.  With one chain per CTA, B*H chains on S resident
// CTAs take ceil(B*H / S) rounds, and the last round is rarely full (768 chains on 148 SMs: 6 rounds for 5.19 rounds' worth
// of work).  So the chunks of all chains, chain after chain, are cut into S equal ranges, one per CTA (the wrap-around
// rule of preemptive scheduling).  A range is [the end of a chain | whole chains | the start of a chain]; the CTA works the
// START piece first and the END piece last.  The two pieces of a cut chain belong to neighbouring CTAs: CTA i works the
// start at the beginning of its time and leaves the state in the chain's final-state buffer, CTA i + 1 takes it up at
// the end of its time.  A chain is no longer than a range, so the start is finished by the time the end is due (equal
// speeds assumed; otherwise the wait is short, and bounded).  Results are bit for bit those of the uncut chain.
// CTA i only ever waits for CTA i - 1, which was dispatched before it, and which waits for nothing before it publishes.
struct WorkSplit {
    int ctas, per_cta, per_chain, total;  // CTAs; chunks per range (the last may be shorter); chunks per chain; chunks in all
    unsigned* flags;                      // one word per CTA, zero at launch: the state of its start piece is ready; null: no chain is cut
};
struct WorkRange {
    int first, n, h, t;  // first chunk (chain-major), chunks, chunks in the start piece (worked first), in the end piece (worked last)
    __device__ __forceinline__ WorkRange(const WorkSplit& s, int cta) {
        first = cta * s.per_cta;
        n = min(s.per_cta, s.total - first);
        h = (first + n) % s.per_chain;
        t = (s.per_chain - first % s.per_chain) % s.per_chain;
    }
    // chain and chunk (in processing order) of position v of the CTA's work
    __device__ __forceinline__ void locate(int v, int per_chain, int& chain, int& chunk) const {
        const int x = v < h ? first + n - h + v : v < n - t ? first + t + v - h : first + v - (n - t);
        chain = (int)((unsigned)x / (unsigned)per_chain);
        chunk = x - chain * per_chain;
    }
    // whether position v, whose chunk is `chunk`, does not continue the chain of position v - 1
    __device__ __forceinline__ bool starts_segment(int v, int chunk) const { return v == 0 || chunk == 0 || (t > 0 && v == n - t); }
};
__device__ __forceinline__ void publish_handoff(unsigned* flag) {
    asm volatile("st.release.gpu.global.u32 [%0], 1;" ::"l"(flag) : "memory");
}
// Bounded like every wait of this library (see mbar_wait_bounded and HANDOFF_WAIT_LIMIT).
__device__ __forceinline__ void wait_handoff(const unsigned* flag, volatile int* abort, int* status) {
    const long long start = clock64();
    for (;;) {
        unsigned ready;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(ready) : "l"(flag) : "memory");
        if (ready || *abort) return;
        if (clock64() - start > HANDOFF_WAIT_LIMIT) {
            give_up(abort, status);
            return;
        }
        __nanosleep(200);
    }
}

// Tensor addressing shared by all launchers: element (b,t,h,0) of a [B,T,H,N] tensor.
struct Strides {
    long long b, t, h;  // in elements
};

}  // namespace wkv7
