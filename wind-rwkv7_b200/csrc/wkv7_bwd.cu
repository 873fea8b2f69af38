// WKV7 backward for sm_100a, fp32 tensors (single or triple TF32 products; bf16 tensors: wkv7_bwd_bf16.cu): one CTA per
// (batch, head) chain, 4 warps, chunks of 16 time steps walked in reverse; the gradient dS of the state stays in registers.
// attn with triple TF32 and scratch: dS is walked by a kernel of its own (wkv7_bwd_walk32_kernel), then all chunks are worked in
// parallel (PAR).
//
// Replaces the reference's backward_kernel (wind_rwkv/rwkv7/attn.cu:131-326).  The forward
// intermediates of a chunk are rebuilt from the fp32 chunk-start state S0 the forward wrote (exact fp32; in the
// single-TF32 class the tensor core reads the upper 19 bits of it as an operand, no conversion instruction).
// With the forward's notation (wq, wa, kwi, bwi, fw, QK, QB, AK, AB, AI = (I-AB)^-1, U) and
// dSf = dS * fw[None,:]:
//     du   = QB^T dY + bwi dSf^T          dabu = AI^T du
//     dV   = QK^T dY + kwi dSf^T + AK^T dabu
//     dAB = stril(dabu U^T)  dAK = stril(dabu V^T)  dQB = tril(dY U^T)  dQK = tril(dY V^T)
//     DA = dAB bwi + dAK kwi + dabu S0     DQ = dQB bwi + dQK kwi + dY S0
//     DB = dAB^T wa + dQB^T wq + U dSf     DK = dAK^T wa + dQK^T wq + V dSf
//     da = P_{t-1} DA   dq = P_t DQ   db = DB / P_t   dk = DK / P_t
//     dS0 = dSf + dY^T wq + dabu^T wa
// The decay gradient uses that w enters only through the running log-decay c_t = sum_{s<=t}
// -exp(w_s): every scaled operand is (input * exp(+-c)), so
//     d/dc_t = wq.DQ - kwi.DK - bwi.DB (row t) + wa.DA (row t+1),   d/dc_L += sum_i dS[i,:] S'[i,:]
// and dlogdecay_k = sum_{t>=k} d/dc_t; dw = dlogdecay * (-exp(w)).  The last term for chunk c-1
// equals sum_i dS0_c[i,:] S0_c[i,:], which is formed while chunk c is processed and carried.
//
// With LN = true the kernel is the backward of the fused attn_ln op (reference:
// wind_rwkv/rwkv7/attn_ln.cu:40-104, 237-464): `dy` is then the gradient of the fused output; the
// chunk's recurrence output Y is rebuilt, the GroupNorm / bonus / gate backward runs on it in the
// transposed register layout (three cross-warp reductions per time step through shared memory),
// and its result replaces dY for everything below.  Parameter gradients are accumulated in
// registers over the whole chain and written as per-(batch, head) partials (no atomics).
//
// Stage B (rows = value index, per warp, no cross-warp traffic): U^T, du^T, dabu^T, dV^T, dS0.
// Stage C (contractions over the value index, warp owns 16 key columns): the four score
// gradients and DA, DQ, DB, DK with S0 and dSf read from shared memory.
#include <cuda.h>
#include <algorithm>
#include <cstddef>
#include <cstring>

#include "wkv7_kernels.h"

namespace wkv7 {

struct alignas(64) CkptMaps { CUtensorMap ck, ckm; };  // checkpoint states, matrices

constexpr int SS = N + 8;  // row stride (floats) of the [value][key] state buffers
constexpr int MAT_BLK = 8 * 4 * SCS;  // floats per block of the matrices buffer
static_assert(SCS == L + 8, "the matrix loads copy boxes of L + 8 floats per row");
// All fp32 tiles of this kernel (operands, scores, score gradients, U, dabu, the two state buffers)
// carry the column swizzle xcol<1>() of wkv7_common.cuh: each is read both along and across its
// contraction index.

// Staging tiles [time][channel]: 256-byte rows padded by 16 bytes.
constexpr int ROWB = N * 4 + 16, TILEB = L * ROWB;
constexpr int YS = 20;  // row stride (floats) of the per-warp transposition scratch
__device__ __forceinline__ int st_at(int row, int col) { return row * ROWB + col * 4; }  // byte offset of element (row, col)

// PAR: two CTAs an SM (3072 chunks: 148 us; with one, 233): v and dy in one set, requested after stage C; the score gradients in the place of
// the matrices, which come after the chunk's last barrier.
template <int PREC, bool LN, bool PAR> struct BwdSmem {
    static constexpr int SETS = PAR ? 1 : 2;
    alignas(16) unsigned char st_in[5][TILEB];  // q, w, k, a, b (dead after the scan)
    alignas(16) unsigned char st_v[SETS][TILEB];
    alignas(16) unsigned char st_dy[SETS][TILEB];
    alignas(16) unsigned char st_g[LN ? 2 : 1][LN ? TILEB : 16];
    alignas(16) float wq[L * OPS], wa[L * OPS], kwi[L * OPS], bwi[L * OPS];
    alignas(16) float cum[L * OPS];                  // running log-decay; fp32 class: P~_t
    alignas(16) float lw[PREC == 3 ? L * OPS : 4];   // single-TF32 path derives it from cum
    // The chunk's four 16x16 matrices AK, QK, AI^T, QB (matrix m, row r: row group 2m + r/8 of the record's 64-row operand
    // tile), filled by two bulk tensor loads: rows with (r & 4) == 0 form a dense block of [8 row groups][4 rows][24 floats]
    // (16 values, 8 floats of fill), the other rows a second block whose rows start with the fill.  See mat_at().
    alignas(128) float mats[2 * MAT_BLK];
    // Score gradients (stage C).  While stage B runs they are dead, and the same bytes serve as
    // the per-warp transposition scratch for dv / dg and as the GroupNorm reduction buffers.
    static constexpr int SCRATCH_FLOATS = WARPS * L * YS + WARPS * L * 5;
    static constexpr int SGRAD_FLOATS = 4 * L * SCS > SCRATCH_FLOATS ? 4 * L * SCS : SCRATCH_FLOATS;
    alignas(16) float sgrad_[PAR ? 4 : SGRAD_FLOATS];
    __device__ __forceinline__ float* sgrad() { return PAR ? mats : sgrad_; }  // score gradient i at sgrad() + i * L * SCS
    static_assert(!PAR || 4 * L * SCS <= 2 * MAT_BLK, "room for the score gradients");
    // attn_ln: Ut, Dt, Yt are dead between stage C and the next chunk's stage B and double as the output staging tiles
    alignas(LN ? 1024 : 16) float Ut[L * OPS];  // U and dabu as [time][value]
    alignas(16) float Dt[L * OPS];
    alignas(16) float Yt[LN ? L * OPS : 4];      // recurrence-output gradient as [time][value]
    // Chunk-start state [value][key], filled by two bulk tensor loads per chunk: rows with (row & 4) == 0 form a dense
    // block of 32 rows x 72 floats (64 values, 8 floats of fill), the other rows a second block whose rows start with
    // the 8 floats of fill (the load starts at column -8).  See s0_at().
    alignas(128) float S0s[N * SS];
    alignas(16) float dSs[N * SS];  // dSf as [value][key], column swizzle 1
    alignas(8) uint64_t s0_bar;     // completion of the state loads
    volatile int abort, zero;       // abort: set when a bounded wait gave up; zero stays 0 (see mbar_landed_uncounted)
    alignas(16) float fw[N];
    alignas(16) float Gp[2][WARPS][N];
    alignas(16) float lnp[LN ? 3 * N : 4];
    float bdot[L], sbon[L];
};

__device__ __forceinline__ float bst_elem(const unsigned char* tile, int row, int col) { return *reinterpret_cast<const float*>(tile + st_at(row, col)); }
// two adjacent elements (col even) of a staging tile
__device__ __forceinline__ float2 bst_pair(const unsigned char* tile, int row, int col) { return *reinterpret_cast<const float2*>(tile + st_at(row, col)); }
// A operand [m = time][k = value] straight from a staging tile laid out [time][value]
template <int PREC> __device__ __forceinline__ FragA<PREC> fragA_mk_st(const unsigned char* tile, int k0, int g, int t4) {
    FragA<PREC> f;
    float2 lo = bst_pair(tile, g, k0 + 2 * t4), hi = bst_pair(tile, g + 8, k0 + 2 * t4);
    f.x[0].set(lo.x); f.x[1].set(hi.x); f.x[2].set(lo.y); f.x[3].set(hi.y);
    return f;
}
// B operand [k = value][n = time] from a staging tile laid out [time][value]
template <int PREC> __device__ __forceinline__ FragB<PREC> fragB_nk_st(const unsigned char* tile, int n0, int k0, int g, int t4) {
    FragB<PREC> f;
    float2 v = bst_pair(tile, n0 + g, k0 + 2 * t4);
    f.x[0].set(v.x); f.x[1].set(v.y);
    return f;
}
// A operand [m = value][k = time] (the transpose) from a staging tile laid out [time][value]
template <int PREC> __device__ __forceinline__ FragA<PREC> fragA_km_st(const unsigned char* tile, int m0, int k0, int g, int t4) {
    FragA<PREC> f;
    const int tr = k0 + 2 * t4, vc = m0 + g;
    f.x[0].set(bst_elem(tile, tr, vc));
    f.x[1].set(bst_elem(tile, tr, vc + 8));
    f.x[2].set(bst_elem(tile, tr + 1, vc));
    f.x[3].set(bst_elem(tile, tr + 1, vc + 8));
    return f;
}

// Epilogue stores.  A thread holds columns (2*t4, 2*t4+1) of two adjacent 8-column tiles; stored as they
// are, a warp-wide store writes 16 bytes per row (half a 32-byte sector).  Lanes t4 and t4^1 swap one
// pair, after which the even lane holds columns 4m..4m+3 of the first tile and the odd lane the same
// columns of the second tile (m = t4 / 2): 16-byte stores, whole sectors per row.
// `row` points at column 16*warp of the output row; live = false (rows beyond the end of the sequence) keeps the
// exchange but skips the store.
__device__ __forceinline__ void store_quad(float* row, float a0, float a1, float b0, float b1, int t4, bool live) {
    const bool odd = t4 & 1;
    const float g0 = __shfl_xor_sync(0xffffffffu, odd ? a0 : b0, 1), g1 = __shfl_xor_sync(0xffffffffu, odd ? a1 : b1, 1);
    const float4 v = odd ? make_float4(g0, g1, b0, b1) : make_float4(a0, a1, g0, g1);
    if (live) *reinterpret_cast<float4*>(row + 8 * (t4 & 1) + 4 * (t4 >> 1)) = v;
}

// Offset of element (row = value, col = key) of the chunk-start state in shared memory.  With the 72-float row pitch
// (8 banks) both access patterns of the tensor-core fragments are free of bank conflicts: lanes over rows g = 0..3 or
// 4..7 of one block with 8-byte loads, and lanes over rows 0,2,4,6 (or 1,3,5,7) x 8 columns, where the second block's
// shift by 8 floats separates rows r and r + 4.
constexpr int S0_BLK = 32 * SS;
// Offset of element (row, col) of matrix m (0 AK, 1 QK, 2 AI^T, 3 QB) in the matrices buffer; the same split by row bit 2
// and the same shift of the second block by 8 floats as for the state, here with the 24-float row pitch.
__device__ __forceinline__ int mat_at(int m, int row, int col) {
    return ((row >> 2) & 1) * (MAT_BLK + 8) + ((2 * m + (row >> 3)) * 4 + (row & 3)) * SCS + col;
}
__device__ __forceinline__ int s0_at(int row, int col) {
    return ((row >> 2) & 1) * (S0_BLK + 8) + (((row >> 3) << 2) | (row & 3)) * SS + col;
}
static_assert(SS == N + 8, "the state loads copy boxes of N + 8 floats per row");

// Waits (polling, bounded) for a phase of the state-load barrier: the library's common wait, which the forward's
// self-test exercises on barriers nothing arrives on.
__device__ __forceinline__ bool s0_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* status) {
    return mbar_wait_bounded<false>(bar, parity, abort, status);
}

// PAR: the state gradients at the chunks' ends are given (wkv7_bwd_walk32_kernel), so that no chunk depends on another one and a CTA
// takes `per` of the list of all chains' steps it0 .. it0 + count - 1 (counted from the end of the sequence).
struct Walked { const float* tiles; int it0, count, per, total; };
constexpr int TILE_FLOATS = N * SS;  // a state gradient as the kernel keeps it in shared memory: pitch SS, columns xcol<1>
// d += a b; with SPLIT the products with a lower part go to d2
template <int PREC, bool SPLIT> __device__ __forceinline__ void mma2(float (&d)[4], float (&d2)[4], const FragA<PREC>& a, const FragB<PREC>& b) {
    if (!SPLIT) {
        mma<PREC>(d, a, b);
        return;
    }
    mma_tf32_raw(d2, a.x[0].l, a.x[1].l, a.x[2].l, a.x[3].l, b.x[0].h, b.x[1].h);
    mma_tf32_raw(d, a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].h, b.x[1].h);
    mma_tf32_raw(d2, a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].l, b.x[1].l);
}
// TAIL: the sequence length is not a multiple of 16 (an instantiation of its own, so that whole-chunk sequences carry
// none of the row tests).
template <int PREC, bool LN, bool TAIL, bool PAR>
__global__ void __launch_bounds__(THREADS, PAR ? 2 : 1) wkv7_bwd_kernel(BwdParams p, Walked wk, const __grid_constant__ CkptMaps cmaps) {
    stream_wait();
    if (PAR) stream_release();  // (all SMs are full; with the last chunk, as below: B8 T512 H12 forward and backward 286.4 instead of 284.6 us)
    static_assert(!(PAR && LN), "attn_ln's state gradient needs the gradient of the recurrence output first");
    using Smem = BwdSmem<PREC, LN, PAR>;
    static_assert(!PAR || sizeof(Smem) + 1024 <= 116736, "two CTAs per SM");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const long long bh = blockIdx.x;  // (not PAR)
    const long long bi = bh / p.H, hi = bh % p.H;
    const long long base = PAR ? 0 : bi * p.st.b + hi * p.st.h;
    const int nchunks = (int)((p.T + L - 1) / L);  // the last chunk may be partial: its missing rows read as zeros
    constexpr bool has_tail = TAIL;
    const float* gin[5] = {(const float*)p.r + base, (const float*)p.w + base, (const float*)p.k + base,
                         (const float*)p.a + base, (const float*)p.b + base};
    const float* gv = (const float*)p.v + base;
    const float* gdy = (const float*)p.dy + base;
    float* gout[5] = {(float*)p.dr + base, (float*)p.dw + base, (float*)p.dk + base, (float*)p.da + base, (float*)p.db + base};
    float* gdv = (float*)p.dv + base;
    // position `it` of the CTA's list: chain, chunk, and (PAR) element offset of the chain
    struct Item { long long bh, off; int c, t; };
    const int items = PAR ? min(wk.per, wk.total - (int)blockIdx.x * wk.per) : nchunks;
    auto item = [&](int it) {
        if (!PAR) return Item{bh, 0, nchunks - 1 - it, it};
        const int x = (int)blockIdx.x * wk.per + it, chain = (int)((unsigned)x / (unsigned)wk.count), t = x - chain * wk.count;
        const int b = (int)((unsigned)chain / (unsigned)p.H);
        return Item{chain, b * p.st.b + (chain - b * (int)p.H) * p.st.h, nchunks - 1 - wk.it0 - t, t};
    };
    const float* gg = LN ? (const float*)p.g + base : nullptr;
    float* gdg = LN ? (float*)p.dg + base : nullptr;
    constexpr uint32_t ROW_BYTES = N * 4;

    if (LN) {
        for (int i = tid; i < 3 * N; i += THREADS) sm.lnp[i] = p.params[(long long)(i / N) * p.H * N + hi * N + (i % N)];
    }
    // stage-B scratch aliased onto the score-gradient buffers
    float* const dvsc = sm.sgrad_ + (PAR ? 0 : warp * (L * YS));  // (PAR has neither)
    float* const red = sm.sgrad_ + (PAR ? 0 : WARPS * L * YS);  // [WARPS][L][2]
    float* const red2 = red + WARPS * L * 2;                                             // [WARPS][L][3]
    float dlnw_acc[2] = {0.f, 0.f}, dlnb_acc[2] = {0.f, 0.f}, dbon_acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    // Carried decay term for the last chunk: sum_i dsT[i,:] * sT[i,:] (zero without dsT).
    for (int i = tid; i < WARPS * N; i += THREADS) sm.Gp[1][i / N][i % N] = 0.f;
    if (tid == 0) {
        sm.abort = sm.zero = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.s0_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (!PAR && p.dsT && p.sT && tid < N) {
        const float* d = p.dsT + bh * N * N;
        const float* s = p.sT + bh * N * N;
        float acc = 0.f;
        for (int i = 0; i < N; ++i) acc += d[i * N + tid] * s[i * N + tid];
        sm.Gp[1][0][tid] = acc;
    }

    // iteration `it` handles chunk c = nchunks-1-it.  All threads fetch 16-byte pieces with
    // cp.async; a chunk's loads are issued one iteration ahead and waited for before the barrier
    // that ends the iteration.
    constexpr int CH = ROW_BYTES / 16;
    auto issue_in = [&](const Item& n) {
        const int c = n.c;
        for (int i = tid; i < 5 * L * CH; i += THREADS) {
            const int ten = i / (L * CH), row = (i / CH) % L, ch = i % CH;
            const long long tt = (long long)c * L + row;
            if (has_tail) cp_async16_zfill(sm.st_in[ten] + st_at(row, ch * 4),
                             reinterpret_cast<const unsigned char*>(gin[ten] + n.off + (tt < p.T ? tt : p.T - 1) * p.st.t) + ch * 16, tt < p.T);
            else cp_async16(sm.st_in[ten] + st_at(row, ch * 4), reinterpret_cast<const unsigned char*>(gin[ten] + n.off + tt * p.st.t) + ch * 16);
        }
    };
    auto issue_vdy = [&](const Item& n, int s) {
        const int c = n.c;
        for (int i = tid; i < (LN ? 3 : 2) * L * CH; i += THREADS) {
            const int ten = i / (L * CH), row = (i / CH) % L, ch = i % CH;
            const long long tt = (long long)c * L + row;
            const float* src = (ten == 0 ? gv : ten == 1 ? gdy : gg) + n.off + (!TAIL || tt < p.T ? tt : p.T - 1) * p.st.t;
            unsigned char* dst = (ten == 0 ? sm.st_v[s] : ten == 1 ? sm.st_dy[s] : sm.st_g[LN ? s : 0]) + st_at(row, ch * 4);
            if (has_tail) cp_async16_zfill(dst, reinterpret_cast<const unsigned char*>(src) + ch * 16, tt < p.T);
            else cp_async16(dst, reinterpret_cast<const unsigned char*>(src) + ch * 16);
        }
    };
    // (by thread 0, after the expectation that counts their bytes, too)
    auto issue_mats = [&](const Item& n) {
        const uint32_t bar = smem_u32(&sm.s0_bar);
        const int record = (int)(n.bh * nchunks + n.c);
        // the matrices: the record keeps them as the forward's operand tiles, 16-byte pieces [row / 8][column / 4][row % 8];
        // seen as [row group][row bit 2][row % 4][piece][4 floats], a box of 6 pieces per row (2 of them beyond the
        // row: zero fill) lands as rows of 24 floats; the second block starts at piece -2
#pragma unroll
        for (int blk = 0; blk < 2; ++blk)
            asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                         ::"r"(smem_u32(sm.mats + blk * MAT_BLK)), "l"(&cmaps.ckm), "r"(bar), "r"(0), "r"(-2 * blk), "r"(0), "r"(blk), "r"(record * (CK_FLOATS / 128) + CK_MATS / 128) : "memory");
    };
    // the checkpoint record of chunk c: its start state and its four 16x16 matrices (QK, QB, AK, AI), which the
    // forward left there so that the scores and the triangular inverse are not rebuilt here
    auto issue_s0 = [&](const Item& n) {
        if (tid == 0) {
            // two boxes of [8][4 rows][72 floats]: rows 8a + b and rows 8a + 4 + b (a < 8, b < 4); the second starts at
            // column -8, so that its fill comes first in each row
            const uint32_t bar = smem_u32(&sm.s0_bar);
            const int record = (int)(n.bh * nchunks + n.c);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(((PAR ? 2 : 1) * N * SS + 2 * MAT_BLK) * 4)) : "memory");
            if (PAR)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(sm.dSs)), "l"(wk.tiles + (n.bh * wk.count + n.t) * TILE_FLOATS), "r"(TILE_FLOATS * 4), "r"(bar) : "memory");
#pragma unroll
            for (int blk = 0; blk < 2; ++blk)
                asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                             ::"r"(smem_u32(sm.S0s + blk * S0_BLK)), "l"(&cmaps.ck), "r"(bar), "r"(-8 * blk), "r"(0), "r"(blk), "r"(0), "r"(record) : "memory");
            if (!PAR) issue_mats(n);
        }
    };
    if (items > 0) {
        issue_in(item(0));
        issue_vdy(item(0), 0);
        issue_s0(item(0));
        if (PAR && tid == 0) issue_mats(item(0));
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncthreads();

    // dS: warp owns value rows 16*warp + {g, g+8}; tile nt covers key columns 8nt..8nt+7.
    float dS[8][4];
    if (!PAR) {
        const float* d = p.dsT ? p.dsT + bh * N * N : nullptr;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            if (d) {
                float2 lo = *reinterpret_cast<const float2*>(d + (16 * warp + g) * N + 8 * nt + 2 * t4);
                float2 hi2 = *reinterpret_cast<const float2*>(d + (16 * warp + g + 8) * N + 8 * nt + 2 * t4);
                // the state gradient is carried as 2^64 dS, the counterpart of the forward's S~ = 2^-64 S (see ANCHOR_LN)
                dS[nt][0] = lo.x * STATE_UNSCALE; dS[nt][1] = lo.y * STATE_UNSCALE; dS[nt][2] = hi2.x * STATE_UNSCALE; dS[nt][3] = hi2.y * STATE_UNSCALE;
            } else {
                dS[nt][0] = dS[nt][1] = dS[nt][2] = dS[nt][3] = 0.f;
            }
        }
    }

    // this thread's offsets into the chunk-start state: rows 16*warp + g (and + 8) at columns 2*t4 + 8*block, and
    // rows 2*t4 (and + 1) + 8*block at column 16*warp + g
    const float* const s0_mk = sm.S0s + s0_at(16 * warp + g, 2 * t4);
    const float* const s0_kn = sm.S0s + s0_at(2 * t4, 16 * warp + g);
    // matrix m as a B operand: [n][k] (row 8*nt + g, columns 8*kk + 2*t4, +1) and [k][n] (rows 8*tb + 2*t4, +1, column 8*sb + g)
    const float* const mat_g = sm.mats + mat_at(0, g, 2 * t4);
    const float* const mat_t = sm.mats + mat_at(0, 2 * t4, g);
    auto mat_nk = [&](int m, int nt, int kk) {
        FragB<PREC> f;
        const float2 v = *reinterpret_cast<const float2*>(mat_g + (2 * m + nt) * (4 * SCS) + 8 * kk);
        f.x[0].setr(v.x); f.x[1].setr(v.y);
        return f;
    };
    auto mat_kn = [&](int m, int sb, int tb) {
        FragB<PREC> f;
        const float* q = mat_t + (2 * m + tb) * (4 * SCS) + 8 * sb;
        f.x[0].setr(q[0]); f.x[1].setr(q[SCS]);
        return f;
    };
    bool live = true;  // this thread has not given up a wait for a record: none is requested after that
    for (int it = 0; it < items; ++it) {
        if (!PAR && it + 1 == items) stream_release();
        const Item now = item(it);
        const int c = now.c;
        const int vs = PAR ? 0 : it & 1, gp_set = it & 1;
        // PAR: this thread's entries of the state at the chunk's end, for the carried decay term (zero for a final state that is not given)
        float2 nx[PAR ? 8 : 1][2];
        if (PAR) {
            const bool last = c + 1 == nchunks;
            const float* q = last ? (p.dsT && p.sT ? p.sT + now.bh * N * N : nullptr) : p.ckpt + (now.bh * nchunks + c + 1) * CK_FLOATS + CK_STATE;
            const float sc = last ? STATE_SCALE : 1.f;
            if (q) q += (16 * warp + g) * N + 2 * t4;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float2 v = q ? *reinterpret_cast<const float2*>(q + 8 * h * N + 8 * nt) : make_float2(0.f, 0.f);
                    nx[PAR ? nt : 0][h] = make_float2(v.x * sc, v.y * sc);
                }
        }
        // ---------------- P1: decay scan and scaled operands -------------------------------------
        {
            decay_scan<float, PREC, 1>(sm.st_in[0], sm.st_in[1], sm.st_in[2], sm.st_in[3], sm.st_in[4], ROWB, sm.wq, sm.wa,
                                  sm.kwi, sm.bwi, sm.fw, sm.cum, PREC == 3 ? sm.lw : nullptr, warp, lane,
                                  TAIL ? (int)min((long long)L, p.T - (long long)c * L) : L);
            if (LN) {  // bonus dot  sum_j r_j k_j bonus_j  per time step: 8 threads per row
                const int row = tid >> 3, part = tid & 7;
                float acc = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int ch = part * 8 + i;
                    acc += bst_elem(sm.st_in[0], row, ch) * bst_elem(sm.st_in[2], row, ch) * sm.lnp[2 * N + ch];
                }
                acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                acc += __shfl_xor_sync(0xffffffffu, acc, 2);
                acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                if (part == 0) sm.bdot[row] = acc;
            }
        }
        __syncthreads();  // (A)
        if (it + 1 < items) {
            issue_in(item(it + 1));
            if (!PAR) issue_vdy(item(it + 1), vs ^ 1);
        }

        // ---------------- stage B: rows = value index -----------------------------------------
        const unsigned char* vt = sm.st_v[vs];
        const unsigned char* dyt = sm.st_dy[vs];
        FragA<PREC> vf[2], dyf[2];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            vf[kk] = fragA_km_st<PREC>(vt, 16 * warp, 8 * kk, g, t4);
            if (!LN) dyf[kk] = fragA_km_st<PREC>(dyt, 16 * warp, 8 * kk, g, t4);
        }
        // dS <- dSf = dS * fw, then du and the first part of dV.  None of this needs the chunk-start state, so the
        // attn kernel does it before it waits for the state's copy; attn_ln needs the state first (for dy).
        float du[2][4] = {}, dV[2][4] = {};
        float X[2][4] = {};
        if (!LN) live = s0_wait(&sm.s0_bar, it & 1, &sm.abort, p.status) && live;  // this chunk's start state has landed
        // attn: the X = S0 wa^T products ride in the same loop, six independent accumulator chains instead of four, then two
        auto carry = [&](float (&gp)[16]) {  // sum over the rows of gp, a thread's part of it: [2 * nt + e] for key column 8 * nt + 2 * t4 + e
            // Sum over the eight row lanes g as a reduce-scatter: every step halves the values a lane carries (8 + 4 + 2
            // shuffles instead of 3 per value), and lane g ends with the two sums of tile nt = bit-reversed g.
            const bool b0 = g & 1, b1 = g & 2, b2 = g & 4;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float send = b0 ? gp[i] : gp[i + 8], keep = b0 ? gp[i + 8] : gp[i];
                gp[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float send = b1 ? gp[i] : gp[i + 4], keep = b1 ? gp[i + 4] : gp[i];
                gp[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float send = b2 ? gp[i] : gp[i + 2], keep = b2 ? gp[i + 2] : gp[i];
                gp[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
            }
            const int nt_own = (b2 ? 1 : 0) + (b1 ? 2 : 0) + (b0 ? 4 : 0);
            *reinterpret_cast<float2*>(&sm.Gp[PAR ? gp_set ^ 1 : gp_set][warp][8 * nt_own + 2 * t4]) = make_float2(gp[0], gp[1]);
        };
        auto du_dv = [&]() {
            float* const own = sm.dSs + (16 * warp + g) * SS;  // PAR: dS comes through shared memory, dSf goes there at once
            if (PAR) {
                float gp[16];
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    float* q = own + xcol<1>(g, 8 * nt + 2 * t4);
                    const float2 f = *reinterpret_cast<const float2*>(sm.fw + 8 * nt + 2 * t4), lo = *reinterpret_cast<const float2*>(q), hi2 = *reinterpret_cast<const float2*>(q + 8 * SS);
                    const float2 (&n2)[2] = nx[PAR ? nt : 0];
                    gp[2 * nt] = lo.x * n2[0].x + hi2.x * n2[1].x;
                    gp[2 * nt + 1] = lo.y * n2[0].y + hi2.y * n2[1].y;
                    *reinterpret_cast<float2*>(q) = make_float2(lo.x * STATE_SCALE * f.x, lo.y * STATE_SCALE * f.y);
                    *reinterpret_cast<float2*>(q + 8 * SS) = make_float2(hi2.x * STATE_SCALE * f.x, hi2.y * STATE_SCALE * f.y);
                }
                carry(gp);
                __syncwarp();
            }
#pragma unroll
            for (int nt = 0; nt < (PAR ? 0 : 8); ++nt) {
                const float2 f = *reinterpret_cast<const float2*>(sm.fw + 8 * nt + 2 * t4);  // P~_L = 2^64 P_L
                dS[nt][0] = dS[nt][0] * STATE_SCALE * f.x; dS[nt][1] = dS[nt][1] * STATE_SCALE * f.y;
                dS[nt][2] = dS[nt][2] * STATE_SCALE * f.x; dS[nt][3] = dS[nt][3] * STATE_SCALE * f.y;
            }
#pragma unroll
            for (int sb = 0; sb < 2; ++sb)
#pragma unroll
                for (int tb = sb; tb < 2; ++tb) {
                    mma<PREC>(du[sb], dyf[tb], mat_kn(3, sb, tb));
                    mma<PREC>(dV[sb], dyf[tb], mat_kn(1, sb, tb));
                }
            // (PAR: rolled, so that a chunk's code fits the instruction cache; the small terms apart, a third of the dependent products)
            float small[PAR ? 6 : 1][4] = {};
#pragma unroll PAR ? 1 : 8
            for (int kk = 0; kk < 8; ++kk) {
                FragA<PREC> a;
                if (PAR) {
                    const float* q = own + xcol<1>(g, 8 * kk + 2 * t4);
                    const float2 lo = *reinterpret_cast<const float2*>(q), hi2 = *reinterpret_cast<const float2*>(q + 8 * SS);
                    a.x[0].set(lo.x); a.x[1].set(hi2.x); a.x[2].set(lo.y); a.x[3].set(hi2.y);
                } else {
                    a = fragA_from_acc<PREC>(dS[PAR ? 0 : kk]);
                }
#pragma unroll
                for (int sb = 0; sb < 2; ++sb) {
                    mma2<PREC, PAR>(du[sb], small[PAR ? sb : 0], a, fragB_nk<PREC, true, 1>(sm.bwi, OPS, 8 * sb, 8 * kk, g, t4));
                    mma2<PREC, PAR>(dV[sb], small[PAR ? 2 + sb : 0], a, fragB_nk<PREC, true, 1>(sm.kwi, OPS, 8 * sb, 8 * kk, g, t4));
                }
                if (!LN) {
                    FragA<PREC> a0;
                    const float2 lo = *reinterpret_cast<const float2*>(s0_mk + 8 * kk), hi2 = *reinterpret_cast<const float2*>(s0_mk + 4 * SS + 8 * kk);
                    a0.x[0].setr(lo.x); a0.x[1].setr(hi2.x); a0.x[2].setr(lo.y); a0.x[3].setr(hi2.y);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma2<PREC, PAR>(X[nt], small[PAR ? 4 + nt : 0], a0, fragB_nk<PREC, true, 1>(sm.wa, OPS, 8 * nt, 8 * kk, g, t4));
                }
            }
#pragma unroll
            for (int i = 0; i < (PAR ? 8 : 0); ++i) {
                du[i >> 2][i & 3] += small[PAR ? i >> 2 : 0][i & 3];
                dV[i >> 2][i & 3] += small[PAR ? 2 + (i >> 2) : 0][i & 3];
                X[i >> 2][i & 3] += small[PAR ? 4 + (i >> 2) : 0][i & 3];
            }
        };
        if (!LN) du_dv();
        if (LN) live = s0_wait(&sm.s0_bar, it & 1, &sm.abort, p.status) && live;
        float U[2][4] = {};
        float dvx[2][4] = {};  // LN: bonus-term contribution to dv
        {
            float Y[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < (LN ? 8 : 0); ++kk) {
                FragA<PREC> a;
                {
                    const float2 lo = *reinterpret_cast<const float2*>(s0_mk + 8 * kk), hi2 = *reinterpret_cast<const float2*>(s0_mk + 4 * SS + 8 * kk);
                    a.x[0].setr(lo.x); a.x[1].setr(hi2.x); a.x[2].setr(lo.y); a.x[3].setr(hi2.y);
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    mma<PREC>(X[nt], a, fragB_nk<PREC, true, 1>(sm.wa, OPS, 8 * nt, 8 * kk, g, t4));
                    if (LN) mma<PREC>(Y[nt], a, fragB_nk<PREC, true, 1>(sm.wq, OPS, 8 * nt, 8 * kk, g, t4));
                }
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) {
                    mma<PREC>(X[nt], vf[kk], mat_nk(0, nt, kk));
                    if (LN) mma<PREC>(Y[nt], vf[kk], mat_nk(1, nt, kk));
                }
            FragA<PREC> xa[2] = {fragA_from_acc<PREC>(X[0]), fragA_from_acc<PREC>(X[1])};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) mma<PREC>(U[nt], xa[kk], mat_kn(2, nt, kk));
            if (LN) {
                // ---- rebuild Y, then GroupNorm / bonus / gate backward in the [value][time] layout ----
                FragA<PREC> ua0[2] = {fragA_from_acc<PREC>(U[0]), fragA_from_acc<PREC>(U[1])};
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int kk = 0; kk <= nt; ++kk) mma<PREC>(Y[nt], ua0[kk], mat_nk(3, nt, kk));
                // statistics: per-warp mean and centred sum of squares over 16 rows, merged below
                // (a thread's four time steps i4 = 2 * nt + e go through every shuffle level together; sums that only one
                // lane has to store are formed as a reduce-scatter over the row lanes, which halves the values per level)
                const bool b0 = g & 1, b1 = g & 2, b2 = g & 4;
                {
                    float sy[4], q2[4];
#pragma unroll
                    for (int i4 = 0; i4 < 4; ++i4) sy[i4] = Y[i4 >> 1][i4 & 1] + Y[i4 >> 1][(i4 & 1) + 2];
#pragma unroll
                    for (int m = 4; m <= 16; m <<= 1)
#pragma unroll
                        for (int i4 = 0; i4 < 4; ++i4) sy[i4] += __shfl_xor_sync(0xffffffffu, sy[i4], m);
#pragma unroll
                    for (int i4 = 0; i4 < 4; ++i4) {
                        sy[i4] *= (1.f / 16.f);  // the warp's mean
                        const float d0 = Y[i4 >> 1][i4 & 1] - sy[i4], d1 = Y[i4 >> 1][(i4 & 1) + 2] - sy[i4];
                        q2[i4] = d0 * d0 + d1 * d1;
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float send = b0 ? q2[i] : q2[i + 2], keep = b0 ? q2[i + 2] : q2[i];
                        q2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
                    }
                    {
                        const float send = b1 ? q2[0] : q2[1], keep = b1 ? q2[1] : q2[0];
                        q2[0] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
                    }
                    q2[0] += __shfl_xor_sync(0xffffffffu, q2[0], 16);
                    if (!b2) {  // this lane holds time step i4 = 2 * b0 + b1
                        const int tq = 8 * (b0 ? 1 : 0) + 2 * t4 + (b1 ? 1 : 0);
                        red[(warp * L + tq) * 2 + 0] = b0 ? (b1 ? sy[3] : sy[2]) : (b1 ? sy[1] : sy[0]);
                        red[(warp * L + tq) * 2 + 1] = q2[0];
                    }
                }
                __syncthreads();  // (D1)
                const unsigned char* gt = sm.st_g[LN ? vs : 0];
                float xh[2][4], dxh[2][4], rstd_t[4];
                float asum[16];  // [a1 | a2 | a3 | unused][i4]
#pragma unroll
                for (int i4 = 0; i4 < 4; ++i4) asum[12 + i4] = 0.f;
#pragma unroll
                for (int i4 = 0; i4 < 4; ++i4) {
                    const int nt = i4 >> 1, e = i4 & 1, tq = 8 * nt + 2 * t4 + e;
                    float mu = 0.f, m2 = 0.f;
#pragma unroll
                    for (int w2 = 0; w2 < WARPS; ++w2) mu += red[(w2 * L + tq) * 2];
                    mu *= 0.25f;
#pragma unroll
                    for (int w2 = 0; w2 < WARPS; ++w2) {
                        const float dm = red[(w2 * L + tq) * 2] - mu;
                        m2 += red[(w2 * L + tq) * 2 + 1] + 16.f * dm * dm;
                    }
                    const float rstd = 1.f / sqrtf(m2 * (1.f / N) + p.eps);
                    rstd_t[i4] = rstd;
                    const float bd = sm.bdot[tq];
                    float a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
                    for (int hrow = 0; hrow < 2; ++hrow) {
                        const int vc = 16 * warp + g + 8 * hrow, i = e + 2 * hrow;
                        const float x = (Y[nt][i] - mu) * rstd;
                        const float ve = bst_elem(vt, tq, vc), ge = bst_elem(gt, tq, vc), de = bst_elem(dyt, tq, vc);
                        const float z = x * sm.lnp[vc] + sm.lnp[N + vc] + bd * ve;
                        const float dz = de * ge;
                        Y[nt][i] = de * z;  // dg, stored below
                        dlnw_acc[hrow] += dz * x;
                        dlnb_acc[hrow] += dz;
                        dvx[nt][i] = dz * bd;
                        const float dx = dz * sm.lnp[vc];
                        xh[nt][i] = x;
                        dxh[nt][i] = dx;
                        a1 += dx; a2 += dx * x; a3 += dz * ve;
                    }
                    asum[i4] = a1; asum[4 + i4] = a2; asum[8 + i4] = a3;
                }
                {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float send = b0 ? asum[i] : asum[i + 8], keep = b0 ? asum[i + 8] : asum[i];
                        asum[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float send = b1 ? asum[i] : asum[i + 4], keep = b1 ? asum[i + 4] : asum[i];
                        asum[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float send = b2 ? asum[i] : asum[i + 2], keep = b2 ? asum[i + 2] : asum[i];
                        asum[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
                    }
                    // the lane now holds entries 8 * b0 + 4 * b1 + 2 * b2 + {0, 1}: sum number 2 * b0 + b1 of time steps i4 = 2 * b2 + {0, 1}
                    const int which = (b0 ? 2 : 0) + (b1 ? 1 : 0);
                    if (which < 3) {
                        const int tq = 8 * (b2 ? 1 : 0) + 2 * t4;
                        red2[(warp * L + tq) * 3 + which] = asum[0];
                        red2[(warp * L + tq + 1) * 3 + which] = asum[1];
                    }
                }
                // dg out, through the per-warp scratch tile for 16-byte stores
                {
                    float* sc = dvsc;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        const int tq = 8 * nt + 2 * t4;
                        sc[tq * YS + g] = Y[nt][0];
                        sc[(tq + 1) * YS + g] = Y[nt][1];
                        sc[tq * YS + g + 8] = Y[nt][2];
                        sc[(tq + 1) * YS + g + 8] = Y[nt][3];
                    }
                    __syncwarp();
                    const int row = lane >> 1, hf = lane & 1;
                    const uint4* src = reinterpret_cast<const uint4*>(sc + row * YS + 8 * hf);
                    uint4* dst = reinterpret_cast<uint4*>(gdg + ((long long)c * L + row) * p.st.t + 16 * warp + 8 * hf);
                    if (!TAIL || (long long)c * L + row < p.T) {
                        dst[0] = src[0];
                        dst[1] = src[1];
                    }
                    __syncwarp();
                }
                __syncthreads();  // (D2)
#pragma unroll
                for (int i4 = 0; i4 < 4; ++i4) {
                    const int nt = i4 >> 1, e = i4 & 1, tq = 8 * nt + 2 * t4 + e;
                    float m1 = 0.f, m2 = 0.f, sb = 0.f;
#pragma unroll
                    for (int w2 = 0; w2 < WARPS; ++w2) {
                        m1 += red2[(w2 * L + tq) * 3];
                        m2 += red2[(w2 * L + tq) * 3 + 1];
                        sb += red2[(w2 * L + tq) * 3 + 2];
                    }
                    m1 *= (1.f / N); m2 *= (1.f / N);
                    if (warp == 0 && g == 0) sm.sbon[tq] = sb;
#pragma unroll
                    for (int hrow = 0; hrow < 2; ++hrow) {
                        const int i = e + 2 * hrow;
                        Y[nt][i] = rstd_t[i4] * (dxh[nt][i] - m1 - xh[nt][i] * m2);  // gradient of the recurrence output
                    }
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    dyf[nt] = fragA_from_acc<PREC>(Y[nt]);
                    const int tq = 8 * nt + 2 * t4, vc = 16 * warp + g;
                    const int c0 = xcol<1>(tq, vc), c1 = xcol<1>(tq, vc + 8);  // rows tq, tq+1 share the swizzle
                    sm.Yt[tq * OPS + c0] = pre<PREC>(Y[nt][0]); sm.Yt[(tq + 1) * OPS + c0] = pre<PREC>(Y[nt][1]);
                    sm.Yt[tq * OPS + c1] = pre<PREC>(Y[nt][2]); sm.Yt[(tq + 1) * OPS + c1] = pre<PREC>(Y[nt][3]);
                }
            }
        }
        if (LN) du_dv();
        float dabu[2][4] = {};
        {
            FragA<PREC> da2[2] = {fragA_from_acc<PREC>(du[0]), fragA_from_acc<PREC>(du[1])};
#pragma unroll
            for (int nb = 0; nb < 2; ++nb)
#pragma unroll
                for (int kb = nb; kb < 2; ++kb) mma<PREC>(dabu[nb], da2[kb], mat_nk(2, nb, kb));
        }
        FragA<PREC> dbf[2] = {fragA_from_acc<PREC>(dabu[0]), fragA_from_acc<PREC>(dabu[1])};
#pragma unroll
        for (int sb = 0; sb < 2; ++sb)
#pragma unroll
            for (int tb = sb; tb < 2; ++tb) mma<PREC>(dV[sb], dbf[tb], mat_kn(0, sb, tb));

        if (PAR) {  // dv out, whole sectors of eight values
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const long long row = (long long)c * L + 8 * nt + 2 * t4 + e;
                    float* q = gdv + now.off + row * p.st.t + 16 * warp + g;
                    if (!TAIL || row < p.T) { q[0] = dV[nt][e]; q[8] = dV[nt][e + 2]; }
                }
        } else {  // transposed through a per-warp scratch tile for 16-byte stores
            float* sc = dvsc;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int tq = 8 * nt + 2 * t4;
                sc[tq * YS + g] = dV[nt][0] + dvx[nt][0];
                sc[(tq + 1) * YS + g] = dV[nt][1] + dvx[nt][1];
                sc[tq * YS + g + 8] = dV[nt][2] + dvx[nt][2];
                sc[(tq + 1) * YS + g + 8] = dV[nt][3] + dvx[nt][3];
            }
            __syncwarp();
            const int row = lane >> 1, hf = lane & 1;
            const uint4* src = reinterpret_cast<const uint4*>(sc + row * YS + 8 * hf);
            uint4* dst = reinterpret_cast<uint4*>(gdv + now.off + ((long long)c * L + row) * p.st.t + 16 * warp + 8 * hf);
            if (!TAIL || (long long)c * L + row < p.T) {
                dst[0] = src[0];
                dst[1] = src[1];
            }
        }
        // dSf, U, dabu to shared memory for stage C
#pragma unroll
        for (int nt = 0; nt < (PAR ? 0 : 8); ++nt) {
            *reinterpret_cast<float2*>(sm.dSs + (16 * warp + g) * SS + xcol<1>(g, 8 * nt + 2 * t4)) = make_float2(pre<PREC>(dS[nt][0]), pre<PREC>(dS[nt][1]));
            *reinterpret_cast<float2*>(sm.dSs + (16 * warp + g + 8) * SS + xcol<1>(g, 8 * nt + 2 * t4)) = make_float2(pre<PREC>(dS[nt][2]), pre<PREC>(dS[nt][3]));
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int tq = 8 * nt + 2 * t4, vc = 16 * warp + g;
            const int c0 = xcol<1>(tq, vc), c1 = xcol<1>(tq, vc + 8);  // rows tq, tq+1 share the swizzle
            sm.Ut[tq * OPS + c0] = pre<PREC>(U[nt][0]); sm.Ut[(tq + 1) * OPS + c0] = pre<PREC>(U[nt][1]);
            sm.Ut[tq * OPS + c1] = pre<PREC>(U[nt][2]); sm.Ut[(tq + 1) * OPS + c1] = pre<PREC>(U[nt][3]);
            sm.Dt[tq * OPS + c0] = pre<PREC>(dabu[nt][0]); sm.Dt[(tq + 1) * OPS + c0] = pre<PREC>(dabu[nt][1]);
            sm.Dt[tq * OPS + c1] = pre<PREC>(dabu[nt][2]); sm.Dt[(tq + 1) * OPS + c1] = pre<PREC>(dabu[nt][3]);
        }
        // dS0 = dSf + dY^T wq + dabu^T wa ; carried decay term sum_i dS0[i,:] S0[i,:]
        if (!PAR) {
            float gp[16];  // this thread's two rows
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) {
                    mma<PREC>(dS[nt], dyf[kk], fragB_kn<PREC, true, 1>(sm.wq, OPS, 8 * nt, 8 * kk, g, t4));
                    mma<PREC>(dS[nt], dbf[kk], fragB_kn<PREC, true, 1>(sm.wa, OPS, 8 * nt, 8 * kk, g, t4));
                }
                const float2 lo = *reinterpret_cast<const float2*>(s0_mk + 8 * nt);
                const float2 hi2 = *reinterpret_cast<const float2*>(s0_mk + 4 * SS + 8 * nt);
                gp[2 * nt] = dS[nt][0] * lo.x + dS[nt][2] * hi2.x;
                gp[2 * nt + 1] = dS[nt][1] * lo.y + dS[nt][3] * hi2.y;
            }
            carry(gp);
        }
        __syncthreads();  // (C1)
        // ---------------- stage C: contractions over the value index --------------------------
        float DA[2][4] = {}, DQ[2][4] = {}, DB[2][4] = {}, DK[2][4] = {};
        {
            // one score gradient per warp: 0 dQK = tril(dY V^T), 1 dAK = stril(dabu V^T),
            // 2 dQB = tril(dY U^T), 3 dAB = stril(dabu U^T)
            float d[2][4] = {};
            const bool strict = warp & 1;
            float* dst = sm.sgrad() + warp * (L * SCS);  // 0 dQK, 1 dAK, 2 dQB, 3 dAB
            // (rolled, as far as registers allow no less: the chunk loop is 100 KB of code in the triple-TF32 class, three times the
            // instruction cache; 96 chains of 32 chunks 339 -> 325 us)
#pragma unroll PAR ? 1 : 2
            for (int kk = 0; kk < 8; ++kk) {
                FragA<PREC> aD = fragA_mk<PREC, true, 1>(sm.Dt, OPS, 0, 8 * kk, g, t4);
                FragA<PREC> aY = LN ? fragA_mk<PREC, true, 1>(sm.Yt, OPS, 0, 8 * kk, g, t4) : fragA_mk_st<PREC>(dyt, 8 * kk, g, t4);
                FragA<PREC> aU = fragA_mk<PREC, true, 1>(sm.Ut, OPS, 0, 8 * kk, g, t4);
                FragA<PREC> aV = fragA_mk_st<PREC>(vt, 8 * kk, g, t4);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    FragB<PREC> bsc;  // [contraction][row of half nt] of U or V: registers of its A fragment
                    bsc.x[0] = (warp >> 1) ? aU.x[nt] : aV.x[nt];
                    bsc.x[1] = (warp >> 1) ? aU.x[2 + nt] : aV.x[2 + nt];
                    mma<PREC>(d[nt], strict ? aD : aY, bsc);
                    FragB<PREC> bS;
                    bS.x[0].setr(s0_kn[4 * kk * SS + 8 * nt]); bS.x[1].setr(s0_kn[(4 * kk + 1) * SS + 8 * nt]);
                    FragB<PREC> bD = fragB_kn<PREC, true, 1>(sm.dSs, SS, 16 * warp + 8 * nt, 8 * kk, g, t4);
                    mma<PREC>(DA[nt], aD, bS);
                    mma<PREC>(DQ[nt], aY, bS);
                    mma<PREC>(DB[nt], aU, bD);
                    mma<PREC>(DK[nt], aV, bD);
                }
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int s = 8 * nt + 2 * t4;
                auto keep = [&](int tq, int ss) { return strict ? ss < tq : ss <= tq; };
                *reinterpret_cast<float2*>(dst + g * SCS + xcol<1>(g, s)) =
                    make_float2(keep(g, s) ? pre<PREC>(d[nt][0]) : 0.f, keep(g, s + 1) ? pre<PREC>(d[nt][1]) : 0.f);
                *reinterpret_cast<float2*>(dst + (g + 8) * SCS + xcol<1>(g, s)) =
                    make_float2(keep(g + 8, s) ? pre<PREC>(d[nt][2]) : 0.f, keep(g + 8, s + 1) ? pre<PREC>(d[nt][3]) : 0.f);
            }
        }
        if (PAR) fence_async_smem();  // dSs was written here and comes by bulk copy next
        __syncthreads();  // (C2) score gradients visible; S0s (and dSs) free
        if (it + 1 < items && live) issue_s0(item(it + 1));
        if (PAR && it + 1 < items) issue_vdy(item(it + 1), 0);
        cp_async_commit();

#pragma unroll 1
        for (int kk = 0; kk < 2; ++kk) {
            const float *dQK = sm.sgrad(), *dAK = dQK + L * SCS, *dQB = dQK + 2 * L * SCS, *dAB = dQK + 3 * L * SCS;
            FragA<PREC> aAB = fragA_mk<PREC, true, 1>(dAB, SCS, 0, 8 * kk, g, t4), aAK = fragA_mk<PREC, true, 1>(dAK, SCS, 0, 8 * kk, g, t4);
            FragA<PREC> aQB = fragA_mk<PREC, true, 1>(dQB, SCS, 0, 8 * kk, g, t4), aQK = fragA_mk<PREC, true, 1>(dQK, SCS, 0, 8 * kk, g, t4);
            FragA<PREC> tAB = fragA_km<PREC, true, 1>(dAB, SCS, 0, 8 * kk, g, t4), tAK = fragA_km<PREC, true, 1>(dAK, SCS, 0, 8 * kk, g, t4);
            FragA<PREC> tQB = fragA_km<PREC, true, 1>(dQB, SCS, 0, 8 * kk, g, t4), tQK = fragA_km<PREC, true, 1>(dQK, SCS, 0, 8 * kk, g, t4);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int n0 = 16 * warp + 8 * nt;
                FragB<PREC> bb = fragB_kn<PREC, true, 1>(sm.bwi, OPS, n0, 8 * kk, g, t4), bk = fragB_kn<PREC, true, 1>(sm.kwi, OPS, n0, 8 * kk, g, t4);
                FragB<PREC> ba = fragB_kn<PREC, true, 1>(sm.wa, OPS, n0, 8 * kk, g, t4), bq = fragB_kn<PREC, true, 1>(sm.wq, OPS, n0, 8 * kk, g, t4);
                mma<PREC>(DA[nt], aAB, bb); mma<PREC>(DA[nt], aAK, bk);
                mma<PREC>(DQ[nt], aQB, bb); mma<PREC>(DQ[nt], aQK, bk);
                mma<PREC>(DB[nt], tAB, ba); mma<PREC>(DB[nt], tQB, bq);
                mma<PREC>(DK[nt], tAK, ba); mma<PREC>(DK[nt], tQK, bq);
            }
        }
        // ---------------- epilogue: thread holds rows g, g+8 x key columns n0+2*t4, +1 ---------
        float outv[5][2][2][2];  // [dq, dw, dk, da, db][tile][row half][column]
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int key = 16 * warp + 8 * nt + 2 * t4;
            float x[2][2], e2[2][2], lwv[2][2];  // [row half][column]
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                const int tq = g + 8 * hrow;
                const int kx = xcol<1>(tq, key);
                const float2 cu = *reinterpret_cast<const float2*>(sm.cum + tq * OPS + kx);
                float2 lwp;
                float2 up = make_float2(STATE_UNSCALE, STATE_UNSCALE);  // P~ before the first step
                if (PREC == 3) {
                    lwp = *reinterpret_cast<const float2*>(sm.lw + tq * OPS + kx);
                    if (tq > 0) up = *reinterpret_cast<const float2*>(sm.cum + (tq - 1) * OPS + xcol<1>(tq - 1, key));
                } else {  // running log-decay difference; row -1 is zero
                    const float2 cp = tq > 0 ? *reinterpret_cast<const float2*>(sm.cum + (tq - 1) * OPS + xcol<1>(tq - 1, key)) : make_float2(0.f, 0.f);
                    lwp = make_float2(cu.x - cp.x, cu.y - cp.y);
                }
                const float2 oq = *reinterpret_cast<const float2*>(sm.wq + tq * OPS + kx);
                const float2 oa = *reinterpret_cast<const float2*>(sm.wa + tq * OPS + kx);
                const float2 okw = *reinterpret_cast<const float2*>(sm.kwi + tq * OPS + kx);
                const float2 ob = *reinterpret_cast<const float2*>(sm.bwi + tq * OPS + kx);
                const float cuv[2] = {cu.x, cu.y}, lwa[2] = {lwp.x, lwp.y};
                const float wqv[2] = {oq.x, oq.y}, wav[2] = {oa.x, oa.y}, kwv[2] = {okw.x, okw.y}, bwv[2] = {ob.x, ob.y};
                float o_q[2], o_k[2], o_a[2], o_b[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = e + 2 * hrow;
                    const float incl = PREC == 3 ? cuv[e] : decay_up<PREC>(cuv[e]);   // P~_t, as the scan formed it
                    const float inv = rcp_p<PREC>(incl);
                    // P_{t-1} = exp(cum_{t-1}) with cum_{t-1} = cum_t - lw_t (0 for the first row): an exponential on the idle
                    // special-function unit instead of two shuffles for the row above; fp32 class: from the row above (an exponential is 15 instructions)
                    const float non = PREC == 3 ? (e ? up.y : up.x) : decay_up<PREC>(cuv[e] - lwa[e]);
                    o_a[e] = non * DA[nt][i];
                    o_q[e] = incl * DQ[nt][i];
                    o_b[e] = inv * DB[nt][i];
                    o_k[e] = inv * DK[nt][i];
                    if (LN) {  // bonus term: y += (sum_j q_j k_j bonus_j) v
                        const float sbv = sm.sbon[tq], bo = sm.lnp[2 * N + key + e];
                        const float q_raw = wqv[e] * inv, k_raw = kwv[e] * incl;
                        o_q[e] += sbv * k_raw * bo;
                        o_k[e] += sbv * q_raw * bo;
                        dbon_acc[nt][e] += sbv * q_raw * k_raw;
                    }
                    e2[hrow][e] = wav[e] * DA[nt][i];
                    x[hrow][e] = wqv[e] * DQ[nt][i] - kwv[e] * DK[nt][i] - bwv[e] * DB[nt][i] + e2[hrow][e];
                    lwv[hrow][e] = lwa[e];
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    outv[0][nt][hrow][e] = o_q[e]; outv[2][nt][hrow][e] = o_k[e];
                    outv[3][nt][hrow][e] = o_a[e]; outv[4][nt][hrow][e] = o_b[e];
                }
            }
            // inclusive suffix sum over the 16 time rows (rows live in lanes g = 0..7, two halves)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int d = 1; d < 8; d <<= 1) {
                    const float yl = __shfl_down_sync(0xffffffffu, x[0][e], 4 * d);
                    const float yh = __shfl_down_sync(0xffffffffu, x[1][e], 4 * d);
                    if (g + d < 8) { x[0][e] += yl; x[1][e] += yh; }
                }
                const float tot_hi = __shfl_sync(0xffffffffu, x[1][e], t4);
                x[0][e] += tot_hi;
            }
            const float2 Gc = make_float2(
                sm.Gp[(it & 1) ^ 1][0][key] + sm.Gp[(it & 1) ^ 1][1][key] + sm.Gp[(it & 1) ^ 1][2][key] + sm.Gp[(it & 1) ^ 1][3][key],
                sm.Gp[(it & 1) ^ 1][0][key + 1] + sm.Gp[(it & 1) ^ 1][1][key + 1] + sm.Gp[(it & 1) ^ 1][2][key + 1] + sm.Gp[(it & 1) ^ 1][3][key + 1]);
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                const float d0 = (x[hrow][0] - e2[hrow][0] + Gc.x) * lwv[hrow][0];
                const float d1 = (x[hrow][1] - e2[hrow][1] + Gc.y) * lwv[hrow][1];
                outv[1][nt][hrow][0] = d0; outv[1][nt][hrow][1] = d1;
            }
        }
        {
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                const long long off = now.off + ((long long)c * L + g + 8 * hrow) * p.st.t + 16 * warp;
                const bool live = !TAIL || (long long)c * L + g + 8 * hrow < p.T;  // uniform over the lanes that exchange values
#pragma unroll
                for (int ten = 0; ten < 5; ++ten)
                    store_quad(gout[ten] + off, outv[ten][0][hrow][0], outv[ten][0][hrow][1], outv[ten][1][hrow][0], outv[ten][1][hrow][1], t4, live);
            }
        }
        cp_async_wait<0>();
        if (PAR) fence_async_smem();  // the score gradients' place is filled by bulk copies next
        __syncthreads();  // (E)
        if (PAR && tid == 0 && it + 1 < items && live) issue_mats(item(it + 1));
    }

    if (LN) {
        // per-(batch, head) partial parameter gradients: ws[b][0..2][h*N + channel]
        float* ws = p.dparams_ws + bi * 3 * p.H * N + hi * N;
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
            float a = dlnw_acc[hrow], b2 = dlnb_acc[hrow];
            a += __shfl_xor_sync(0xffffffffu, a, 1); a += __shfl_xor_sync(0xffffffffu, a, 2);
            b2 += __shfl_xor_sync(0xffffffffu, b2, 1); b2 += __shfl_xor_sync(0xffffffffu, b2, 2);
            if (t4 == 0) {
                ws[16 * warp + g + 8 * hrow] = a;
                ws[p.H * N + 16 * warp + g + 8 * hrow] = b2;
            }
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float a = dbon_acc[nt][e];
                a += __shfl_xor_sync(0xffffffffu, a, 4); a += __shfl_xor_sync(0xffffffffu, a, 8); a += __shfl_xor_sync(0xffffffffu, a, 16);
                if (g == 0) ws[2 * p.H * N + 16 * warp + 8 * nt + 2 * t4 + e] = a;
            }
    }
    if (!PAR && p.ds0) {
        float* o = p.ds0 + bh * N * N;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            *reinterpret_cast<float2*>(o + (16 * warp + g) * N + 8 * nt + 2 * t4) = make_float2(dS[nt][0] * STATE_SCALE, dS[nt][1] * STATE_SCALE);
            *reinterpret_cast<float2*>(o + (16 * warp + g + 8) * N + 8 * nt + 2 * t4) = make_float2(dS[nt][2] * STATE_SCALE, dS[nt][3] * STATE_SCALE);
        }
    }
    if (tid == 0 && sm.abort) mbar_landed_uncounted(&sm.s0_bar, &sm.zero, p.status);
}

// ---- the state gradient alone, fp32 ------------------------------------------------------------------------------------------------
// The products that carry dS from chunk to chunk (stage B's du, dabu and dS0), one CTA per chain, triple TF32.  Four chain warps (16 value
// rows of dS each, no exchange between them); WALK_PREP groups of four warps fetch a chunk's inputs and scan it, and split its operands
// into the two TF32 parts once instead of at each of their uses; WALK_SLOTS chunks in flight.  Leaves dS at the end of every chunk in
// `tiles`, from where the chunk kernel (PAR) takes all chunks over all SMs.  With a chunk's whole work on the chain it took 20 000 cycles,
// most of them for fetching its 90 KB of code.
// Bound by the chain of dependent products, 3300 cycles a chunk (two preparation groups: 3700).  Backward in us, one kernel -> walk and
// chunks: 96 chains of 32 chunks 288 -> 203, 96 of 256 2251 -> 1469, 296 of 32 574 -> 513, 1024 of 32 1969 -> 1784, 2048 of 16 1867 -> 1818.
constexpr int WALK_SLOTS = 4, WALK_PREP = 3, WALK_THREADS = THREADS * (1 + WALK_PREP);
struct Walk32Slot {
    alignas(16) unsigned char dy[TILEB];
    alignas(16) float mats[2 * L * L];               // AI^T, QB as the record holds them
    alignas(16) float op[3][2][L * OPS];             // wq, wa, bwi: upper and lower part, column swizzle xcol<1>
    alignas(16) float fw[N];
};
struct Walk32Smem {
    alignas(16) unsigned char raw[WALK_PREP][4][TILEB];  // q, w, a, b
    Walk32Slot slot[WALK_SLOTS];
    uint64_t ready[WALK_SLOTS], free[WALK_SLOTS];
    volatile int abort;
};
static_assert(sizeof(Walk32Smem) <= 232448, "one CTA per SM");

template <bool TAIL>
__global__ void __launch_bounds__(WALK_THREADS, 1) wkv7_bwd_walk32_kernel(BwdParams p, float* tiles, int it0, int count) {
    stream_wait();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Walk32Smem& sm = *reinterpret_cast<Walk32Smem*>(smem_raw);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, t4 = lane & 3, w = warp & 3;
    const int bh = blockIdx.x, bi = bh / (int)p.H, hi = bh - bi * (int)p.H, nchunks = (int)((p.T + L - 1) / L), c0 = nchunks - 1 - it0;
    const long long base = bi * p.st.b + hi * p.st.h;
    if (tid == 0) {
        for (int i = 0; i < WALK_SLOTS; ++i) {
            mbar_init(&sm.ready[i], WARPS);
            mbar_init(&sm.free[i], WARPS);
        }
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp >= WARPS) {
        // ---- preparation: group `grp` takes every WALK_PREP-th chunk
        const int grp = warp / WARPS - 1, gt = tid & (THREADS - 1);
        const float* in[5] = {(const float*)p.r + base, (const float*)p.w + base, (const float*)p.a + base, (const float*)p.b + base, (const float*)p.dy + base};
        auto piece = [&](void* dst, const float* src, int n, int row) {  // 16 bytes of step n's chunk, rows beyond the sequence as zeros
            const long long tt = (long long)(c0 - n) * L + row;
            if (TAIL) cp_async16_zfill(dst, src + (tt < p.T ? tt : p.T - 1) * p.st.t, tt < p.T);
            else cp_async16(dst, src + tt * p.st.t);
        };
        const int prow = gt / (N / 4), pch = 4 * (gt % (N / 4));  // a thread's pieces: rows prow, prow + 8
        auto fetch = [&](int n) {  // q, w, a, b
#pragma unroll
            for (int ten = 0; ten < 4; ++ten)
#pragma unroll
                for (int r = prow; r < L; r += 8) piece(sm.raw[grp][ten] + st_at(r, pch), in[ten] + pch, n, r);
        };
        auto fetch_slot = [&](int n) {  // dy and the record's matrices
            Walk32Slot& t = sm.slot[n % WALK_SLOTS];
#pragma unroll
            for (int r = prow; r < L; r += 8) piece(t.dy + st_at(r, pch), in[4] + pch, n, r);
            cp_async16(t.mats + 4 * gt, p.ckpt + ((long long)bh * nchunks + c0 - n) * CK_FLOATS + CK_AI + 4 * gt);
            static_assert(2 * L * L == 4 * THREADS, "a piece per thread");
        };
        auto group_bar = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); };
        const int row = lane & 15, j0 = 16 * w + 8 * (lane >> 4), at = row * OPS + xcol<1>(row, j0);
        const bool flip = (row >> 2) & 1;
        auto split = [&](float (*op)[L * OPS], const float (&x)[8]) {
            float h[8], l[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                h[i] = __uint_as_float(tf32_rna(x[i]));
                l[i] = __uint_as_float(tf32_rna(x[i] - h[i]));
            }
            store8(op[0] + at, h, flip);
            store8(op[1] + at, l, flip);
        };
        if (grp < count) fetch(grp);
        for (int n = grp; n < count; n += WALK_PREP) {
            if (n >= WALK_SLOTS) mbar_wait_bounded<true>(&sm.free[n % WALK_SLOTS], (n / WALK_SLOTS - 1) & 1, &sm.abort, p.status);
            fetch_slot(n);
            cp_async_commit();
            cp_async_wait<0>();
            group_bar();  // everyone's pieces have landed
            Walk32Slot& t = sm.slot[n % WALK_SLOTS];
            const unsigned char (*raw)[TILEB] = sm.raw[grp];
            const int off = st_at(row, j0);
            float lw[8], cum[8], x[8], o[8];
            load8<float>(raw[1] + off, lw);
            const int live = TAIL ? (int)min((long long)L, p.T - (long long)(c0 - n) * L) : L;
#pragma unroll
            for (int i = 0; i < 8; ++i) cum[i] = lw[i] = row < live ? fmaxf(-exp_p<3>(lw[i]), MIN_STEP_LOG_DECAY) : 0.f;  // as decay_scan()
#pragma unroll
            for (int d = 1; d < 16; d <<= 1)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float up = __shfl_up_sync(0xffffffffu, cum[i], d, 16);
                    if (row >= d) cum[i] += up;
                }
            load8<float>(raw[2] + off, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = x[i] * decay_up<3>(cum[i] - lw[i]);
            split(t.op[1], o);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                cum[i] = decay_up<3>(cum[i]);
                if (row == 15) t.fw[j0 + i] = cum[i];
            }
            load8<float>(raw[0] + off, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = x[i] * cum[i];
            split(t.op[0], o);
            load8<float>(raw[3] + off, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = x[i] * rcp_p<3>(cum[i]);
            split(t.op[2], o);
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.ready[n % WALK_SLOTS]);
            group_bar();  // the raw tiles have been read
            if (n + WALK_PREP < count) fetch(n + WALK_PREP);
        }
        stream_release();  // (at most WALK_SLOTS chunks before the end)
        cp_async_wait<0>();
        return;
    }
    // ---- the chain: value rows 16 w + {g, g + 8} of dS, carried as in wkv7_bwd_kernel
    const int bg = (g >> 2) & 1, bt = (t4 >> 1) & 1;  // element offsets under xcol<1> (pitch 72)
    const int mkE = g * OPS + 2 * t4 + 8 * bg, mkO = mkE - 16 * bg, knE = 2 * t4 * OPS + g + 8 * bt, knO = knE - 16 * bt;
    auto mk = [&](int kk) { return (kk & 1 ? mkO : mkE) + 8 * kk; };
    auto kn = [&](int nb) { return (nb & 1 ? knO : knE) + 8 * nb; };
    auto put = [](FragB<3>& f, int i, float h, float l) { f.x[i].h = __float_as_uint(h); f.x[i].l = __float_as_uint(l); };
    float dS[8][4];
    const long long st = (long long)bh * N * N + (16 * w + g) * N + 2 * t4;
    {
        const float* src = it0 ? p.ds0 : p.dsT;  // a later pass goes on from where the earlier one left it
        const float scale = it0 ? 1.f : STATE_UNSCALE;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 lo = src ? *reinterpret_cast<const float2*>(src + st + 8 * nt) : make_float2(0.f, 0.f);
            const float2 hi2 = src ? *reinterpret_cast<const float2*>(src + st + 8 * N + 8 * nt) : make_float2(0.f, 0.f);
            dS[nt][0] = lo.x * scale; dS[nt][1] = lo.y * scale; dS[nt][2] = hi2.x * scale; dS[nt][3] = hi2.y * scale;
        }
    }
    float* out = tiles + (long long)bh * count * TILE_FLOATS + 16 * w * SS;
    for (int n = 0; n < count; ++n, out += TILE_FLOATS) {
        const int s = n % WALK_SLOTS;
        const Walk32Slot& t = sm.slot[s];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            *reinterpret_cast<float2*>(out + mk(nt)) = make_float2(dS[nt][0], dS[nt][1]);
            *reinterpret_cast<float2*>(out + 8 * SS + mk(nt)) = make_float2(dS[nt][2], dS[nt][3]);
        }
        mbar_wait_bounded<false>(&sm.ready[s], (n / WALK_SLOTS) & 1, &sm.abort, p.status);
        const FragA<3> dyf[2] = {fragA_km_st<3>(t.dy, 16 * w, 0, g, t4), fragA_km_st<3>(t.dy, 16 * w, 8, g, t4)};
        // matrix m (0 AI^T, 1 QB): element (row, col) of the record's operand tiles
        auto mat = [&](int m, int row, int col) { return t.mats + m * L * L + (row >> 3) * 128 + (col >> 2) * 32 + (row & 7) * 4 + (col & 3); };
        auto B_kn = [&](int op, int nb, int kk) {
            const float *q = t.op[op][0] + 8 * kk * OPS + kn(nb), *l = q + L * OPS;
            FragB<3> f;
            put(f, 0, q[0], l[0]); put(f, 1, q[OPS], l[OPS]);
            return f;
        };
        // (the three terms of a product apart: the sums over the keys are what the chain waits for)
        float du[2][4] = {}, du_l[2][4] = {}, du_r[2][4] = {}, dabu[2][4] = {}, dabu_s[2][4] = {};
#pragma unroll
        for (int sb = 0; sb < 2; ++sb)
#pragma unroll
            for (int tb = sb; tb < 2; ++tb) {
                FragB<3> b;
                b.x[0].set(*mat(1, 8 * tb + 2 * t4, 8 * sb + g)); b.x[1].set(*mat(1, 8 * tb + 2 * t4 + 1, 8 * sb + g));
                mma2<3, true>(du[sb], du_r[sb], dyf[tb], b);
            }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const float2 f = *reinterpret_cast<const float2*>(t.fw + 8 * kk + 2 * t4);
            dS[kk][0] = dS[kk][0] * STATE_SCALE * f.x; dS[kk][1] = dS[kk][1] * STATE_SCALE * f.y;
            dS[kk][2] = dS[kk][2] * STATE_SCALE * f.x; dS[kk][3] = dS[kk][3] * STATE_SCALE * f.y;
            const FragA<3> a = fragA_from_acc<3>(dS[kk]);
#pragma unroll
            for (int sb = 0; sb < 2; ++sb) {
                const float* q = t.op[2][0] + 8 * sb * OPS + mk(kk);
                const float2 h = *reinterpret_cast<const float2*>(q), l = *reinterpret_cast<const float2*>(q + L * OPS);
                FragB<3> b;
                put(b, 0, h.x, l.x); put(b, 1, h.y, l.y);
                mma_tf32_raw(du[sb], a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].h, b.x[1].h);
                mma_tf32_raw(du_l[sb], a.x[0].l, a.x[1].l, a.x[2].l, a.x[3].l, b.x[0].h, b.x[1].h);
                mma_tf32_raw(du_r[sb], a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].l, b.x[1].l);
            }
            mma<3>(dS[kk], dyf[0], B_kn(0, kk, 0));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) du[i >> 2][i & 3] += du_l[i >> 2][i & 3] + du_r[i >> 2][i & 3];
        const FragA<3> da2[2] = {fragA_from_acc<3>(du[0]), fragA_from_acc<3>(du[1])};
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int kb = nb; kb < 2; ++kb) {
                FragB<3> b;
                const float2 v = *reinterpret_cast<const float2*>(mat(0, 8 * nb + g, 8 * kb + 2 * t4));
                b.x[0].set(v.x); b.x[1].set(v.y);
                mma2<3, true>(dabu[nb], dabu_s[nb], da2[kb], b);
            }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) mma<3>(dS[nt], dyf[1], B_kn(0, nt, 1));
#pragma unroll
        for (int i = 0; i < 8; ++i) dabu[i >> 2][i & 3] += dabu_s[i >> 2][i & 3];
        const FragA<3> dbf[2] = {fragA_from_acc<3>(dabu[0]), fragA_from_acc<3>(dabu[1])};
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            mma<3>(dS[nt], dbf[0], B_kn(1, nt, 0));
            mma<3>(dS[nt], dbf[1], B_kn(1, nt, 1));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.free[s]);
    }
    const float scale = it0 + count < nchunks ? 1.f : STATE_SCALE;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        *reinterpret_cast<float2*>(p.ds0 + st + 8 * nt) = make_float2(dS[nt][0] * scale, dS[nt][1] * scale);
        *reinterpret_cast<float2*>(p.ds0 + st + 8 * N + 8 * nt) = make_float2(dS[nt][2] * scale, dS[nt][3] * scale);
    }
}

// How many chunks of each chain are walked at a time: tiles of at most 512 MB, longer sequences take several passes, the walk going on
// from ds0.  0: not at all.  With three chunks the second launch costs what it saves (144 chains: 78 us in one kernel, 81 in two).  Each pass
// starts two kernels and loads and stores the whole dS, and of many chains only a few chunks fit: one kernel / walk in us, chunks a pass in
// brackets: 2048 chains of 64 7376 / 7118 (14), 2640 of 32 4682 / 4656 (11), 2912 of 32 5176 / 5196 (10), 4096 of 64 14346 / 14626 (7), 8192
// of 8 3654 / 3986 (3), 32000 of 8 14122 / 18143 (1).  Hence the line at 11, 2647 chains: beyond it whole sequences in one pass would gain 2 % at most.
static int walk32_chunks(long long chains, long long chunks) {
    constexpr long long BYTES = 512LL << 20, PASS = 11;
    if (chains == 0 || chunks < 4 || chains > BYTES / (PASS * TILE_FLOATS * 4)) return 0;
    return (int)std::min(chunks, BYTES / (chains * TILE_FLOATS * 4));
}
size_t bwd32_workspace_bytes(long long B, long long T, long long H) {
    return WORK_FLAG_BYTES + (size_t)(B * H * walk32_chunks(B * H, (T + L - 1) / L)) * TILE_FLOATS * sizeof(float);
}

// dparams[i][c] = sum over batch of the per-(batch, head) partials, in a fixed order.
__global__ void reduce_dparams_kernel(const float* __restrict__ ws, float* __restrict__ out, long long B, long long n3) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n3) return;
    float acc = 0.f;
    for (long long b = 0; b < B; ++b) acc += ws[b * n3 + i];
    out[i] = acc;
}

// Tensor map of a bf16 [B,T,H,N] tensor with element strides st; box = one head, 16 time steps, 64 channels,
// 128-byte swizzle.  Encoded through the runtime's driver-entry-point query (no link against libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}
// Tensor map over the states of `records` checkpoint records (fp32 [64][64] at the start of each record of CK_FLOATS
// floats), seen as [record][a = row / 8][row bit 2][b = row % 4][column]; a box is the 32 rows of one value of bit 2,
// N + 8 floats wide (the part outside the 64 columns reads as zero).
bool encode_ckpt_state_map(CUtensorMap* m, const float* ckpt, long long records) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[5] = {(cuuint64_t)N, 4, 2, 8, (cuuint64_t)records};
    const cuuint64_t strides[4] = {N * 4, 4 * N * 4, 8 * N * 4, (cuuint64_t)CK_FLOATS * 4};
    const cuuint32_t box[5] = {(cuuint32_t)SS, 4, 1, 8, 1};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float*>(ckpt + CK_STATE), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Tensor map over the matrices part of the checkpoint records.  A record is 40 row groups of 128 floats (32 of state, then
// 8 of matrices: [AK;QK], AI, QB as operand tiles, a row group = [4 pieces][8 rows][4 floats]); the map sees the whole
// buffer as [row group][row bit 2][row % 4][piece][4 floats]; a box is the rows of one value of bit 2 in 8 row groups,
// 6 pieces wide (pieces 4, 5 do not exist and read as zero).
bool encode_ckpt_mats_map(CUtensorMap* m, const float* ckpt, long long records) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    static_assert(CK_FLOATS % 128 == 0 && CK_MATS % 128 == 0, "records and their matrices part are whole row groups");
    const cuuint64_t dims[5] = {4, 4, 4, 2, (cuuint64_t)(records * (CK_FLOATS / 128))};
    const cuuint64_t strides[4] = {32 * 4, 4 * 4, 16 * 4, 128 * 4};
    const cuuint32_t box[5] = {4, (cuuint32_t)(SCS / 4), 4, 1, 8};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float*>(ckpt), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool encode_bthn_map(CUtensorMap* m, void* base, long long B, long long T, long long H, const Strides& st) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)N, (cuuint64_t)H, (cuuint64_t)T, (cuuint64_t)B};
    // a dimension of extent 1 may carry any stride; give it a valid (16-byte multiple, non-zero) one
    auto sb = [&](long long s, long long fallback) { return (cuuint64_t)((s > 0 ? s : fallback) * 2); };
    const cuuint64_t strides[3] = {sb(st.h, N), sb(st.t, H * N), sb(st.b, T * H * N)};
    const cuuint32_t box[4] = {(cuuint32_t)N, 1, (cuuint32_t)L, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int PREC, bool LN> static int launch_bwd_t(const BwdParams& p, cudaStream_t stream) {
    constexpr bool WALK = PREC == 3 && !LN;
    const long long chains = p.B * p.H, chunks = (p.T + L - 1) / L;
    const int walked = WALK && p.flags && p.ds0 ? walk32_chunks(chains, chunks) : 0;
    auto kern = p.T % L ? wkv7_bwd_kernel<PREC, LN, true, false> : wkv7_bwd_kernel<PREC, LN, false, false>;
    if (walked) kern = p.T % L ? wkv7_bwd_kernel<PREC, LN, true, WALK> : wkv7_bwd_kernel<PREC, LN, false, WALK>;
    const int smem = (int)(walked ? sizeof(BwdSmem<PREC, LN, WALK>) : sizeof(BwdSmem<PREC, LN, false>));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return kLaunchFailed;
    CkptMaps cmaps;
    memset(&cmaps, 0, sizeof(cmaps));
    const long long records = chains * chunks;
    if (!(encode_ckpt_state_map(&cmaps.ck, p.ckpt, records) && encode_ckpt_mats_map(&cmaps.ckm, p.ckpt, records)))
        return kLaunchFailed;
    if (walked) {
        auto walk = p.T % L ? wkv7_bwd_walk32_kernel<true> : wkv7_bwd_walk32_kernel<false>;
        const int slots = 2 * sm_count();
        if (cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Walk32Smem)) != cudaSuccess) return kLaunchFailed;
        float* tiles = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p.flags) + WORK_FLAG_BYTES);
        for (long long it0 = 0; it0 < chunks; it0 += walked) {
            const int n = (int)std::min<long long>(walked, chunks - it0), total = (int)chains * n, per = (total + slots - 1) / slots;
            if (!launch(walk, dim3((unsigned)chains), WALK_THREADS, sizeof(Walk32Smem), stream, p, tiles, (int)it0, n)) return kLaunchFailed;
            if (!launch(kern, dim3((unsigned)((total + per - 1) / per)), THREADS, smem, stream, p, Walked{tiles, (int)it0, n, per, total}, cmaps)) return kLaunchFailed;
        }
        return kOk;
    }
    if (!launch(kern, dim3((unsigned)chains), THREADS, smem, stream, p, Walked{}, cmaps)) return kLaunchFailed;
    return LN ? launch_reduce_dparams(p, stream) : kOk;
}

int launch_reduce_dparams(const BwdParams& p, cudaStream_t stream) {
    const long long n3 = 3 * p.H * N;
    reduce_dparams_kernel<<<(unsigned)((n3 + 255) / 256), 256, 0, stream>>>(p.dparams_ws, p.dparams, p.B, n3);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

int launch_bwd(const BwdParams& p, int io_dtype, bool ln, cudaStream_t stream) {
    if (io_dtype == 0) return launch_bwd_bf16(p, ln, stream);
    if (io_dtype == 2) return ln ? launch_bwd_t<1, true>(p, stream) : launch_bwd_t<1, false>(p, stream);
    return ln ? launch_bwd_t<3, true>(p, stream) : launch_bwd_t<3, false>(p, stream);
}

}  // namespace wkv7
