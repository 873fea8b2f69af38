// WKV7 backward for sm_100a, bf16 tensors: the mathematics of wkv7_bwd.cu (formulas in its header), 4 working warps and a copy
// warp per CTA, two CTAs per SM, each over its share of the chunks (WorkSplit: chains walked in reverse, the state gradient of
// a cut chain handed on through ds0).
//
// What bounds it.  Per 16-step chunk 840 warp-level TF32 products (8 cycles each on one of four schedulers: 1680 cycles) and
// 3300 shared-memory wavefronts (one a cycle) meet 8700 warp instructions with the dependencies of a chain: with two CTAs an SM
// takes 4400 cycles per chunk (attn, a full machine), the data pipe busy 76 % of them.  The form of wkv7_bwd.cu had it
// busy 81 % of 5035 cycles.  What changed:
//  * equal shares of work instead of whole chains (768 chains on 296 CTAs are 2.6 rounds);
//  * the term of the decay gradient that was carried from the following chunk, sum_i dS[i,:] S'[i,:] with S' = (S0 + V^T kwi +
//    U^T bwi) fw, is formed from what stage C holds: sum_i dSf[i,:] S0[i,:] + sum_t (kwi[t,:] DKs[t,:] + bwi[t,:] DBs[t,:]), DKs =
//    V dSf and DBs = U dSf being the state parts of DK and DB (a reduction over all warps, 16 KB of shared-memory reads and the
//    exchange between chunks less);
//  * bf16 fragments by ldmatrix / stmatrix, the B fragments of the score gradients are the registers of A fragments, two base
//    offsets per access pattern (see mk, kn);
//  * all global traffic by bulk tensor copies from a warp of its own: issued by working warps they cost 15 % at the barriers;
//  * the chunk loop is 29 KB of code: beyond the 32 KB of the instruction cache every chunk streams it in anew at about 6 bytes
//    a cycle (two CTAs: 5100 cycles per chunk for 33 KB), hence the rolled loops;
//  * attn_ln: GroupNorm / bonus / gate backward with one thread per time step and 8 channels (16-byte accesses, shuffles
//    within eight lanes) instead of the transposed accumulator layout with three exchanges between the warps.
// (A pipeline of three or four warp groups - scan, chain, gradients - on one CTA per SM was 1.5 times slower: their different
// code does not fit the instruction cache, and rolled up to fit it a single warp per scheduler and group runs at 5.5 cycles an
// instruction.)
#include <cuda.h>
#include <algorithm>
#include <cstddef>
#include <cstring>

#include "wkv7_kernels.h"

namespace wkv7 {
namespace bf16bwd {

constexpr int NTHREADS = THREADS + 32;  // four working warps and one that issues the bulk copies
constexpr int ROWB = 2 * N;           // bf16 tile row: 128 bytes, 16-byte units XOR-ed with (row % 8)
constexpr int TILE = L * ROWB;
constexpr int SS = N + 8;             // row pitch (floats) of the state tiles
constexpr int S0_BLK = 32 * SS;
constexpr int MAT_BLK = 8 * 4 * SCS;

struct BwdMaps { CUtensorMap in[8], out[7], ck, ckm; };  // q, w, k, a, b, v, dy, g; dq, dw, dk, da, db, dv, dg; checkpoint states, matrices

struct Desc { int bh, bi, hi, c, flags, left; };  // c: chunk index in time; left: chunks of the segment after this one
enum : int { FIRST = 1, LAST = 2, CUT_BEFORE = 4, CUT_AFTER = 8 };  // of a segment; the rest of the chain before / after it is another CTA's

template <bool LN> struct Smem {
    static constexpr int IN = LN ? 8 : 7;          // input tiles of a chunk
    // attn: v and dy (read to the end of stage C) in two sets, so that the next chunk's inputs can be requested as soon as the
    // scan has read q .. b.  attn_ln: one set, requested after stage C's first half (two CTAs have to fit an SM); the recurrence
    // output and its gradient live in the dead q .. b tiles meanwhile.
    static constexpr int SETS = LN ? 1 : 2;
    alignas(1024) unsigned char raw[5][TILE];      // q, w, k, a, b
    alignas(1024) unsigned char vdy[SETS][IN - 5][TILE];  // v, dy (, g)
    alignas(1024) unsigned char out[LN ? 7 : 6][TILE];    // dq, dw, dk, da, db, dv (, dg)
    alignas(128) float S0[N * SS];                 // checkpoint state, layout of s0_at()
    alignas(128) float mats[2 * MAT_BLK];          // AK, QK, AI^T, QB, layout of mat_at()
    // operands, [time][key] (u, dabu: [time][value]) with row pitch OPS and column swizzle xcol<1>
    alignas(16) float wq[L * OPS], wa[L * OPS], kwi[L * OPS], bwi[L * OPS], cum[L * OPS], u[L * OPS], dabu[L * OPS];
    alignas(16) float dS[N * SS];                  // dSf [value][key], layout of s0_at()
    alignas(16) float sgrad[4][L * SCS];           // dQK, dAK, dQB, dAB
    alignas(16) float fw[N];
    alignas(8) uint64_t raw_full, rec_full;
    Desc desc[4];
    volatile int abort, zero;                      // zero stays 0 (see mbar_landed)
    float bdot[LN ? WARPS : 1][L], sbon[L];        // attn_ln: per-warp parts of sum_j r k bonus; sum_i dz v
    __device__ __forceinline__ float* yt() { return reinterpret_cast<float*>(raw[0]); }  // attn_ln: [time][value], pitch OPS
};
static_assert(sizeof(Smem<false>) + 1024 <= 115712 && sizeof(Smem<true>) + 1024 <= 115712, "two CTAs per SM");
static_assert(L * OPS * 4 <= 5 * TILE && L * OPS <= 4 * L * SCS, "aliases");

__device__ __forceinline__ int mat_at(int m, int row, int col) {
    return ((row >> 2) & 1) * (MAT_BLK + 8) + ((2 * m + (row >> 3)) * 4 + (row & 3)) * SCS + col;
}
__device__ __forceinline__ int s0_at(int row, int col) {
    return ((row >> 2) & 1) * (S0_BLK + 8) + (((row >> 3) << 2) | (row & 3)) * SS + col;
}
__device__ __forceinline__ void expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void load4(void* dst, const CUtensorMap* m, uint64_t* bar, int x1, int x2, int x3) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(m), "r"(smem_u32(bar)), "r"(0), "r"(x1), "r"(x2), "r"(x3) : "memory");
}
__device__ __forceinline__ void load5(void* dst, const CUtensorMap* m, uint64_t* bar, int x0, int x1, int x2, int x3, int x4) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(m), "r"(smem_u32(bar)), "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(x4) : "memory");
}
__device__ __forceinline__ void store4(const CUtensorMap* m, const void* src, int x1, int x2, int x3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                 ::"l"(m), "r"(0), "r"(x1), "r"(x2), "r"(x3), "r"(smem_u32(src)) : "memory");
}
template <bool TRANS> __device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void* p) {
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
// A fragment of one 8-wide contraction block from two 8x8 bf16 blocks (rows g | g + 8, two adjacent contraction indices each)
__device__ __forceinline__ FragA<1> frag_bf16(uint32_t lo, uint32_t hi) {
    FragA<1> f;
    f.x[0].h = lo << 16; f.x[2].h = lo & 0xffff0000u;
    f.x[1].h = hi << 16; f.x[3].h = hi & 0xffff0000u;
    return f;
}
// rows = values 16 w + .., contraction = time (two blocks), from a [time][value] tile
__device__ __forceinline__ void frags_value_time(FragA<1> (&f)[2], const unsigned char* tile, int w, int lane) {
    uint32_t r[4];
    const int t = 8 * (lane >> 4) + (lane & 7), unit = 2 * w + ((lane >> 3) & 1);
    ldmatrix4<true>(r, tile + t * ROWB + ((unit ^ (t & 7)) << 4));
    f[0] = frag_bf16(r[0], r[1]);
    f[1] = frag_bf16(r[2], r[3]);
}
// The B fragment [contraction][n = row of half nt] of a matrix whose A fragment is f: the same registers.
__device__ __forceinline__ FragB<1> as_b(const FragA<1>& f, int nt) {
    FragB<1> b;
    b.x[0] = f.x[nt]; b.x[1] = f.x[2 + nt];
    return b;
}

// The scan: a thread has two adjacent time steps x 4 adjacent key channels, so that the running sum takes three shuffle rounds of 4
// channels instead of four of 8 (a shuffle is a pass through the data pipe).  Slot 0 is the earlier or the later one (`late`) of the two,
// such that the raw loads (half-warps: every residue of the row mod 8 once, two channel quads) and the operand stores (quarter-warps: rows 0,
// 2, 4, 6 or 1, 3, 5, 7 of the pitch-72 tiles x two quads) are free of bank conflicts.
// (One step x 8 channels: 782 us at B64 T1024 H12, 117 with its walk at B3 T1003 H16; this: 776 and 115.)
struct ScanLane {
    int row0, quad;  // slot 1: row0 ^ 1; quad: of the head's 16
    bool late;
    __device__ __forceinline__ ScanLane(int w, int lane)
        : row0(2 * ((lane & 3) + ((lane >> 1) & 4)) + ((lane >> 3) & 1)), quad(4 * w + ((lane >> 2) & 1) + ((lane >> 3) & 2)), late((lane >> 3) & 1) {}
    __device__ __forceinline__ int raw(int e) const { const int row = row0 ^ e; return row * ROWB + (((quad >> 1) ^ (row & 7)) << 4) + (quad & 1) * 8; }
    __device__ __forceinline__ int dst(int e) const { const int row = row0 ^ e; return row * OPS + xcol<1>(row, 4 * quad); }
    // w -> running log2 decay through and before the slots' steps; steps from `live` on do not exist
    __device__ __forceinline__ void decay(F2 (&cum)[2][2], F2 (&before)[2][2], int live, int lane) const {
        constexpr float LOG2E = 1.4426950408889634f, FLOOR = MIN_STEP_LOG_DECAY * LOG2E;  // log2 of the per-step decay
        F2 x[2][2];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const F2 l = mul2(cum[e][i], f2(LOG2E, LOG2E)), d = mul2(f2(ex2_approx(l.x), ex2_approx(l.y)), f2(-LOG2E, -LOG2E));
                x[e][i] = (row0 ^ e) < live ? f2(fmaxf(d.x, FLOOR), fmaxf(d.y, FLOOR)) : f2(0.f, 0.f);
            }
        const float f0 = late ? 0.f : -1.f, f1 = late ? -1.f : 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            F2 sum = add2(x[0][i], x[1][i]);
#pragma unroll
            for (int d = 1; d < 4; d <<= 1) {
                const F2 up = f2(__shfl_up_sync(0xffffffffu, sum.x, d, 4), __shfl_up_sync(0xffffffffu, sum.y, d, 4));
                if ((lane & 3) >= d) sum = add2(sum, up);
            }
            const int src = (lane & 0x14) | 3;
            const F2 low = f2(__shfl_sync(0xffffffffu, sum.x, src), __shfl_sync(0xffffffffu, sum.y, src));
            if (late) sum = add2(sum, low);
            cum[0][i] = fma2(x[1][i], f2(f0, f0), sum);  // less the later step's, in the earlier one
            cum[1][i] = fma2(x[0][i], f2(f1, f1), sum);
#pragma unroll
            for (int e = 0; e < 2; ++e) before[e][i] = fma2(x[e][i], f2(-1.f, -1.f), cum[e][i]);
        }
    }
};
__device__ __forceinline__ float4 pre4(const F2 (&v)[2]) { return make_float4(pre<1>(v[0].x), pre<1>(v[0].y), pre<1>(v[1].x), pre<1>(v[1].y)); }

// PAR: the state gradients at the chunks' ends are given (wkv7_bwd_walk_kernel), so that chunks are worked in any order and none is
// carried here; the tiles of steps it0 .. it0 + ws.per_chain - 1 of each chain are in `tiles`.
struct Tiles { const float* base; int it0; };
constexpr int TILE_FLOATS = N * SS;  // layout of s0_at()

template <bool TAIL, bool LN, bool PAR>
__global__ void __launch_bounds__(NTHREADS, 2) wkv7_bwd_bf16_kernel(BwdParams p, WorkSplit ws, Tiles tiles, const __grid_constant__ BwdMaps maps) {
    stream_wait();
    extern __shared__ unsigned char smem_dyn[];
    using Smem = bf16bwd::Smem<LN>;
    Smem& sm = *reinterpret_cast<Smem*>(smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int nchunks = PAR ? (int)((p.T + L - 1) / L) : ws.per_chain;
    const WorkRange work(ws, blockIdx.x);

    auto describe = [&](int n) {
        if (n >= work.n) return;
        Desc d;
        int it;
        if (PAR) {
            const int x = work.first + n;
            d.bh = (int)((unsigned)x / (unsigned)ws.per_chain);
            it = x - d.bh * ws.per_chain;
            d.bi = (int)((unsigned)d.bh / (unsigned)p.H);
            d.hi = d.bh - d.bi * (int)p.H;
            d.c = nchunks - 1 - tiles.it0 - it;
            d.left = min(ws.per_chain - 1 - it, work.n - 1 - n);
            d.flags = 0;
            sm.desc[n & 3] = d;
            return;
        }
        work.locate(n, nchunks, d.bh, it);
        d.bi = (int)((unsigned)d.bh / (unsigned)p.H);
        d.hi = d.bh - d.bi * (int)p.H;
        d.c = nchunks - 1 - it;
        const int end = n < work.h ? work.h : nchunks;  // the start piece is steps 0 .. h - 1 of its chain
        const bool first = work.starts_segment(n, it), last = it + 1 == end;
        d.left = end - 1 - it;
        d.flags = (first ? FIRST : 0) | (last ? LAST : 0) | (first && it > 0 ? CUT_BEFORE : 0) | (last && it + 1 < nchunks ? CUT_AFTER : 0);
        sm.desc[n & 3] = d;
    };
    // (loops not unrolled: everything in the chunk loop counts against the instruction cache)
    auto load_inputs = [&](int n) {
        const Desc& d = sm.desc[n & 3];
        expect(&sm.raw_full, Smem::IN * TILE);
#pragma unroll 1
        for (int i = 0; i < Smem::IN; ++i) load4(i < 5 ? sm.raw[i] : sm.vdy[LN ? 0 : n & 1][i - 5], &maps.in[i], &sm.raw_full, d.hi, d.c * L, d.bi);
    };
    // checkpoint record: state and matrices as two boxes each (rows by their bit 2), see the maps in wkv7_bwd.cu
    auto load_record = [&](int n) {
        const Desc& d = sm.desc[n & 3];
        const int record = d.bh * nchunks + d.c;
        expect(&sm.rec_full, ((PAR ? 2 : 1) * N * SS + 2 * MAT_BLK) * 4);
        if (PAR) {
            const float* src = tiles.base + ((long long)d.bh * ws.per_chain + (nchunks - 1 - d.c - tiles.it0)) * TILE_FLOATS;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(sm.dS)), "l"(src), "r"(TILE_FLOATS * 4), "r"(smem_u32(&sm.rec_full)) : "memory");
        }
#pragma unroll 1
        for (int blk = 0; blk < 2; ++blk) {
            load5(sm.S0 + blk * S0_BLK, &maps.ck, &sm.rec_full, -8 * blk, 0, blk, 0, record);
            load5(sm.mats + blk * MAT_BLK, &maps.ckm, &sm.rec_full, 0, -2 * blk, 0, blk, record * (CK_FLOATS / 128) + CK_MATS / 128);
        }
    };

    if (tid < 2) describe(tid);
    if (tid == 0) {
        mbar_init(&sm.raw_full, 1);
        mbar_init(&sm.rec_full, 1);
        sm.abort = sm.zero = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == WARPS) {
        // ---- copy warp: a bulk tensor copy takes its thread some 200 cycles, which a working warp would make the others wait
        // for at the next barrier.  Takes part in the working warps' barriers.
        int inputs = 1, records = 1;  // loads issued
        if (lane == 0) {
            load_inputs(0);
            load_record(0);
        }
        for (int n = 0; n < work.n; ++n) {
            if (n + 1 == work.n) stream_release();
            const Desc d = sm.desc[n & 3];
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the previous chunk's output tiles have been read
            __syncthreads();  // (A)
            if (lane == 0) {
                if (!LN && n + 1 < work.n && !sm.abort) {
                    load_inputs(n + 1);
                    ++inputs;
                }
                Desc e = sm.desc[(n + 1) & 3];
                if (e.left > (PAR ? 0 : 1)) {  // (not the last but one: the last has flags)
                    --e.c; --e.left;
                    e.flags = 0;
                    sm.desc[(n + 2) & 3] = e;
                } else {
                    describe(n + 2);
                }
            }
            if (LN) {
                __syncthreads();  // (D1)
                __syncthreads();  // (D2)
            }
            __syncthreads();  // (C1)
            const bool more = lane == 0 && n + 1 < work.n && !sm.abort;  // (the working warps are past this chunk's waits for loads)
            __syncthreads();  // (C2)
            if (more) {
                if (LN) {
                    load_inputs(n + 1);
                    ++inputs;
                }
                load_record(n + 1);
                ++records;
            }
            __syncthreads();  // (E)
            if (lane == 0) {
#pragma unroll 1
                for (int i = 0; i < (LN ? 7 : 6); ++i) store4(&maps.out[i], sm.out[i], d.hi, d.c * L, d.bi);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            if ((d.flags & (LAST | CUT_AFTER)) == (LAST | CUT_AFTER) && p.ds0) __syncthreads();
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory must outlive the last stores
            mbar_landed(&sm.raw_full, inputs, &sm.zero, p.status);
            mbar_landed(&sm.rec_full, records, &sm.zero, p.status);
        }
        return;
    }

    // Offsets of this lane's fragment elements in a tile of row pitch 72 with the column swizzle xcol<1>: XOR-ing the column with
    // 8 turns, for a column block kk of 8, into +8 for even and -8 for odd kk, so that two bases per access pattern and
    // immediate offsets are all the address arithmetic there is.
    //   mk: row g, columns 8 kk + 2 t4, +1       kn: rows 2 t4 (and + 1), column 8 nb + g
    const int bg = (g >> 2) & 1, bt = (t4 >> 1) & 1;
    const int mkE = g * OPS + 2 * t4 + 8 * bg, mkO = mkE - 16 * bg, knE = 2 * t4 * OPS + g + 8 * bt, knO = knE - 16 * bt;
    static_assert(SS == OPS && OPS == 72 && SCS == 24, "pitches");
    auto mk = [&](int kk) { return (kk & 1 ? mkO : mkE) + 8 * kk; };
    auto kn = [&](int nb) { return (nb & 1 ? knO : knE) + 8 * nb; };
    auto A_mk = [&](const float* tile, int kk) {  // A operand, rows g, g + 8
        FragA<1> f;
        const float2 lo = *reinterpret_cast<const float2*>(tile + mk(kk)), hi = *reinterpret_cast<const float2*>(tile + 8 * OPS + mk(kk));
        f.x[0].setr(lo.x); f.x[1].setr(hi.x); f.x[2].setr(lo.y); f.x[3].setr(hi.y);
        return f;
    };
    auto B_nk = [&](const float* tile, int sb, int kk) {  // B operand [n][k], rows 8 sb + g
        FragB<1> f;
        const float2 v = *reinterpret_cast<const float2*>(tile + 8 * sb * OPS + mk(kk));
        f.x[0].setr(v.x); f.x[1].setr(v.y);
        return f;
    };
    auto B_kn = [&](const float* tile, int nb, int kk) {  // B operand [k][n], rows 8 kk + 2 t4, +1
        FragB<1> f;
        const float* q = tile + 8 * kk * OPS + kn(nb);
        f.x[0].setr(q[0]); f.x[1].setr(q[OPS]);
        return f;
    };
    // the same two patterns in the 24-float rows of the score gradients, for column blocks 0 and 1
    const int smk0 = g * SCS + 2 * t4 + 8 * bg, smk1 = smk0 - 16 * bg + 8, skn0 = 2 * t4 * SCS + g + 8 * bt, skn1 = skn0 - 16 * bt + 8;
    const int bp = (((g + 7) & 7) >> 2) & 1, pm0 = (g - 1) * OPS + 2 * t4 + 8 * bp, pm1 = pm0 - 16 * bp + 8;  // row g - 1, pattern mk
    // matrix m (0 AK, 1 QK, 2 AI^T, 3 QB) as a B operand: [n][k] (row 8 nt + g, columns 8 kk + 2 t4, +1), [k][n] (rows 8 tb + 2 t4, +1, column 8 sb + g)
    const float *const mat_g = sm.mats + mat_at(0, g, 2 * t4), *const mat_t = sm.mats + mat_at(0, 2 * t4, g);
    auto mat_nk = [&](int m, int nt, int kk) {
        FragB<1> f;
        const float2 v = *reinterpret_cast<const float2*>(mat_g + (2 * m + nt) * (4 * SCS) + 8 * kk);
        f.x[0].setr(v.x); f.x[1].setr(v.y);
        return f;
    };
    auto mat_kn = [&](int m, int sb, int tb) {
        FragB<1> f;
        const float* q = mat_t + (2 * m + tb) * (4 * SCS) + 8 * sb;
        f.x[0].setr(q[0]); f.x[1].setr(q[SCS]);
        return f;
    };
    const int s0_mk = s0_at(16 * warp + g, 2 * t4), s0_kn = s0_at(2 * t4, 16 * warp + g);

    // dS: warp owns value rows 16 warp + {g, g + 8}; tile nt covers key columns 8 nt .. 8 nt + 7.  Carried as 2^64 dS, the
    // counterpart of the forward's S~ = 2^-64 S (see ANCHOR_LN).
    float dS[8][4];
    // attn_ln: parameter gradients of the chain so far: GroupNorm weight, bias (this thread's time steps, channels 8 (tid % 8) ..),
    // bonus (this thread's time steps, its key columns)
    float dlnw[LN ? 8 : 1], dlnb[LN ? 8 : 1], dbon[LN ? 2 : 1][2];
    bool taken_up = false;  // the segment continues another CTA's
    for (int n = 0; n < work.n; ++n) {
        const Desc d = sm.desc[n & 3];
        // ---------------- scan: one thread = two adjacent time steps x 4 adjacent key channels (ScanLane) ----------------
        mbar_wait_bounded<false>(&sm.raw_full, n & 1, &sm.abort, p.status);
        {
            const ScanLane sl(warp, lane);
            F2 q[2][2], cum[2][2], before[2][2], k[2][2], a[2][2], b[2][2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int at = sl.raw(e);
                load4f2(sm.raw[1] + at, cum[e]);
                load4f2(sm.raw[0] + at, q[e]);
                load4f2(sm.raw[2] + at, k[e]);
                load4f2(sm.raw[3] + at, a[e]);
                load4f2(sm.raw[4] + at, b[e]);
            }
            if (LN) {  // bonus dot sum_j r_j k_j bonus_j of these time steps: this warp's 16 channels
                const float4 bo = __ldg(reinterpret_cast<const float4*>(p.params + (2 * p.H + d.hi) * N + 4 * sl.quad));
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const F2 acc = fma2(mul2(q[e][1], k[e][1]), f2(bo.z, bo.w), mul2(mul2(q[e][0], k[e][0]), f2(bo.x, bo.y)));
                    float dot = acc.x + acc.y;
                    dot += __shfl_xor_sync(0xffffffffu, dot, 4);
                    dot += __shfl_xor_sync(0xffffffffu, dot, 16);
                    if (!(lane & 0x14)) sm.bdot[warp][sl.row0 ^ e] = dot;
                }
            }
            sl.decay(cum, before, TAIL ? (int)min((long long)L, p.T - (long long)d.c * L) : L, lane);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                F2 wq[2], wa[2], kw[2], bw[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const F2 ca = add2(cum[e][i], f2(ANCHOR_LOG2, ANCHOR_LOG2)), cp = add2(before[e][i], f2(ANCHOR_LOG2, ANCHOR_LOG2));
                    const float cx = fmaxf(ca.x, -115.f), cy = fmaxf(ca.y, -115.f);
                    const F2 incl = f2(ex2_approx(cx), ex2_approx(cy)), inv = f2(ex2_approx(-cx), ex2_approx(-cy));
                    const F2 non = f2(ex2_approx(fmaxf(cp.x, -115.f)), ex2_approx(fmaxf(cp.y, -115.f)));
                    wq[i] = mul2(q[e][i], incl); wa[i] = mul2(a[e][i], non); kw[i] = mul2(k[e][i], inv); bw[i] = mul2(b[e][i], inv);
                    // P_L (where it underflows, so does dS P_L)
                    if (e == 0 && (lane & 11) == 11) *reinterpret_cast<float2*>(sm.fw + 4 * sl.quad + 2 * i) = make_float2(incl.x * STATE_SCALE, incl.y * STATE_SCALE);
                }
                const int dst = sl.dst(e);
                *reinterpret_cast<float4*>(sm.wq + dst) = pre4(wq);
                *reinterpret_cast<float4*>(sm.wa + dst) = pre4(wa);
                *reinterpret_cast<float4*>(sm.kwi + dst) = pre4(kw);
                *reinterpret_cast<float4*>(sm.bwi + dst) = pre4(bw);
                *reinterpret_cast<float4*>(sm.cum + dst) = make_float4(cum[e][0].x, cum[e][0].y, cum[e][1].x, cum[e][1].y);
            }
        }
        __syncthreads();  // (A)
        if (!PAR && (d.flags & FIRST)) {
#pragma unroll
            for (int i = 0; i < (LN ? 8 : 0); ++i) dlnw[i] = dlnb[i] = 0.f;
            if (LN) dbon[0][0] = dbon[0][1] = dbon[LN ? 1 : 0][0] = dbon[LN ? 1 : 0][1] = 0.f;
            taken_up = d.flags & CUT_BEFORE;
            const float* src = p.dsT;
            float scale = STATE_UNSCALE;
            if (d.flags & CUT_BEFORE) {  // the CTA before this one left its dS in ds0, as carried
                wait_handoff(ws.flags + blockIdx.x - 1, &sm.abort, p.status);
                src = p.ds0;
                scale = 1.f;
            }
            if (src) src += (long long)d.bh * N * N + (16 * warp + g) * N + 2 * t4;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float2 lo = src ? __ldcg(reinterpret_cast<const float2*>(src + 8 * nt)) : make_float2(0.f, 0.f);
                const float2 hi = src ? __ldcg(reinterpret_cast<const float2*>(src + 8 * N + 8 * nt)) : make_float2(0.f, 0.f);
                dS[nt][0] = lo.x * scale; dS[nt][1] = lo.y * scale; dS[nt][2] = hi.x * scale; dS[nt][3] = hi.y * scale;
            }
        }
        // ---------------- stage B: rows = value index ------------------------------------------------------------------
        mbar_wait_bounded<false>(&sm.rec_full, n & 1, &sm.abort, p.status);
        if (PAR) {
            const float* q = sm.dS + s0_mk;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float2 lo = *reinterpret_cast<const float2*>(q + 8 * nt), hi = *reinterpret_cast<const float2*>(q + 4 * SS + 8 * nt);
                dS[nt][0] = lo.x; dS[nt][1] = lo.y; dS[nt][2] = hi.x; dS[nt][3] = hi.y;
            }
        }
        const unsigned char *vt = sm.vdy[LN ? 0 : n & 1][0], *dyt = sm.vdy[LN ? 0 : n & 1][1];
        FragA<1> dyf[2], vf[2];
        frags_value_time(vf, vt, warp, lane);
        float X[2][4] = {}, U[2][4] = {};
        if (!LN) {
            frags_value_time(dyf, dyt, warp, lane);
        } else {
            // ---- recurrence output rebuilt: X, Y = S0 [wa;wq]^T + V^T [AK;QK]^T, U = X AI^T, Y += U QB^T (rows = value)
            float Y[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                FragA<1> s;
                const float2 lo = *reinterpret_cast<const float2*>(sm.S0 + s0_mk + 8 * kk), hi = *reinterpret_cast<const float2*>(sm.S0 + s0_mk + 4 * SS + 8 * kk);
                s.x[0].setr(lo.x); s.x[1].setr(hi.x); s.x[2].setr(lo.y); s.x[3].setr(hi.y);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    mma<1>(X[nt], s, B_nk(sm.wa, nt, kk));
                    mma<1>(Y[nt], s, B_nk(sm.wq, nt, kk));
                }
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) {
                    mma<1>(X[nt], vf[kk], mat_nk(0, nt, kk));
                    mma<1>(Y[nt], vf[kk], mat_nk(1, nt, kk));
                }
            const FragA<1> xa[2] = {fragA_from_acc<1>(X[0]), fragA_from_acc<1>(X[1])};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) mma<1>(U[nt], xa[kk], mat_kn(2, nt, kk));
            const FragA<1> ua[2] = {fragA_from_acc<1>(U[0]), fragA_from_acc<1>(U[1])};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) mma<1>(Y[nt], ua[kk], mat_nk(3, nt, kk));
            float* const yt = sm.yt();
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float* q = yt + 8 * nt * OPS + 16 * warp;
                q[kn(0)] = Y[nt][0]; q[kn(0) + OPS] = Y[nt][1];
                q[kn(1)] = Y[nt][2]; q[kn(1) + OPS] = Y[nt][3];
            }
            __syncthreads();  // (D1)
            // ---- GroupNorm / bonus / gate backward (reference: wind_rwkv/rwkv7/attn_ln.cu:40-104): one thread = one time step x 8
            // value channels, the eight threads of a time step are neighbouring lanes
            {
                const int row = tid >> 3, part = tid & 7, at = row * OPS + xcol<1>(row, 8 * part), bt8 = row * ROWB + ((part ^ (row & 7)) << 4);
                float y[8], v8[8], dy8[8], g8[8], lnw[8], lnb[8];
                load8<float>(reinterpret_cast<const unsigned char*>(yt + at), y);
                load8<__nv_bfloat16>(vt + bt8, v8);
                load8<__nv_bfloat16>(dyt + bt8, dy8);
                load8<__nv_bfloat16>(sm.vdy[0][LN ? 2 : 0] + bt8, g8);
                load8<float>(reinterpret_cast<const unsigned char*>(p.params + d.hi * N + 8 * part), lnw);
                load8<float>(reinterpret_cast<const unsigned char*>(p.params + (p.H + d.hi) * N + 8 * part), lnb);
                auto sum8 = [](float x) {
                    x += __shfl_xor_sync(0xffffffffu, x, 1);
                    x += __shfl_xor_sync(0xffffffffu, x, 2);
                    return x + __shfl_xor_sync(0xffffffffu, x, 4);
                };
                float mu = 0.f, var = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) mu += y[i];
                mu = sum8(mu) * (1.f / N);
#pragma unroll
                for (int i = 0; i < 8; ++i) { y[i] -= mu; var = fmaf(y[i], y[i], var); }
                const float rstd = 1.f / sqrtf(sum8(var) * (1.f / N) + p.eps);
                const float bd = sm.bdot[0][row] + sm.bdot[LN ? 1 : 0][row] + sm.bdot[LN ? 2 : 0][row] + sm.bdot[LN ? 3 : 0][row];
                float a1 = 0.f, a2 = 0.f, a3 = 0.f, dvx[8];
                uint32_t dg[4];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float x = y[i] * rstd, z = fmaf(x, lnw[i], fmaf(bd, v8[i], lnb[i])), dz = dy8[i] * g8[i], dx = dz * lnw[i];
                    g8[i] = dy8[i] * z;  // dg
                    dlnw[LN ? i : 0] = fmaf(dz, x, dlnw[LN ? i : 0]);
                    dlnb[LN ? i : 0] += dz;
                    dvx[i] = dz * bd;
                    a1 += dx; a2 = fmaf(dx, x, a2); a3 = fmaf(dz, v8[i], a3);
                    y[i] = x; dy8[i] = dx;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __nv_bfloat162 v2 = __floats2bfloat162_rn(g8[2 * i], g8[2 * i + 1]);
                    dg[i] = *reinterpret_cast<const uint32_t*>(&v2);
                }
                *reinterpret_cast<uint4*>(sm.out[LN ? 6 : 0] + bt8) = make_uint4(dg[0], dg[1], dg[2], dg[3]);
                const float m1 = sum8(a1) * (1.f / N), m2 = sum8(a2) * (1.f / N);
                a3 = sum8(a3);
                if (part == 0) sm.sbon[row] = a3;
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = pre<1>(rstd * (dy8[i] - m1 - y[i] * m2));  // gradient of the recurrence output
                store8(yt + at, y, (row >> 2) & 1);
                store8(sm.sgrad[0] + at, dvx, (row >> 2) & 1);   // the bonus term's part of dv (score gradients come later)
            }
            __syncthreads();  // (D2)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                const float* q = yt + 8 * kk * OPS + 16 * warp;
                dyf[kk].x[0].setr(q[kn(0)]); dyf[kk].x[1].setr(q[kn(1)]); dyf[kk].x[2].setr(q[kn(0) + OPS]); dyf[kk].x[3].setr(q[kn(1) + OPS]);
            }
        }
        // dS <- dSf = dS fw;  du = QB^T dY + bwi dSf^T,  dV = QK^T dY + kwi dSf^T + AK^T dabu,  X = S0 wa^T + V^T AK^T
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 f = *reinterpret_cast<const float2*>(sm.fw + 8 * nt + 2 * t4);
            dS[nt][0] *= f.x; dS[nt][1] *= f.y; dS[nt][2] *= f.x; dS[nt][3] *= f.y;
        }
        float du[2][4] = {}, dV[2][4] = {};
#pragma unroll
        for (int sb = 0; sb < 2; ++sb)
#pragma unroll
            for (int tb = sb; tb < 2; ++tb) {
                mma<1>(du[sb], dyf[tb], mat_kn(3, sb, tb));
                mma<1>(dV[sb], dyf[tb], mat_kn(1, sb, tb));
                if (!LN) mma<1>(X[tb], vf[sb], mat_nk(0, tb, sb));
            }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const FragA<1> f = fragA_from_acc<1>(dS[kk]);
            // the rounded dSf is what the products below and in stage C use
            float* q = sm.dS + s0_mk + 8 * kk;  // rows g, g + 8 lie four tile rows apart
            *reinterpret_cast<float2*>(q) = make_float2(__uint_as_float(f.x[0].h), __uint_as_float(f.x[2].h));
            *reinterpret_cast<float2*>(q + 4 * SS) = make_float2(__uint_as_float(f.x[1].h), __uint_as_float(f.x[3].h));
            FragA<1> s;
            if (!LN) {
                const float2 lo = *reinterpret_cast<const float2*>(sm.S0 + s0_mk + 8 * kk), hi = *reinterpret_cast<const float2*>(sm.S0 + s0_mk + 4 * SS + 8 * kk);
                s.x[0].setr(lo.x); s.x[1].setr(hi.x); s.x[2].setr(lo.y); s.x[3].setr(hi.y);
            }
#pragma unroll
            for (int sb = 0; sb < 2; ++sb) {
                mma<1>(du[sb], f, B_nk(sm.bwi, sb, kk));
                mma<1>(dV[sb], f, B_nk(sm.kwi, sb, kk));
                if (!LN) mma<1>(X[sb], s, B_nk(sm.wa, sb, kk));
            }
        }
        float dabu[2][4] = {};
        {
            const FragA<1> da2[2] = {fragA_from_acc<1>(du[0]), fragA_from_acc<1>(du[1])}, xa[2] = {fragA_from_acc<1>(X[0]), fragA_from_acc<1>(X[1])};
#pragma unroll
            for (int nb = 0; nb < 2; ++nb)
#pragma unroll
                for (int kb = nb; kb < 2; ++kb) {
                    mma<1>(dabu[nb], da2[kb], mat_nk(2, nb, kb));
                    if (!LN) mma<1>(U[kb], xa[nb], mat_kn(2, kb, nb));
                }
        }
        const FragA<1> dbf[2] = {fragA_from_acc<1>(dabu[0]), fragA_from_acc<1>(dabu[1])};
#pragma unroll
        for (int sb = 0; sb < 2; ++sb)
#pragma unroll
            for (int tb = sb; tb < 2; ++tb) mma<1>(dV[sb], dbf[tb], mat_kn(0, sb, tb));
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            float *q = sm.dabu + 8 * nt * OPS + 16 * warp, *w = sm.u + 8 * nt * OPS + 16 * warp;
            q[kn(0)] = __uint_as_float(dbf[nt].x[0].h); q[kn(0) + OPS] = __uint_as_float(dbf[nt].x[2].h);
            q[kn(1)] = __uint_as_float(dbf[nt].x[1].h); q[kn(1) + OPS] = __uint_as_float(dbf[nt].x[3].h);
            w[kn(0)] = pre<1>(U[nt][0]); w[kn(0) + OPS] = pre<1>(U[nt][1]);
            w[kn(1)] = pre<1>(U[nt][2]); w[kn(1) + OPS] = pre<1>(U[nt][3]);
        }
        if (LN) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const float* q = sm.sgrad[0] + 8 * nt * OPS + 16 * warp;
                dV[nt][0] += q[kn(0)]; dV[nt][1] += q[kn(0) + OPS]; dV[nt][2] += q[kn(1)]; dV[nt][3] += q[kn(1) + OPS];
            }
        }
        {   // dv: accumulator fragments through a transposing matrix store into the [time][value] tile
            uint32_t h[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 v2 = __floats2bfloat162_rn(dV[i >> 1][2 * (i & 1)], dV[i >> 1][2 * (i & 1) + 1]);
                h[i] = *reinterpret_cast<const uint32_t*>(&v2);
            }
            const int t = (lane & 7) + 8 * (lane >> 4), unit = 2 * warp + ((lane >> 3) & 1);
            asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                         ::"r"(smem_u32(sm.out[5] + t * ROWB + ((unit ^ (t & 7)) << 4))), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
        }
        // dS0 = dSf + dY^T wq + dabu^T wa
#pragma unroll
        for (int nt = 0; nt < (PAR ? 0 : 8); ++nt)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                mma<1>(dS[nt], dyf[kk], B_kn(sm.wq, nt, kk));
                mma<1>(dS[nt], dbf[kk], B_kn(sm.wa, nt, kk));
            }
        __syncthreads();  // (C1)
        // ---------------- stage C: contractions over the value index, warp owns 16 key columns -----------------------------
        float DA[2][4] = {}, DQ[2][4] = {}, DB[2][4] = {}, DK[2][4] = {};
        float gs[2] = {0.f, 0.f};  // sum_i dSf[i, key] S0[i, key], key = 16 warp + 8 nt + g, this lane's share of the rows
        {
            // one score gradient per warp: 0 dQK = tril(dY V^T), 1 dAK = stril(dabu V^T), 2 dQB = tril(dY U^T), 3 dAB = stril(dabu U^T)
            float sc[2][4] = {};
            const bool strict = warp & 1, useu = warp >> 1;
            const int lrow = (lane & 15) * ROWB, lunit = ((lane >> 4) ^ (lane & 7)) << 4;
            const float *s0p = sm.S0 + s0_kn, *dsp = sm.dS + s0_kn, *dp = sm.dabu, *up = sm.u, *ytp = sm.yt();
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass, s0p += 16 * SS, dsp += 16 * SS, dp += 32, up += 32, ytp += 32) {
            const unsigned char *yp = dyt + lrow + (lunit ^ (pass << 6)), *vp = vt + lrow + (lunit ^ (pass << 6));
#pragma unroll
            for (int kp = 0; kp < 2; ++kp) {
                uint32_t ry[4], rv[4];
                if (!LN) ldmatrix4<false>(ry, kp ? dyt + lrow + ((lunit ^ (pass << 6)) ^ 32) : yp);
                ldmatrix4<false>(rv, kp ? vt + lrow + ((lunit ^ (pass << 6)) ^ 32) : vp);
#pragma unroll
                for (int k2 = 0; k2 < 2; ++k2) {
                    const int kk = 2 * kp + k2;
                    const FragA<1> aD = A_mk(dp, kk), aU = A_mk(up, kk);
                    const FragA<1> aY = LN ? A_mk(ytp, kk) : frag_bf16(ry[2 * k2], ry[2 * k2 + 1]), aV = frag_bf16(rv[2 * k2], rv[2 * k2 + 1]);
                    FragA<1> sa, sb;
#pragma unroll
                    for (int i = 0; i < 4; ++i) { sa.x[i].h = strict ? aD.x[i].h : aY.x[i].h; sb.x[i].h = useu ? aU.x[i].h : aV.x[i].h; }
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        mma<1>(sc[nt], sa, as_b(sb, nt));
                        FragB<1> bS, bD;
                        const float s0 = s0p[4 * kk * SS + 8 * nt], s1 = s0p[(4 * kk + 1) * SS + 8 * nt];
                        const float e0 = dsp[4 * kk * SS + 8 * nt], e1 = dsp[(4 * kk + 1) * SS + 8 * nt];
                        gs[nt] = fmaf(e0, s0, fmaf(e1, s1, gs[nt]));
                        bS.x[0].setr(s0); bS.x[1].setr(s1);
                        bD.x[0].setr(e0); bD.x[1].setr(e1);
                        mma<1>(DA[nt], aD, bS);
                        mma<1>(DQ[nt], aY, bS);
                        mma<1>(DB[nt], aU, bD);
                        mma<1>(DK[nt], aV, bD);
                    }
                }
            }
            }
            float* q = sm.sgrad[warp];
            const int off = 2 * t4 + (strict ? 1 : 0);  // keep column s where s + strict <= row
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int c = off + 8 * nt, at = nt ? smk1 : smk0;
                *reinterpret_cast<float2*>(q + at) = make_float2(c <= g ? pre<1>(sc[nt][0]) : 0.f, c < g ? pre<1>(sc[nt][1]) : 0.f);
                *reinterpret_cast<float2*>(q + 8 * SCS + at) = make_float2(c <= g + 8 ? pre<1>(sc[nt][2]) : 0.f, c < g + 8 ? pre<1>(sc[nt][3]) : 0.f);
            }
        }
        if (PAR) fence_async_smem();  // dS was written here and comes by bulk copy next
        __syncthreads();  // (C2) score gradients visible; the record's tiles are free
        // the carried part of the decay gradient (see the head of this file)
        float kw[2][2][2], bw[2][2][2], G[2][2];  // kwi, bwi: [tile][row half][column]; [tile][column]
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            float e[2] = {0.f, 0.f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int at = 8 * h * OPS + 16 * warp + mk(nt);
                const float2 x = *reinterpret_cast<const float2*>(sm.kwi + at), y = *reinterpret_cast<const float2*>(sm.bwi + at);
                kw[nt][h][0] = x.x; kw[nt][h][1] = x.y; bw[nt][h][0] = y.x; bw[nt][h][1] = y.y;
#pragma unroll
                for (int i = 0; i < 2; ++i) e[i] = fmaf(kw[nt][h][i], DK[nt][2 * h + i], fmaf(bw[nt][h][i], DB[nt][2 * h + i], e[i]));
            }
            gs[nt] += __shfl_xor_sync(0xffffffffu, gs[nt], 1);
            gs[nt] += __shfl_xor_sync(0xffffffffu, gs[nt], 2);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int m = 4; m <= 16; m <<= 1) e[i] += __shfl_xor_sync(0xffffffffu, e[i], m);
                G[nt][i] = e[i] + __shfl_sync(0xffffffffu, gs[nt], (2 * t4 + i) << 2);
            }
        }
#pragma unroll 1
        for (int kk = 0; kk < 2; ++kk) {
            FragA<1> a[4], t[4];  // dQK, dAK, dQB, dAB and their transposes
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float *q = sm.sgrad[m] + (kk ? smk1 : smk0), *w = sm.sgrad[m] + 8 * kk * SCS;
                const float2 lo = *reinterpret_cast<const float2*>(q), hi = *reinterpret_cast<const float2*>(q + 8 * SCS);
                a[m].x[0].setr(lo.x); a[m].x[1].setr(hi.x); a[m].x[2].setr(lo.y); a[m].x[3].setr(hi.y);
                t[m].x[0].setr(w[skn0]); t[m].x[1].setr(w[skn1]); t[m].x[2].setr(w[skn0 + SCS]); t[m].x[3].setr(w[skn1 + SCS]);
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const FragB<1> bb = B_kn(sm.bwi + 16 * warp, nt, kk), bk = B_kn(sm.kwi + 16 * warp, nt, kk);
                const FragB<1> ba = B_kn(sm.wa + 16 * warp, nt, kk), bq = B_kn(sm.wq + 16 * warp, nt, kk);
                mma<1>(DA[nt], a[3], bb); mma<1>(DQ[nt], a[2], bb); mma<1>(DB[nt], t[3], ba); mma<1>(DK[nt], t[1], ba);
                mma<1>(DA[nt], a[1], bk); mma<1>(DQ[nt], a[0], bk); mma<1>(DB[nt], t[2], bq); mma<1>(DK[nt], t[0], bq);
            }
        }
        // ---------------- outputs: thread holds rows g, g + 8 x columns key, key + 1 ---------------------------------------
#pragma unroll 1
        for (int nt = 0; nt < 2; ++nt) {  // (rolled: the second tile's values move into the first one's registers)
            const int amk = 16 * warp + (nt ? mkO + 8 : mkE), apm = 16 * warp + (nt ? pm1 : pm0), unit = (((2 * warp + nt) ^ g) << 4) + 4 * t4;
            float x[2][2], e2[2][2], lw[2][2], db[2] = {0.f, 0.f};  // [row half][column]
            const float2 bonus = LN ? __ldg(reinterpret_cast<const float2*>(p.params + (2 * p.H + d.hi) * N + 16 * warp + 8 * nt + 2 * t4)) : make_float2(0.f, 0.f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int at = 8 * h * OPS + amk;
                const float2 cu = *reinterpret_cast<const float2*>(sm.cum + at);  // running log2 decay; row -1 is zero
                const float2 cp = g + 8 * h > 0 ? *reinterpret_cast<const float2*>(sm.cum + 8 * h * OPS + apm) : make_float2(0.f, 0.f);
                const float2 oq = *reinterpret_cast<const float2*>(sm.wq + at), oa = *reinterpret_cast<const float2*>(sm.wa + at);
                const float cuv[2] = {cu.x, cu.y}, cpv[2] = {cp.x, cp.y}, wqv[2] = {oq.x, oq.y}, wav[2] = {oa.x, oa.y};
                float r[4][2];  // dq, dk, da, db
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int e = i + 2 * h;
                    const float cc = fmaxf(cuv[i] + ANCHOR_LOG2, -115.f);  // P~_t and its reciprocal, as the scan formed them
                    const float incl = ex2_approx(cc), inv = ex2_approx(-cc), non = ex2_approx(fmaxf(cpv[i] + ANCHOR_LOG2, -115.f));
                    r[0][i] = incl * DQ[0][e];
                    r[1][i] = inv * DK[0][e];
                    r[2][i] = non * DA[0][e];
                    r[3][i] = inv * DB[0][e];
                    if (LN) {  // bonus term: y += (sum_j q_j k_j bonus_j) v
                        const float sb = sm.sbon[g + 8 * h], bo = i ? bonus.y : bonus.x, q_raw = wqv[i] * inv, k_raw = kw[0][h][i] * incl;
                        r[0][i] = fmaf(sb * k_raw, bo, r[0][i]);
                        r[1][i] = fmaf(sb * q_raw, bo, r[1][i]);
                        db[i] = fmaf(sb * q_raw, k_raw, db[i]);
                    }
                    e2[h][i] = wav[i] * DA[0][e];
                    x[h][i] = fmaf(wqv[i], DQ[0][e], e2[h][i]) - fmaf(kw[0][h][i], DK[0][e], bw[0][h][i] * DB[0][e]);
                    lw[h][i] = (cuv[i] - cpv[i]) * 0.6931471805599453f;
                }
                unsigned char* dst = sm.out[0] + (g + 8 * h) * ROWB + unit;
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<__nv_bfloat162*>(dst + (i == 0 ? 0 : i + 1) * TILE) = __floats2bfloat162_rn(r[i][0], r[i][1]);
            }
            // inclusive suffix sum over the 16 time rows (rows live in lanes g = 0..7, two halves)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int s = 1; s < 8; s <<= 1) {
                    const float yl = __shfl_down_sync(0xffffffffu, x[0][i], 4 * s), yh = __shfl_down_sync(0xffffffffu, x[1][i], 4 * s);
                    if (g + s < 8) { x[0][i] += yl; x[1][i] += yh; }
                }
                x[0][i] += __shfl_sync(0xffffffffu, x[1][i], t4);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<__nv_bfloat162*>(sm.out[1] + (g + 8 * h) * ROWB + unit) =
                    __floats2bfloat162_rn((x[h][0] - e2[h][0] + G[0][0]) * lw[h][0], (x[h][1] - e2[h][1] + G[0][1]) * lw[h][1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                DA[0][e] = DA[1][e]; DQ[0][e] = DQ[1][e]; DB[0][e] = DB[1][e]; DK[0][e] = DK[1][e];
                kw[0][e >> 1][e & 1] = kw[1][e >> 1][e & 1]; bw[0][e >> 1][e & 1] = bw[1][e >> 1][e & 1];
            }
            G[0][0] = G[1][0]; G[0][1] = G[1][1];
            if (LN) {  // (the accumulators change places, too: twice per chunk)
                const float s0 = dbon[LN ? 1 : 0][0], s1 = dbon[LN ? 1 : 0][1];
                dbon[LN ? 1 : 0][0] = dbon[0][0] + db[0]; dbon[LN ? 1 : 0][1] = dbon[0][1] + db[1];
                dbon[0][0] = s0; dbon[0][1] = s1;
            }
        }
        fence_async_smem();
        __syncthreads();  // (E)
        if (PAR) continue;
        if (LN && (d.flags & LAST)) {
            // per-(batch, head) partial parameter gradients ws[b][0..2][h*N + channel]; of a cut chain, the later piece adds to
            // what the earlier one (whose state gradient it has taken up) left there
            float* part = sm.dabu;  // [warp][2][64]
#pragma unroll
            for (int i = 0; i < (LN ? 8 : 0); ++i) {
                float x = dlnw[i], y = dlnb[i];
                x += __shfl_xor_sync(0xffffffffu, x, 8); x += __shfl_xor_sync(0xffffffffu, x, 16);
                y += __shfl_xor_sync(0xffffffffu, y, 8); y += __shfl_xor_sync(0xffffffffu, y, 16);
                if (lane < 8) { part[warp * 128 + 8 * lane + i] = x; part[warp * 128 + 64 + 8 * lane + i] = y; }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            float* wsp = p.dparams_ws + (long long)d.bi * 3 * p.H * N + d.hi * N;
            const bool add = taken_up;
            {
                float x = part[tid] + part[128 + tid] + part[256 + tid] + part[384 + tid];
                float* q = wsp + (tid >> 6) * p.H * N + (tid & 63);
                *q = add ? __ldcg(q) + x : x;
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float x = dbon[LN ? nt : 0][i];
                    x += __shfl_xor_sync(0xffffffffu, x, 4); x += __shfl_xor_sync(0xffffffffu, x, 8); x += __shfl_xor_sync(0xffffffffu, x, 16);
                    float* q = wsp + 2 * p.H * N + 16 * warp + 8 * nt + 2 * t4 + i;
                    if (g == 0) *q = add ? __ldcg(q) + x : x;
                }
        }
        if ((d.flags & LAST) && p.ds0) {
            float* dst = p.ds0 + (long long)d.bh * N * N + (16 * warp + g) * N + 2 * t4;
            const float scale = d.flags & CUT_AFTER ? 1.f : STATE_SCALE;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                *reinterpret_cast<float2*>(dst + 8 * nt) = make_float2(dS[nt][0] * scale, dS[nt][1] * scale);
                *reinterpret_cast<float2*>(dst + 8 * N + 8 * nt) = make_float2(dS[nt][2] * scale, dS[nt][3] * scale);
            }
            if (d.flags & CUT_AFTER) {
                __threadfence();
                __syncthreads();
                if (tid == 0) publish_handoff(ws.flags + blockIdx.x);
            }
        }
    }
}

// ---- the state gradient alone ----------------------------------------------------------------------------------------------------
// The products that carry dS from chunk to chunk, as the chunk kernel forms them, in its order and with its rounding (so that results do
// not depend on the number of chains): du = QB^T dY + bwi dSf^T, dabu = AI^T.. du, dS' = dSf + dY^T wq + dabu^T wa.  One CTA per
// chain: 4 chain warps (16 value rows of dS each, no exchange between them), PREP groups of 4 preparing warps (the scan, 16 key columns
// each) that take every PREP-th chunk, two warps that issue the loads; SLOTS chunks in flight.  Leaves dS at the end of every chunk in
// `tiles`, for chunks it0 .. it0 + n - 1 (counted from the end of the sequence).
// Bound by the chain of dependent products, some 1500 cycles a chunk (the one-kernel form: 6200).  Backward of 48 chains of 63 chunks
// 203 -> 115 us, of 8 chains of 256 chunks 745 -> 230 us, of 148 chains of 63 chunks 236 -> 205 us.
constexpr int SLOTS = 6, PREP = 2, WALK_THREADS = 32 * (WARPS * (1 + PREP) + 2);
struct WalkSlot {
    alignas(1024) unsigned char raw[5][TILE];  // q, w, a, b, dy
    alignas(128) float mats[2 * L * L];        // AI^T, QB as the record holds them
    alignas(16) float wq[L * OPS], wa[L * OPS], bwi[L * OPS], fw[N];
};
struct WalkSmem {
    WalkSlot slot[SLOTS];
    uint64_t raw_full[SLOTS], ready[SLOTS], free[SLOTS];
    volatile int abort, drain;
};
static_assert(sizeof(WalkSmem) + 1024 <= 232448, "one CTA per SM");

template <bool TAIL>
__global__ void __launch_bounds__(WALK_THREADS, 1) wkv7_bwd_walk_kernel(BwdParams p, float* tiles, int it0, int count, const __grid_constant__ BwdMaps maps) {
    stream_wait();
    extern __shared__ unsigned char smem_dyn[];
    WalkSmem& sm = *reinterpret_cast<WalkSmem*>(smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, t4 = lane & 3, w = warp & 3;
    const int bh = blockIdx.x, bi = bh / (int)p.H, hi = bh - bi * (int)p.H, nchunks = (int)((p.T + L - 1) / L), c0 = nchunks - 1 - it0;
    if (tid == 0) {
        for (int i = 0; i < SLOTS; ++i) {
            mbar_init(&sm.raw_full[i], 1);
            mbar_init(&sm.ready[i], WARPS);
            mbar_init(&sm.free[i], WARPS);
        }
        sm.abort = sm.drain = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int bg = (g >> 2) & 1, bt = (t4 >> 1) & 1;  // element offsets as in wkv7_bwd_bf16_kernel
    const int mkE = g * OPS + 2 * t4 + 8 * bg, mkO = mkE - 16 * bg, knE = 2 * t4 * OPS + g + 8 * bt, knO = knE - 16 * bt;
    auto mk = [&](int kk) { return (kk & 1 ? mkO : mkE) + 8 * kk; };
    auto kn = [&](int nb) { return (nb & 1 ? knO : knE) + 8 * nb; };
    auto B_kn = [&](const float* tile, int nb, int kk) {
        FragB<1> f;
        const float* q = tile + 8 * kk * OPS + kn(nb);
        f.x[0].setr(q[0]); f.x[1].setr(q[OPS]);
        return f;
    };

    if (warp >= WARPS * (1 + PREP)) {
        // ---- loads
        if (lane != 0) return;
        const int map_of[5] = {0, 1, 3, 4, 6};
        int n = warp & 1;
        for (; n < count; n += 2) {
            const int s = n % SLOTS, c = c0 - n;
            if (n >= SLOTS && !mbar_wait_bounded<true>(&sm.free[s], (n / SLOTS - 1) & 1, &sm.abort, p.status)) break;
            WalkSlot& t = sm.slot[s];
            expect(&sm.raw_full[s], 5 * TILE + sizeof(t.mats));
#pragma unroll
            for (int i = 0; i < 5; ++i) load4(t.raw[i], &maps.in[map_of[i]], &sm.raw_full[s], hi, c * L, bi);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(t.mats)), "l"(p.ckpt + ((long long)bh * nchunks + c) * CK_FLOATS + CK_AI), "r"((int)sizeof(t.mats)), "r"(smem_u32(&sm.raw_full[s]))
                         : "memory");
        }
        stream_release();  // (at most SLOTS chunks before the end)
        // shared memory must outlive the loads, also where a wait has given up (n: the first of this warp's loads not issued)
        for (int i = max(warp & 1, n - SLOTS); i < n; i += 2) mbar_wait_bounded<true>(&sm.raw_full[i % SLOTS], (i / SLOTS) & 1, &sm.drain, p.status);
        return;
    }
    if (warp >= WARPS) {
        // ---- preparation: this warp's 16 key columns of every PREP-th chunk
        const ScanLane sl(w, lane);
        for (int n = warp / WARPS - 1; n < count; n += PREP) {
            const int s = n % SLOTS;
            WalkSlot& t = sm.slot[s];
            mbar_wait_bounded<true>(&sm.raw_full[s], (n / SLOTS) & 1, &sm.abort, p.status);
            F2 cum[2][2], before[2][2];
#pragma unroll
            for (int e = 0; e < 2; ++e) load4f2(t.raw[1] + sl.raw(e), cum[e]);
            sl.decay(cum, before, TAIL ? (int)min((long long)L, p.T - (long long)(c0 - n) * L) : L, lane);  // as wkv7_bwd_bf16_kernel does
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int at = sl.raw(e), dst = sl.dst(e);
                F2 q[2], a[2], b[2], wq[2], wa[2], bw[2];
                load4f2(t.raw[0] + at, q);
                load4f2(t.raw[2] + at, a);
                load4f2(t.raw[3] + at, b);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const F2 ca = add2(cum[e][i], f2(ANCHOR_LOG2, ANCHOR_LOG2)), cp = add2(before[e][i], f2(ANCHOR_LOG2, ANCHOR_LOG2));
                    const float cx = fmaxf(ca.x, -115.f), cy = fmaxf(ca.y, -115.f);
                    const F2 incl = f2(ex2_approx(cx), ex2_approx(cy)), inv = f2(ex2_approx(-cx), ex2_approx(-cy));
                    const F2 non = f2(ex2_approx(fmaxf(cp.x, -115.f)), ex2_approx(fmaxf(cp.y, -115.f)));
                    wq[i] = mul2(q[i], incl); wa[i] = mul2(a[i], non); bw[i] = mul2(b[i], inv);
                    if (e == 0 && (lane & 11) == 11) *reinterpret_cast<float2*>(t.fw + 4 * sl.quad + 2 * i) = make_float2(incl.x * STATE_SCALE, incl.y * STATE_SCALE);
                }
                *reinterpret_cast<float4*>(t.wq + dst) = pre4(wq);
                *reinterpret_cast<float4*>(t.wa + dst) = pre4(wa);
                *reinterpret_cast<float4*>(t.bwi + dst) = pre4(bw);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.ready[s]);
        }
        return;
    }
    // ---- the chain: value rows 16 w + {g, g + 8} of dS, carried as in wkv7_bwd_bf16_kernel
    float dS[8][4];
    const long long st = (long long)bh * N * N + (16 * w + g) * N + 2 * t4;
    {
        const float* src = it0 ? p.ds0 : p.dsT;  // a later pass goes on from where the earlier one left it
        const float scale = it0 ? 1.f : STATE_UNSCALE;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 lo = src ? *reinterpret_cast<const float2*>(src + st + 8 * nt) : make_float2(0.f, 0.f);
            const float2 hi = src ? *reinterpret_cast<const float2*>(src + st + 8 * N + 8 * nt) : make_float2(0.f, 0.f);
            dS[nt][0] = lo.x * scale; dS[nt][1] = lo.y * scale; dS[nt][2] = hi.x * scale; dS[nt][3] = hi.y * scale;
        }
    }
    float* out = tiles + (long long)bh * count * TILE_FLOATS + s0_at(16 * w + g, 2 * t4);
    for (int n = 0; n < count; ++n, out += TILE_FLOATS) {
        const int s = n % SLOTS;
        const WalkSlot& t = sm.slot[s];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            *reinterpret_cast<float2*>(out + 8 * nt) = make_float2(dS[nt][0], dS[nt][1]);
            *reinterpret_cast<float2*>(out + 4 * SS + 8 * nt) = make_float2(dS[nt][2], dS[nt][3]);
        }
        mbar_wait_bounded<false>(&sm.ready[s], (n / SLOTS) & 1, &sm.abort, p.status);
        FragA<1> dyf[2];
        frags_value_time(dyf, t.raw[4], w, lane);
        // matrix m (0 AI^T, 1 QB): element (row, col) of the record's operand tiles
        auto mat = [&](int m, int row, int col) { return t.mats + m * L * L + (row >> 3) * 128 + (col >> 2) * 32 + (row & 7) * 4 + (col & 3); };
        float du[2][4] = {}, dabu[2][4] = {};
#pragma unroll
        for (int sb = 0; sb < 2; ++sb)
#pragma unroll
            for (int tb = sb; tb < 2; ++tb) {
                FragB<1> b;
                b.x[0].setr(*mat(1, 8 * tb + 2 * t4, 8 * sb + g)); b.x[1].setr(*mat(1, 8 * tb + 2 * t4 + 1, 8 * sb + g));
                mma<1>(du[sb], dyf[tb], b);
            }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const float2 f = *reinterpret_cast<const float2*>(t.fw + 8 * kk + 2 * t4);
            dS[kk][0] *= f.x; dS[kk][1] *= f.y; dS[kk][2] *= f.x; dS[kk][3] *= f.y;
            const FragA<1> a = fragA_from_acc<1>(dS[kk]);
#pragma unroll
            for (int sb = 0; sb < 2; ++sb) {
                FragB<1> b;
                const float2 v = *reinterpret_cast<const float2*>(t.bwi + 8 * sb * OPS + mk(kk));
                b.x[0].setr(v.x); b.x[1].setr(v.y);
                mma<1>(du[sb], a, b);
            }
            mma<1>(dS[kk], dyf[0], B_kn(t.wq, kk, 0));
        }
        const FragA<1> da2[2] = {fragA_from_acc<1>(du[0]), fragA_from_acc<1>(du[1])};
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int kb = nb; kb < 2; ++kb) {
                FragB<1> b;
                const float2 v = *reinterpret_cast<const float2*>(mat(0, 8 * nb + g, 8 * kb + 2 * t4));
                b.x[0].setr(v.x); b.x[1].setr(v.y);
                mma<1>(dabu[nb], da2[kb], b);
            }
        const FragA<1> dbf[2] = {fragA_from_acc<1>(dabu[0]), fragA_from_acc<1>(dabu[1])};
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) mma<1>(dS[nt], dbf[0], B_kn(t.wa, nt, 0));
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) mma<1>(dS[nt], dyf[1], B_kn(t.wq, nt, 1));
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) mma<1>(dS[nt], dbf[1], B_kn(t.wa, nt, 1));
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

}  // namespace bf16bwd

// When the state gradients are walked ahead of the rest, and how many chunks of each chain at a time (0: not).  One CTA per chain and
// all of a chunk's work in it is bound by the latency of a chunk (6200 cycles) while SMs are idle; the walk takes 1/5 of that and
// the rest spreads over the machine.  With as many chains as SMs it still pays; beyond, a walk has its second round.
// The tiles of a pass are kept below 512 MB; longer sequences take several passes, the walk going on from ds0.
// attn_ln is never walked: its walk would need the gradient of the recurrence output first.
static int walk_chunks(long long chains, long long chunks, bool ln) {
    if (ln || chains == 0 || chains > sm_count() || chunks < 4) return 0;
    return (int)std::min(chunks, std::max(1LL, (512LL << 20) / (chains * bf16bwd::TILE_FLOATS * 4)));
}
size_t bwd_workspace_bytes(long long B, long long T, long long H, bool ln) {
    return WORK_FLAG_BYTES + (size_t)(B * H * walk_chunks(B * H, (T + L - 1) / L, ln)) * bf16bwd::TILE_FLOATS * sizeof(float);
}

template <bool LN> static int launch_bwd_bf16_t(const BwdParams& p, cudaStream_t stream) {
    using namespace bf16bwd;
    const long long chains = p.B * p.H, chunks = (p.T + L - 1) / L;
    const int walked = p.flags && p.ds0 ? walk_chunks(chains, chunks, LN) : 0;
    auto kern = p.T % L ? wkv7_bwd_bf16_kernel<true, LN, false> : wkv7_bwd_bf16_kernel<false, LN, false>;
    if (walked) kern = p.T % L ? wkv7_bwd_bf16_kernel<true, LN, !LN> : wkv7_bwd_bf16_kernel<false, LN, !LN>;
    const int smem = (int)sizeof(Smem<LN>) + 1024;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return kLaunchFailed;
    BwdMaps maps;
    memset(&maps, 0, sizeof(maps));
    const void* in[8] = {p.r, p.w, p.k, p.a, p.b, p.v, p.dy, p.g};
    void* out[7] = {p.dr, p.dw, p.dk, p.da, p.db, p.dv, p.dg};
    for (int i = 0; i < (LN ? 8 : 7); ++i)
        if (!encode_bthn_map(&maps.in[i], const_cast<void*>(in[i]), p.B, p.T, p.H, p.st)) return kLaunchFailed;
    for (int i = 0; i < (LN ? 7 : 6); ++i)
        if (!encode_bthn_map(&maps.out[i], out[i], p.B, p.T, p.H, p.st)) return kLaunchFailed;
    const long long records = p.B * p.H * ((p.T + L - 1) / L);
    if (!(encode_ckpt_state_map(&maps.ck, p.ckpt, records) && encode_ckpt_mats_map(&maps.ckm, p.ckpt, records))) return kLaunchFailed;
    if (walked) {
        auto walk = p.T % L ? wkv7_bwd_walk_kernel<true> : wkv7_bwd_walk_kernel<false>;
        const int wsmem = (int)sizeof(WalkSmem) + 1024, slots = 2 * sm_count();
        if (cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, wsmem) != cudaSuccess) return kLaunchFailed;
        float* tiles = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p.flags) + WORK_FLAG_BYTES);
        for (long long it0 = 0; it0 < chunks; it0 += walked) {
            const int n = (int)std::min<long long>(walked, chunks - it0), total = (int)chains * n, per = (total + slots - 1) / slots;
            if (!launch(walk, dim3((unsigned)chains), WALK_THREADS, wsmem, stream, p, tiles, (int)it0, n, maps)) return kLaunchFailed;
            if (!launch(kern, dim3((unsigned)((total + per - 1) / per)), NTHREADS, smem, stream, p, WorkSplit{0, per, n, total, nullptr}, Tiles{tiles, (int)it0}, maps)) return kLaunchFailed;
        }
        return kOk;
    }
    const WorkSplit ws = plan_work(chains, chunks, 2, p.ds0 ? p.flags : nullptr);
    if (ws.flags && cudaMemsetAsync(ws.flags, 0, ws.ctas * sizeof(unsigned), stream) != cudaSuccess) return kLaunchFailed;
    if (!launch(kern, dim3((unsigned)ws.ctas), NTHREADS, smem, stream, p, ws, Tiles{}, maps)) return kLaunchFailed;
    return LN ? launch_reduce_dparams(p, stream) : kOk;
}

int launch_bwd_bf16(const BwdParams& p, bool ln, cudaStream_t stream) {
    return ln ? launch_bwd_bf16_t<true>(p, stream) : launch_bwd_bf16_t<false>(p, stream);
}

}  // namespace wkv7
