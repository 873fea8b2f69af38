// WKV7 forward on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory), bf16 IO.
//
// Same mathematics as wkv7_fwd.cu (the reference's forward_kernel, wind_rwkv/rwkv7/attn.cu:11-106, and
// with LN = true its fused GroupNorm + bonus + gate variant, wind_rwkv/rwkv7/attn_ln.cu:106-212),
// different machine mapping.  One CTA per SM walks its share of the chunks (WorkSplit: whole chains and at most two pieces of
// cut ones).  The 64x64 state S[value][key] lives in tensor memory and is never held in registers: per 16-step chunk one
// elected thread issues 24 tcgen05.mma instructions (M = 64 value rows, TF32 operands, fp32 accumulate)
//     ahead   [X | Yp] = V^T [AK;QK]^T,  S' = V^T kwf        needs no state: issued while the chunk before it drains; A = V^T from
//                                                            tensor memory, S' in the next of four state buffers
//     hop 1   [X | Yp] += S [wa;wq]^T                        A = S straight from tensor memory
//             S' += S diag(fw)                               eight N = 8 products apply the decay; issued while hop 1 drains
//     hop 2   S' += X (AI^T bwf),  Y = Yp + X (QB AI)^T      A = X from tensor memory
// with kwf = kwi*fw, bwf = bwi*fw, so the column scaling of the state never touches a CUDA core.  U = X AI^T itself is never
// formed: AI^T bwf and QB AI come from two small products off the chain.  An accumulator that the next product reads as its A
// operand needs an explicit completion wait (tcgen05.commit -> mbarrier); only same-accumulator products are ordered by the
// tensor pipe.
// What bounds it: three things at once, none of which is saturated alone.  The chain's two round trips (1000 cycles a chunk in the
// running kernel, 560 alone: 210 for a product, its commit and the wait, 5 to 38 for each further product); the latency from a chunk's
// operand tiles to its completion, some 5500 cycles, over the four chunks in flight (a fifth group would leave 72 registers a thread, where
// preparation takes 96, and all 512 columns of tensor memory are in use); and the shared-memory data pipe, some 1000 wavefronts of
// loads and stores a chunk and 360 of operand reads, that both stand in.  About 1450 cycles a chunk without checkpoints
// (B8 T65536 H40), 1800 with (B64 T1024 H12: 338 us, 4.7 TB/s of HBM traffic).  Before the V parts went ahead of the chain and off shared
// memory, and the scores, the inverse and the fold each had warps of their own: 1550 and 1860.
//
// Warp roles (128 (G+2) threads).  Warps 0..4G-1 are G preparation groups of four warps, each working on its own chunk (c, c+G, ...).
// Eight service warps serve all groups, each a stage of a chunk's way to the chain (a warp takes some 500 cycles per stage, so that a
// stage shared with another one makes chunks wait): 4G, 4G+1 read the scores back from their quarter of tensor memory, mask them and write
// AK, AB, QK, QB; 4G+2, 4G+6 invert (I - AB) (even and odd groups); 4G+4, 4G+5, 4G+7 form the two fold products; 4G+3 issues
// the chain.  The kernel's hot code has to stay small: its warps run different parts of it at the same
// time out of one instruction cache, and 10 KB more of it cost 30 % once all SMs missed at the same time.
// (Not better: the scores by mma.sync in the preparation warps - every operand is read four times, 1.2 times slower; forming the
// inverse's two 8x8 blocks in lanes 0-15 only, 1 % slower.)
//
// Shared-memory operand layouts (the tiles are produced by threads, not copied):
//   K-major (contraction index contiguous): 16-byte chunks [row/8][k/4][row%8][k%4], descriptor
//     LBO = 128 B (next k-chunk), SBO = bytes per 8-row group, no swizzle.
//   MN-major TF32 (kwf, bwf: contraction index = time): only the 128-byte swizzle with 32-byte
//     base exists for 32-bit MN-major operands: rows of 32 channels (128 B) per time step, the
//     32-byte unit index XOR-ed with (t % 4); LBO = stride between the two 32-channel halves,
//     SBO = 512 B (four time steps).
// Checkpoint states leave through shared memory: tensor memory holds one state row per lane, so a warp-wide
// store from registers can write one 32-byte sector per lane at best (512 wavefronts of the SM's L1 data
// pipe per 16 KB state).  Instead each thread writes its row into a 128-byte-swizzled staging tile (two
// [64 rows][32 floats] halves in the dead [wa;wq] / [kwi;bwi] tiles, conflict-free 8-byte stores) and one
// thread issues two tensor-map bulk stores (cp.async.bulk.tensor.2d, shared -> global), which undo the
// swizzle: the record in global memory stays plain row-major.
// Every wait on an mbarrier is bounded; a wait that runs out raises an abort flag that makes all
// later waits of the CTA return at once, records kDeviceTimeout and lets the CTA finish (its loads and products
// in flight are waited for, tensor memory is released).
#include <cuda.h>
#include <cstring>

#include "wkv7_kernels.h"
namespace wkv7 {
namespace tc {

constexpr int ROWB = 2 * N;         // staging row of a bf16 input tile: 128 bytes, its eight 16-byte segments XOR-ed with (row % 8)
constexpr int RAW_TILE = L * ROWB;  // 2048

// per-group shared memory (byte offsets; tensor-core tiles first, all 1024-byte aligned)
constexpr int G_WAQ = 0;       // [wa;wq]   32 rows x 64, K-major            8192
constexpr int G_KB = 8192;     // [kwi;bwi] 32 rows x 64, K-major            8192 (directly after WAQ: the M = 64 score
                               //                                                 product reads rows 32..63 from here, unused);
                               // time step s of every eight in row kb_row(s): the score product's columns then come back as
                               // 8x4 blocks with a column per lane, which stmatrix can store
constexpr int G_V = 16384;     // attn_ln's epilogue only: V [time][value], bf16, 16-byte units XOR-ed with the row   2048 (of 4096)
constexpr int G_KWF = 20480;   // kwf [time][key]    MN-major                4096
constexpr int G_BWF = 24576;   // bwf [time][key]    MN-major                4096
constexpr int G_SC = 28672;    // [AK;QK]  32 rows x 16, K-major             2048
constexpr int G_AI = 30720;    // AI^T     16 x 16, K-major                  1024
constexpr int G_QB = 31744;    // QB       16 x 16, K-major                  1024
static_assert(G_AI == G_SC + 2048 && G_QB == G_AI + 1024, "[AK;QK], AI^T, QB must be contiguous: they leave as one bulk copy");
constexpr int G_DF = 32768;    // eight 8x8 diagonal blocks of fw, K-major   2048
constexpr int G_ABT = 34816;   // AB transposed, fp32 [16][ABS]              1536
constexpr int G_QBU = 34816;   // QB AI, 16 x 16, K-major (AB is dead by then) 1024
constexpr int G_RAW = 36864;   // q, w, k, a, b, v staging                   6 * 2048
constexpr int G_Y = 49152;            // the chunk's output as [time][value], bf16, 128-byte swizzle             2048
constexpr int G_GRAW = G_Y + 2048;    // attn_ln only: the gate tile                                            2048
constexpr int G_BYTES_PLAIN = G_GRAW;  // 50 KB
constexpr int G_Z0 = G_QB, G_Z1 = G_Y;  // affine maps only (which have neither): zeros                          2 * 256
static_assert(G_Z0 < G_DF && G_DF + 2048 <= G_Z1, "descriptors have positive strides");
constexpr int G_BYTES_LN = G_GRAW + RAW_TILE;  // 52 KB
static_assert(G_RAW % 1024 == 0 && G_RAW + 6 * RAW_TILE <= G_Y && G_Y % 1024 == 0 && G_BYTES_PLAIN % 1024 == 0 && G_BYTES_LN % 1024 == 0, "tile alignment");
// attn_ln epilogue scratch inside the kwf / bwf tiles, which are dead once the chain step has completed
constexpr int LN_YS = 68;                  // row stride (floats) of the fp32 [time][value] staging of Y
constexpr int LN_PART = L * LN_YS * 4;     // byte offset of the per-warp partial sums [4][16][2] behind it

// tensor-memory columns (32-bit each, 128 lanes; the M = 64 products use lanes 0-15 of each 32-lane quarter)
constexpr int C_S = 0;       // four 64-column state buffers: chunk c reads c % 4 and writes (c + 1) % 4
constexpr int C_INIT = 256;  // start state of the next segment (written by the group that prepares its first chunk)
constexpr int C_XY = 320;    // + 32 * group: X (16) | Y (16) of the group's chunk; before that its score products,
                             // [AK|AB] in lanes 0-15, [QK|QB] in lanes 32-47 (columns permuted, see G_KB)
constexpr int C_V = 448;     // + 16 * group: V^T [value][time] of the group's chunk

// Any wait of this kernel may stand still while one of its groups waits for the state of a cut chain: the chain warp (full), the
// score, inverse and fold warps (score, mats, inv), and the other groups (done).
constexpr long long WAIT_LIMIT = ACROSS_HANDOFF_LIMIT;

// The decay of the state, S' = S diag(P_L), is a product of TF32 operands: the tensor core reads S cut off after 10 mantissa bits, and
// P_L is rounded to as many.  Where a state lasts for many chunks, both errors must not have a sign of their own, or the state
// shrinks, or decays at another rate than asked for:
//  * S_CUT makes up for the mean loss of the cut, half a unit of 2^-10, by E[m] / E[m^2] = 2 / 3 for mantissas m in [1, 2) that are spread
//    evenly over their logarithm;
//  * P_L is rounded up or down at random, with bits of the chunk's operands, so that a constant decay is right on average (the
//    result still depends on the chunk's inputs alone).
// Relative L2 errors of y and sT against 64 bits, T = 8192 (rounding y costs 1.7e-3; before: cut and rounded to nearest):
//   w ~ N(-7, 0.25^2)                    2.9e-3, 2.3e-3 -> 1.9e-3, 0.9e-3      b a tenth as large: 8.9e-3, 9.1e-3 -> 2.2e-3, 1.4e-3
//   w constant in time, N(-9, 0.3^2), b a tenth as large: 1.8e-2, 2.0e-2 -> 2.6e-3, 2.0e-3
// A second product with what the first one lacks of P_L is only as good as that (2.4e-3, 1.6e-3), and its time is 3 % of a
// forward without checkpoints.
constexpr float S_CUT = 3.3e-4f;

// One chunk of the CTA's work list, as its preparation group (and the chain thread) need it.
struct ChunkDesc {
    long long off;   // element offset of (batch, time 0, head) in the inputs
    int bh, c;       // chain and chunk within it
    int c_end;       // end of the segment (the chunks of this chain that follow one another in the list)
    int flags;
    int bi, hi;      // batch entry, head
    int prev_first;  // SEG_FIRST: list position of the previous segment's first chunk if that lies less than G back, else -1
};
enum : int { SEG_FIRST = 1, SEG_LAST = 2 };  // first / last chunk of a segment

struct Ctrl {
    uint64_t full[4], done[4], score[4], raw[4], gate[4], mats[4], inv[4], rec[4], hop;
    uint32_t tmem_base;
    volatile int abort;
    ChunkDesc desc[4][4];      // [group][own-chunk number mod 4]: where the chunk lies (written one iteration ahead by the group)
    float bdot[4][2][4][L];    // attn_ln: per-warp partial bonus dots [group][iteration parity][warp][time]
    // abort path only, a set per warp: completion of its products, and what its waits take in place of the abort flag
    uint64_t drain[24];
    volatile int never_set[24];
};

// Bounded wait for the phase with the given parity.  Returns at once when the CTA has aborted.
// SLEEP: the thread is suspended by the hardware (try_wait with a time hint) instead of polling, so
// that the many warps that wait for the chain do not take issue slots from the warps that work; the
// chain's own short waits poll.
template <bool SLEEP>
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, Ctrl* ctrl, int* status, long long limit = WAIT_LIMIT) {
    mbar_wait_bounded<SLEEP>(bar, parity, &ctrl->abort, status, limit);
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {  // has the phase completed? (waits for the hardware's time limit)
    uint32_t ok;
    asm volatile("{\n.reg .pred P;\nmbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\nselp.u32 %0, 1, 0, P;\n}\n"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok;
}
// Abort path, by the thread of each warp that issues: waits, bounded and regardless of the CTA's abort flag, for the products and the
// load that this warp may have in flight, so that neither tensor memory nor shared memory is released under them.
__device__ __forceinline__ void abort_drain(Ctrl* ctrl, int warp, uint64_t* load, int* status) {
    volatile int* never_set = &ctrl->never_set[warp];
    *never_set = 0;
    mbar_init(&ctrl->drain[warp], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
    tc_commit(&ctrl->drain[warp]);
    const uint32_t since = clock();  // the kernel's own limit: products may stand behind a warp that still waits for a hand-off
    while (!mbar_test(&ctrl->drain[warp], 0) && !*never_set)
        if ((uint32_t)clock() - since > (uint32_t)WAIT_LIMIT) give_up(never_set, status);
    if (load) mbar_landed_uncounted(load, never_set, status);
}
// named barrier of one preparation group (the id in a register: a switch over immediate ids costs instruction-cache space)
__device__ __forceinline__ void group_bar(int grp) { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); }

// shared-memory matrix descriptor (sm_100 version field set); byte offsets are added to the low word
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t saddr, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t saddr) {  // 128-byte swizzle with 32-byte base
    return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)(2048 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46) | (1ull << 61);
}
// instruction descriptor: fp32 accumulate, TF32 operands
__host__ __device__ constexpr uint32_t idesc(int n, bool b_mn, int m = 64) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(d), "r"(a), "l"(b), "r"(id), "r"(acc) : "memory");
}
// 16 consecutive columns of this thread's lane
__device__ __forceinline__ void tmem_ld16(uint32_t ta, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]),"=r"(v[1]),"=r"(v[2]),"=r"(v[3]),"=r"(v[4]),"=r"(v[5]),"=r"(v[6]),"=r"(v[7]),"=r"(v[8]),"=r"(v[9]),"=r"(v[10]),"=r"(v[11]),"=r"(v[12]),"=r"(v[13]),"=r"(v[14]),"=r"(v[15]) : "r"(ta));
}
// the 16 lanes of an M = 64 product's quarter x 16 columns in the mma.sync accumulator layout: registers 4j..4j+3 = rows
// lane/4, lane/4 + 8 x columns 8j + 2(lane%4), +1
__device__ __forceinline__ void tmem_ld_frag(uint32_t ta, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(v[0]),"=r"(v[1]),"=r"(v[2]),"=r"(v[3]),"=r"(v[4]),"=r"(v[5]),"=r"(v[6]),"=r"(v[7]) : "r"(ta));
}
__device__ __forceinline__ void tmem_ld_frag4(uint32_t ta, uint32_t* v) {  // 32 columns
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]),"=r"(v[1]),"=r"(v[2]),"=r"(v[3]),"=r"(v[4]),"=r"(v[5]),"=r"(v[6]),"=r"(v[7]),"=r"(v[8]),"=r"(v[9]),"=r"(v[10]),"=r"(v[11]),"=r"(v[12]),"=r"(v[13]),"=r"(v[14]),"=r"(v[15]) : "r"(ta));
}
__device__ __forceinline__ void tmem_st_frag(uint32_t ta, const uint32_t* v) {  // the layout of tmem_ld_frag
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
        :: "r"(v[0]),"r"(v[1]),"r"(v[2]),"r"(v[3]),"r"(v[4]),"r"(v[5]),"r"(v[6]),"r"(v[7]), "r"(ta) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t ta, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        :: "r"(v[0]),"r"(v[1]),"r"(v[2]),"r"(v[3]),"r"(v[4]),"r"(v[5]),"r"(v[6]),"r"(v[7]),"r"(v[8]),"r"(v[9]),"r"(v[10]),"r"(v[11]),"r"(v[12]),"r"(v[13]),"r"(v[14]),"r"(v[15]), "r"(ta) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// (The conversion instruction cvt.rna.tf32 is one instead of two, but slow: the operand tiles took 1750 cycles with it, 750
// without.)
__device__ __forceinline__ float rnd(float x) { return __uint_as_float(tf32_rna(x)); }

__device__ __forceinline__ int kb_row(int s) { return (s & 8) | ((s & 3) << 1) | ((s >> 2) & 1); }
// byte offset of the 16-byte chunk holding (row, k..k+3) in a K-major tile; sbo = bytes per 8-row group
__device__ __forceinline__ int kchunk(int row, int kc, int sbo) { return (row >> 3) * sbo + kc * 128 + (row & 7) * 16; }

constexpr int ABS = 20;  // row pitch (floats) of the transposed AB: rows of 16-byte pieces and single columns are both conflict-free
// AI = (I - AB)^-1 (AB strictly lower triangular) into the K-major tile of AI^T, one warp.  In 8x8 blocks, AI = [X11, 0; X21, X22] with
// X21 = X22 A21 X11: the two diagonal blocks by right-looking substitution side by side (7 dependent steps instead of 15, a lane per
// column), then the two products, all 32 lanes.  ABt[s][t] = AB[t][s]; its blocks are overwritten once they have been used.
template <int S_> __device__ __forceinline__ void tri_fetch_tc(F2 (&dst)[4], const float* At) {  // row S_ of the block, entries > S_
#pragma unroll
    for (int v = (S_ + 1) / 4; v < 2; ++v) {
        const float4 x = *reinterpret_cast<const float4*>(At + S_ * ABS + 4 * v);
        dst[2 * v] = f2(x.x, x.y); dst[2 * v + 1] = f2(x.z, x.w);
    }
}
template <int S_> __device__ __forceinline__ void tri_step_tc(F2 (&r)[4], const F2 (&c)[4], F2 (&cn)[4], const float* At) {
    if (S_ + 1 < 7) tri_fetch_tc<(S_ + 1 < 7 ? S_ + 1 : 0)>(cn, At);
    const float ms = S_ & 1 ? r[S_ / 2].y : r[S_ / 2].x;
    if (!(S_ & 1)) r[S_ / 2].y = fmaf(c[S_ / 2].y, ms, r[S_ / 2].y);
#pragma unroll
    for (int h = S_ / 2 + 1; h < 4; ++h) r[h] = fma2(c[h], f2(ms, ms), r[h]);
}
__device__ __forceinline__ void tri_inverse_tc(float* ABt, unsigned char* AIt, int lane) {
    const int c = lane & 7, blk = (lane >> 3) & 1, p = lane >> 3;  // (lanes 16..31 repeat 0..15 up to the products)
    {
        const float* At = ABt + 8 * blk * (ABS + 1);
        F2 r[4], ca[4], cb[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) r[h] = f2(2 * h == c ? 1.f : 0.f, 2 * h + 1 == c ? 1.f : 0.f);
        tri_fetch_tc<0>(ca, At);
        tri_step_tc<0>(r, ca, cb, At);  tri_step_tc<1>(r, cb, ca, At);
        tri_step_tc<2>(r, ca, cb, At);  tri_step_tc<3>(r, cb, ca, At);
        tri_step_tc<4>(r, ca, cb, At);  tri_step_tc<5>(r, cb, ca, At);
        tri_step_tc<6>(r, ca, cb, At);
        __syncwarp();
        if (lane < 16) {
            // X11[.][c] to row 8 + c (zeros and unused until now), X22[.][c] to row c (A11's place)
            float* x = ABt + (8 * (1 - blk) + c) * ABS;
            *reinterpret_cast<float4*>(x) = make_float4(r[0].x, r[0].y, r[1].x, r[1].y);
            *reinterpret_cast<float4*>(x + 4) = make_float4(r[2].x, r[2].y, r[3].x, r[3].y);
#pragma unroll
            for (int q = 0; q < 2; ++q)
                *reinterpret_cast<float4*>(AIt + blk * 512 + (2 * blk + q) * 128 + c * 16) =
                    make_float4(rnd(r[2 * q].x), rnd(r[2 * q].y), rnd(r[2 * q + 1].x), rnd(r[2 * q + 1].y));
        } else {  // AI^T below its diagonal blocks
            *reinterpret_cast<float4*>(AIt + 512 + blk * 128 + c * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
    }
    // column c, rows 2 p, 2 p + 1 of T = A21 X11 and of X21 = X22 T
    auto col_product = [&](const float* mt, const float* col) {
        F2 acc[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const float4 x = *reinterpret_cast<const float4*>(col + 4 * v);
            const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 m = *reinterpret_cast<const float2*>(mt + (4 * v + i) * ABS + 2 * p);
                acc[i & 1] = fma2(f2(m.x, m.y), f2(xs[i], xs[i]), acc[i & 1]);
            }
        }
        return add2(acc[0], acc[1]);
    };
    float* t = ABt + (8 + c) * ABS + 8;
    const F2 tc = col_product(ABt + 8, ABt + (8 + c) * ABS);
    *reinterpret_cast<float2*>(t + 2 * p) = make_float2(tc.x, tc.y);  // (A22's place)
    __syncwarp();
    const F2 x = col_product(ABt, t);
    *reinterpret_cast<float2*>(AIt + (2 + (p >> 1)) * 128 + c * 16 + (p & 1) * 8) = make_float2(rnd(x.x), rnd(x.y));
}

// 16 bytes of an operand tile; R: round to TF32 (nearest) first, otherwise the tensor core
// truncates the low 13 mantissa bits when it reads the operand
template <bool R> __device__ __forceinline__ float4 quad4(const F2 (&f)[2]) {
    return R ? make_float4(rnd(f[0].x), rnd(f[0].y), rnd(f[1].x), rnd(f[1].y)) : make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
}
template <bool R> __device__ __forceinline__ F2 rnd2(F2 a) { return R ? f2(rnd(a.x), rnd(a.y)) : a; }
// four 8x4 blocks of 32-bit elements, 16 bytes of each of their rows at the address of lane 8 * block + row: lane 4 r + c has element (r, c)
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t saddr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}
__device__ __forceinline__ void stmatrix4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// A 16x16 matrix into a K-major operand tile, rounded to TF32: x[4 j + 2 h + e] is row lane / 4 + 8 h, column 8 j + 4 e + lane % 4.
// Entries with column > row + keep are written as zero.
__device__ __forceinline__ void store_frag16(uint32_t tile, const uint32_t* x, int lane, int keep) {
    const uint32_t at = tile + ((lane >> 3) & 1) * 128 + (lane >> 4) * 512 + (lane & 7) * 16;  // blocks (h, e) = (0, 0), (0, 1), (1, 0), (1, 1)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = (lane >> 2) + 8 * (i >> 1), col = 8 * j + 4 * (i & 1) + (lane & 3);
            v[i] = col <= row + keep ? tf32_rna(__uint_as_float(x[4 * j + i])) : 0u;
        }
        stmatrix4(at + j * 256, v[0], v[1], v[2], v[3]);
    }
}
__device__ __forceinline__ uint32_t pack_bf16x2_rn(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// AFF: the segments of a sequence cut in time as affine maps, S -> S M + R (wkv7_time_split.cu).  The state has 128 rows, R in lanes 0-63 and
// M in lanes 64-127 of tensor memory (M = 128 products; V^T has zeros there): one walk over the chunks instead of two, and without the
// output's products, tiles and stores.  R starts from zero (a sequence's first segment: from s0), M from the identity; they leave
// through sT and sM.
// TAIL: the sequence length is not a multiple of 16 (a build of its own, so that whole-chunk sequences carry none of
// the row tests in their register budget).
struct alignas(64) FwdMaps { CUtensorMap ck, y, in[6], g; };  // checkpoint states; output; q, w, k, a, b, v; gate

template <int G, bool RND, bool LN, bool TAIL, bool AFF>
__global__ void __launch_bounds__(128 * (G + 2), 1) wkv7_fwd_tc_kernel(FwdParams p, WorkSplit ws, const __grid_constant__ FwdMaps maps) {
    using IoT = __nv_bfloat16;
    constexpr int G_BYTES = LN ? G_BYTES_LN : G_BYTES_PLAIN;
    constexpr int NCOLS = 512, M = AFF ? 128 : 64, NX = AFF ? 16 : 32;  // rows of the state; columns X | Yp or X alone
    static_assert(!(AFF && LN), "the maps have no output");
    static_assert(C_XY + 32 * G <= C_V && C_V + 16 * G <= NCOLS, "tensor memory columns");
    // Register reallocation (G == 4 only).  setmaxnreg.inc blocks, without a bound, until the CTA's
    // register pool can satisfy it, and the pool is what the CTA was launched with: 768 threads x 80
    // registers (65536 / 768 rounded down to a multiple of 8; build.py checks that ptxas reports 80).
    // The raised and lowered counts must therefore fit into that pool exactly or with room to spare.
    constexpr int LAUNCH_REGS = 80, PREP_REGS = 96, SERVICE_REGS = 48;
    static_assert(G != 4 || 128 * G * PREP_REGS + 256 * SERVICE_REGS <= 128 * (G + 2) * LAUNCH_REGS, "setmaxnreg would never be satisfied");
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* sm = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(sm + G * G_BYTES);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // provably warp-uniform
    const int nchunks = ws.per_chain;  // the last chunk may be partial: its missing rows read as zeros
    const WorkRange work(ws, blockIdx.x);
    const int tail = TAIL ? (int)(p.T - (long long)(nchunks - 1) * L) : L;  // time steps of the last chunk (1..16)

    if (tid == 0) {
        for (int g = 0; g < G; ++g) {
            mbar_init(&ctrl->full[g], AFF ? 2 : 3);
            mbar_init(&ctrl->mats[g], AFF ? 1 : 2);
            mbar_init(&ctrl->inv[g], 1);
            mbar_init(&ctrl->rec[g], 1);
            mbar_init(&ctrl->done[g], 1);
            mbar_init(&ctrl->score[g], 1);
            mbar_init(&ctrl->raw[g], 1);
            mbar_init(&ctrl->gate[g], 1);
        }
        mbar_init(&ctrl->hop, 1);
        ctrl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // descriptors of every group's first two chunks
    auto describe = [&](int g, int k) {
        const int v = g + k * G;
        if (v >= work.n) return;
        ChunkDesc d;
        work.locate(v, nchunks, d.bh, d.c);
        d.bi = (int)((unsigned)d.bh / (unsigned)p.H);
        d.hi = d.bh - d.bi * (int)p.H;
        d.off = d.bi * p.st.b + d.hi * p.st.h;
        d.c_end = v < work.h ? work.h : nchunks;  // the start piece is chunks 0 .. h - 1 of its chain
        d.flags = (work.starts_segment(v, d.c) ? SEG_FIRST : 0) | (d.c + 1 == d.c_end ? SEG_LAST : 0);
        d.prev_first = -1;
        if (d.flags & SEG_FIRST)
            for (int u = v - 1; u >= 0 && u > v - G; --u) {
                int ub, uc;
                work.locate(u, nchunks, ub, uc);
                if (work.starts_segment(u, uc)) { d.prev_first = u; break; }
            }
        ctrl->desc[g][k & 3] = d;
    };
    if (tid < 2 * G) describe(tid >> 1, tid & 1);
    // the off-diagonal zeros of the decay blocks are written once
    for (int i = tid; i < G * (2048 / 16); i += blockDim.x)
        *reinterpret_cast<uint4*>(sm + (i / 128) * G_BYTES + G_DF + (i % 128) * 16) = make_uint4(0, 0, 0, 0);
    if (AFF)  // zeros before and after them: products of 16 columns (the least with 128 rows) take a block and one of these
        for (int i = tid; i < G * 32; i += blockDim.x)
            *reinterpret_cast<uint4*>(sm + (i / 32) * G_BYTES + (i & 16 ? G_Z1 : G_Z0) + (i & 15) * 16) = make_uint4(0, 0, 0, 0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctrl->tmem_base)), "r"(NCOLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctrl->tmem_base;

    // Start state of a segment -> tensor memory and its checkpoint: warp wq of the group owns lanes 32 wq .. 32 wq + 31, of
    // which lanes 0-15 hold value rows 16 wq .. 16 wq + 15.  A chain's first chunk starts from s0 (or zeros); a chain that
    // the list cuts starts from the state that the CTA before this one left in sT (see WorkSplit).
    auto load_state = [&](const ChunkDesc& d, int wq) {
        const int sbh = d.bh, sc = d.c;
        const uint32_t ta = tmem + C_INIT;
        if (d.prev_first >= 0) mbar_wait<true>(&ctrl->done[d.prev_first % G], (d.prev_first / G) & 1, ctrl, p.status);  // its start state has been used
        const int row = AFF ? 32 * wq + lane : 16 * wq + (lane & 15), i = row & 63;
        if (sc > 0) wait_handoff(ws.flags + blockIdx.x - 1, &ctrl->abort, p.status);
        const float* src = sc > 0 ? p.sT : p.s0;
        if (AFF) {
            const int entry = (int)((unsigned)d.bi / (unsigned)p.nseg);
            if (sc > 0) src = (row < 64 ? p.sT : p.sM) + (long long)sbh * N * N;
            else src = row < 64 && p.s0 && d.bi == entry * p.nseg ? p.s0 + (long long)(entry * (int)p.H + d.hi) * N * N : nullptr;
            if (src) src += i * N;
        } else if (src) {
            src += (long long)sbh * N * N + i * N;
        }
        float* ck = (p.ckpt && lane < 16) ? p.ckpt + ((long long)sbh * nchunks + sc) * CK_FLOATS + i * N : nullptr;
#pragma unroll 1
        for (int cb = 0; cb < N; cb += 16) {
            uint32_t v[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float4 x = src ? __ldcg(reinterpret_cast<const float4*>(src + cb + 4 * q)) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (AFF && sc == 0 && row >= 64) {  // identity
                    const int j = i - cb - 4 * q;
                    x = make_float4(j == 0, j == 1, j == 2, j == 3);
                }
                x.x *= STATE_SCALE; x.y *= STATE_SCALE; x.z *= STATE_SCALE; x.w *= STATE_SCALE;  // the state is carried as S~ = 2^-64 S (see ANCHOR_LN)
                v[4 * q] = __float_as_uint(x.x); v[4 * q + 1] = __float_as_uint(x.y); v[4 * q + 2] = __float_as_uint(x.z); v[4 * q + 3] = __float_as_uint(x.w);
                if (ck) *reinterpret_cast<float4*>(ck + cb + 4 * q) = x;
            }
            tmem_st16(ta + ((uint32_t)(32 * wq) << 16) + cb, v);
        }
        tmem_st_wait();
    };

    if (warp >= 4 * G) {
        // ------------------------------ service warps -----------------------------------------
        if (G == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SERVICE_REGS));
        const int q = warp & 3;  // (of the score and fold warps:) tensor-memory lanes 0-15 or 32-47
        const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16);
        if (warp == 4 * G + 3) {
          if (elect_one()) {
            const uint32_t sb = smem_u32(sm);
            int seg_first = 0;  // list position at which the next segment begins
            // The V parts of chunk c's products, X | Yp and S', need no state: they are issued while the chunk before it drains.
            // The group has read the results of its previous chunk by the time it is full, so the buffers about to be written
            // (X | Y of this group, and the state buffer, last read for chunk c - 4) are free.
            auto start_chunk = [&](int c) {
                const int g = c % G;
                const uint32_t gb = sb + g * G_BYTES, Sn = tmem + C_S + 64 * ((c + 1) & 3), XY = tmem + C_XY + 32 * g;
                const uint64_t dSC = desc_kmajor(gb + G_SC, 512), dKWF = desc_mnmajor(gb + G_KWF);
                const uint32_t V = tmem + C_V + 16 * g;
                mbar_wait<false>(&ctrl->full[g], (c / G) & 1, ctrl, p.status);
                tc_fence_after();
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) mma_ts(XY, V + 8 * ks, dSC + (uint64_t)(ks * 16), idesc(NX, false, M), ks > 0);
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) mma_ts(Sn, V + 8 * ks, dKWF + (uint64_t)(ks * 64), idesc(64, true, M), ks > 0);
            };
            start_chunk(0);
            for (int c = 0; c < work.n; ++c) {  // position in the CTA's list
                const int g = c % G, k = c / G;
                const uint32_t gb = sb + g * G_BYTES;
                const uint64_t dWAQ = desc_kmajor(gb + G_WAQ, 2048), dQBU = desc_kmajor(gb + G_QBU, 512), dDF = desc_kmajor(gb + G_DF, 256);
                const uint64_t dBWU = desc_mnmajor(gb + G_BWF);
                const uint32_t Sn = tmem + C_S + 64 * ((c + 1) & 3), XY = tmem + C_XY + 32 * g;
                uint32_t Sa = tmem + C_S + 64 * (c & 3);
                if (c == seg_first) {
                    Sa = tmem + C_INIT;
                    seg_first = c < work.h ? work.h : c < work.n - work.t ? min(c + nchunks, work.n - work.t) : work.n;
                }
                // hop 1
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) mma_ts(XY, Sa + 8 * ks, dWAQ + (uint64_t)(ks * 16), idesc(NX, false, M), 1);
                tc_commit(&ctrl->hop);
                // the decay of the old state goes into the other buffer while hop 1 drains
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    if (!AFF) {
                        mma_ts(Sn + 8 * s, Sa + 8 * s, dDF + (uint64_t)(s * 16), idesc(8, false), 1);
                    } else {  // rows 0-7 and 8-15 of the operand: the block and zeros, or zeros and the block
                        const uint32_t blk = gb + G_DF + 256 * s;
                        mma_ts(Sn + 16 * (s >> 1), Sa + 8 * s, s & 1 ? desc_kmajor(gb + G_Z0, blk - (gb + G_Z0)) : desc_kmajor(blk, gb + G_Z1 - blk), idesc(16, false, M), 1);
                    }
                }
                mbar_wait<false>(&ctrl->hop, c & 1, ctrl, p.status);
                tc_fence_after();
                // hop 2: the X part of the state update and of Y
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) mma_ts(Sn, XY + 8 * ks, dBWU + (uint64_t)(ks * 64), idesc(64, true, M), 1);
#pragma unroll
                for (int ks = 0; ks < (AFF ? 0 : 2); ++ks) mma_ts(XY + 16, XY + 8 * ks, dQBU + (uint64_t)(ks * 16), idesc(16, false, M), 1);
                tc_commit(&ctrl->done[g]);
                if (c + 1 < work.n) start_chunk(c + 1);
                mbar_wait<false>(&ctrl->done[g], k & 1, ctrl, p.status);  // S' is the next chunk's A operand
                tc_fence_after();
            }
          }
        } else if (AFF && (warp == 4 * G + 1 || warp == 4 * G + 7)) {
            // (QK, QB and QB AI are for the output)
        } else if (warp == 4 * G || warp == 4 * G + 1) {
            // ---- score warps: warp 4G reads [AK|AB], warp 4G + 1 reads [QK|QB]
            for (int r = 0; r < work.n; ++r) {
                const int gr = r % G;
                unsigned char* gs = sm + gr * G_BYTES;
                mbar_wait<true>(&ctrl->score[gr], (r / G) & 1, ctrl, p.status);
                tc_fence_after();
                uint32_t x[16];
                tmem_ld_frag4(tq + C_XY + 32 * gr, x);
                tmem_ld_wait();
                tc_fence_before();
                // the previous chunk's matrices have left for its checkpoint record
                if (p.ckpt && r >= G) mbar_wait<true>(&ctrl->rec[gr], (r / G - 1) & 1, ctrl, p.status);
                if (q == 0) {  // AB, strictly lower, kept transposed for the inverse
                    float* ABt = reinterpret_cast<float*>(gs + G_ABT);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = (lane >> 2) + 8 * ((i >> 1) & 1), col = 8 * (i >> 2) + 4 * (i & 1) + (lane & 3);
                        ABt[col * ABS + row] = col < row ? __uint_as_float(x[8 + i]) : 0.f;
                    }
                } else {
                    store_frag16(smem_u32(gs + G_QB), x + 8, lane, 0);
                }
                store_frag16(smem_u32(gs + G_SC + 1024 * q), x, lane, q ? 0 : -1);          // AK (strictly lower) or QK (lower triangular)
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->mats[gr]);
            }
        } else if (q == 2) {
            // ---- inverse warps (even and odd groups: each barrier has one warp that sees all its phases)
            for (int c = 0; c < work.n; ++c) {
                const int g = c % G, k = c / G;
                if ((g ^ (warp >> 2)) & 1) continue;
                unsigned char* gs = sm + g * G_BYTES;
                mbar_wait<true>(&ctrl->mats[g], k & 1, ctrl, p.status);
                tri_inverse_tc(reinterpret_cast<float*>(gs + G_ABT), gs + G_AI, lane);
                fence_async_smem();
                __syncwarp();
                if (elect_one()) {
                    mbar_arrive(&ctrl->inv[g]);
                    // The chunk's four 16x16 matrices go into its checkpoint record: the three tiles [AK;QK], AI^T, QB are
                    // contiguous in shared memory and are stored as they are, by one bulk copy.
                    if (p.ckpt) {
                        const ChunkDesc& d = ctrl->desc[g][k & 3];
                        float* ckm = p.ckpt + ((long long)d.bh * nchunks + d.c) * CK_FLOATS + CK_MATS;
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                     ::"l"(__cvta_generic_to_global(ckm)), "r"(smem_u32(gs + G_SC)), "n"(4 * L * L * 4) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        mbar_arrive(&ctrl->rec[g]);
                    }
                }
                __syncwarp();
            }
        } else {
            // ---- fold warps: U = X AI^T, so U bwf = X (AI^T bwf) and U QB^T = X (QB AI)^T: one dependent tensor-core round trip per chunk
            // less for the chain.  Warps 4G + 4, 4G + 5 form 32 key columns of AI^T bwf each, in the place of bwf, warp 4G + 7 QB AI.
            // (mma.sync: as tcgen05 products they read 104 wavefronts of operands instead of 64, 64 rows of A for 32 or 16 used ones, and
            // the results came back through tensor memory.)
            const int g8 = lane >> 2, t4 = lane & 3;
            const uint32_t at = (lane >> 4) * 512 + ((lane >> 3) & 1) * 128 + (lane & 7) * 16;  // A operands: 8x4 blocks (rows 0-7 | 8-15) x (4 columns | the next 4)
            for (int c = 0; c < work.n; ++c) {
                const int g = c % G;
                unsigned char* gs = sm + g * G_BYTES;
                mbar_wait<true>(&ctrl->inv[g], (c / G) & 1, ctrl, p.status);
                uint32_t ai[2][4];
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) ldmatrix4(ai[kb], smem_u32(gs + G_AI) + at + kb * 256);
                if (q == 3) {
                    float acc[2][4] = {};
#pragma unroll
                    for (int kb = 0; kb < 2; ++kb) {
                        uint32_t a[4];
                        ldmatrix4(a, smem_u32(gs + G_QB) + at + kb * 256);
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt) mma_tf32_raw(acc[nt], a[0], a[2], a[1], a[3], ai[kb][2 * nt], ai[kb][2 * nt + 1]);  // B = AI^T by rows
                    }
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            *reinterpret_cast<float2*>(gs + G_QBU + kchunk(g8 + 8 * h, 2 * nt + (t4 >> 1), 512) + (t4 & 1) * 8) = make_float2(rnd(acc[nt][2 * h]), rnd(acc[nt][2 * h + 1]));
                } else {
                    unsigned char* bw = gs + G_BWF + q * 2048;
                    float acc[4][4] = {};
#pragma unroll
                    for (int kb = 0; kb < 2; ++kb)
#pragma unroll
                        for (int nt = 0; nt < 4; ++nt) {  // contraction slots t4, t4 + 4 are time steps t4, t4 + 4 of the eight
                            const unsigned char* b = bw + (8 * kb + t4) * 128 + ((nt ^ t4) << 5) + g8 * 4;
                            mma_tf32_raw(acc[nt], ai[kb][0], ai[kb][2], ai[kb][1], ai[kb][3], *reinterpret_cast<const uint32_t*>(b), *reinterpret_cast<const uint32_t*>(b + 512));
                        }
                    __syncwarp();  // bwf has been read
#pragma unroll
                    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            *reinterpret_cast<float2*>(bw + (g8 + 8 * h) * 128 + ((nt ^ (g8 & 3)) << 5) + t4 * 8) = make_float2(rnd(acc[nt][2 * h]), rnd(acc[nt][2 * h + 1]));
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->full[g]);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------ preparation group ---------------------------------------
        if (G == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PREP_REGS));
        const int grp = warp >> 2, wg = warp & 3, gt = tid & 127;
        unsigned char* gs = sm + grp * G_BYTES;
        const uint32_t tlane = tmem + ((uint32_t)(32 * wg) << 16);
        // The raw tiles of own chunk number ko by bulk tensor loads (16 rows of 128 bytes, 16-byte units XOR-ed with the row;
        // rows beyond the end of the sequence arrive as zeros).  One thread of the group.
        auto load_tile = [&](const CUtensorMap& m, int at, const ChunkDesc& d, uint64_t* bar) {
            asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                         ::"r"(smem_u32(gs + at)), "l"(&m), "r"(smem_u32(bar)), "r"(0), "r"(d.hi), "r"(d.c * L), "r"(d.bi) : "memory");
        };
        auto expect_bytes = [&](uint64_t* bar, int bytes) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
        };
        auto load_raw = [&](int ko) {
            if (ctrl->abort) return;  // (the last one's wait may have given up)
            const ChunkDesc& d = ctrl->desc[grp][ko & 3];
            expect_bytes(&ctrl->raw[grp], (AFF ? 5 : 6) * RAW_TILE);
#pragma unroll
            for (int ten = AFF ? 1 : 0; ten < 6; ++ten) load_tile(maps.in[ten], G_RAW + ten * RAW_TILE, d, &ctrl->raw[grp]);
        };
        // The output tile of own chunk number kk, once all of the group's warps have written it.
        auto store_y = [&](int kk) {
            if (wg == 1 && elect_one()) {
                const ChunkDesc& d = ctrl->desc[grp][kk & 3];
                asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                             ::"l"(&maps.y), "r"(0), "r"(d.hi), "r"(d.c * L), "r"(d.bi), "r"(smem_u32(gs + G_Y)) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            __syncwarp();
        };
        // Results of own chunk number kk (list position vv): Y^T into the output tile (which leaves after the group's next barrier),
        // the chunk-end state to the checkpoint (or the final state).  All of it is read before the group announces its next chunk.
        auto read_results = [&](int kk) {
            mbar_wait<true>(&ctrl->done[grp], kk & 1, ctrl, p.status);
            if (LN) mbar_wait<true>(&ctrl->gate[grp], kk & 1, ctrl, p.status);
            tc_fence_after();
            const ChunkDesc& d = ctrl->desc[grp][kk & 3];
            const int vv = grp + kk * G, cc = d.c;
            const bool seg_last = d.flags & SEG_LAST;
            float* sdst = AFF ? (seg_last ? (wg < 2 ? p.sT : p.sM) + (long long)d.bh * N * N : nullptr)
                        : seg_last ? (p.sT ? p.sT + (long long)d.bh * N * N : nullptr)
                                   : (p.ckpt ? p.ckpt + ((long long)d.bh * nchunks + cc + 1) * CK_FLOATS : nullptr);
            if (AFF) {
            } else if (!LN) {
                // Y^T [value][time], read as accumulator fragments, goes as bf16 through a transposing matrix store into the
                // [time][value] tile (128-byte rows, 16-byte units XOR-ed with the row as the tensor map's swizzle wants), which
                // leaves by one bulk tensor store; the map clips rows beyond the end of the sequence.
                uint32_t yv[8];
                tmem_ld_frag(tlane + C_XY + 32 * grp + 16, yv);
                tmem_ld_wait();
                uint32_t h[4];  // 8x8 blocks: values 0-7 | 8-15 of time steps 0-7, then of time steps 8-15
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = pack_bf16x2_rn(__uint_as_float(yv[2 * j]), __uint_as_float(yv[2 * j + 1]));
                const int t = (lane & 7) + 8 * (lane >> 4), unit = 2 * wg + ((lane >> 3) & 1);  // row address of block lane / 8
                asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                             ::"r"(smem_u32(gs + G_Y + t * 128 + ((unit ^ (t & 7)) << 4))), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
            } else {
                // attn_ln epilogue (reference: wind_rwkv/rwkv7/attn_ln.cu:176-205): GroupNorm over the head's 64
                // value channels of each time step, + bonus dot * v, * gate.  Y^T goes to shared memory as
                // fp32 [time][value] (in the dead kwf / bwf tiles); then one thread = one time step x 8 value channels.
                float* ysf = reinterpret_cast<float*>(gs + G_KWF);
                float* part = reinterpret_cast<float*>(gs + G_KWF + LN_PART);
                {
                    uint32_t yv[8];
                    tmem_ld_frag(tlane + C_XY + 32 * grp + 16, yv);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        ysf[(8 * (i >> 2) + 2 * (lane & 3) + (i & 1)) * LN_YS + 16 * wg + (lane >> 2) + 8 * ((i >> 1) & 1)] = __uint_as_float(yv[i]);
                }
                group_bar(grp);
                const int t = lane & 15, i0 = 16 * wg + 8 * (lane >> 4);
                float yv8[8];
                {
                    const float4 a4 = *reinterpret_cast<const float4*>(ysf + t * LN_YS + i0), b4 = *reinterpret_cast<const float4*>(ysf + t * LN_YS + i0 + 4);
                    yv8[0] = a4.x; yv8[1] = a4.y; yv8[2] = a4.z; yv8[3] = a4.w; yv8[4] = b4.x; yv8[5] = b4.y; yv8[6] = b4.z; yv8[7] = b4.w;
                }
                // sums about a pivot (the row's first element) keep the one-pass variance well conditioned
                const float pivot = ysf[t * LN_YS];
                float s1 = 0.f, s2 = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) { const float dd = yv8[i] - pivot; s1 += dd; s2 = fmaf(dd, dd, s2); }
                s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
                s2 += __shfl_xor_sync(0xffffffffu, s2, 16);
                if (lane < 16) *reinterpret_cast<float2*>(part + (wg * L + t) * 2) = make_float2(s1, s2);
                group_bar(grp);
                {
                    float a1 = 0.f, a2 = 0.f, bd = 0.f;
#pragma unroll
                    for (int w2 = 0; w2 < 4; ++w2) {
                        const float2 pp = *reinterpret_cast<const float2*>(part + (w2 * L + t) * 2);
                        a1 += pp.x; a2 += pp.y;
                        bd += ctrl->bdot[grp][kk & 1][w2][t];
                    }
                    const float md = a1 * (1.f / N);
                    const float mu = pivot + md;
                    const float rstd = rsqrtf(fmaxf(a2 * (1.f / N) - md * md, 0.f) + p.eps);
                    float vval[8];  // v of this chunk was kept aside, the gate has its own double buffer
                    load8<IoT>(gs + G_V + t * 128 + (((i0 >> 3) ^ (t & 7)) << 4), vval);
                    float gv[8];
                    load8<IoT>(gs + G_GRAW + t * ROWB + (((i0 >> 3) ^ (t & 7)) << 4), gv);
                    float o8[8];
                    const float* lnp = p.params + d.hi * N + i0;  // GroupNorm weight, then bias: 32 bytes each per thread, in L1
                    const float4 w0 = __ldg(reinterpret_cast<const float4*>(lnp)), w1 = __ldg(reinterpret_cast<const float4*>(lnp) + 1);
                    const float4 b0 = __ldg(reinterpret_cast<const float4*>(lnp + p.H * N)), b1 = __ldg(reinterpret_cast<const float4*>(lnp + p.H * N) + 1);
                    const float lw8[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w}, lb8[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) o8[i] = ((yv8[i] - mu) * rstd * lw8[i] + lb8[i] + bd * vval[i]) * gv[i];
                    uint4 pk;
                    pk.x = pack_bf16x2_rn(o8[0], o8[1]); pk.y = pack_bf16x2_rn(o8[2], o8[3]);
                    pk.z = pack_bf16x2_rn(o8[4], o8[5]); pk.w = pack_bf16x2_rn(o8[6], o8[7]);
                    *reinterpret_cast<uint4*>(gs + G_Y + t * 128 + (((i0 >> 3) ^ (t & 7)) << 4)) = pk;
                }
            }
            if (LN) {  // (the staging tiles are about to be written again)
                fence_async_smem();
                group_bar(grp);
                store_y(kk);
            }
            if (sdst && !seg_last) {
                // checkpoint state: exact fp32 (the backward's tensor-core products read its upper 19 bits, its carried
                // decay term all of them), staged in the swizzled layout the tensor-map store expects: half h = columns 32h..32h+31,
                // row i at i*128 bytes, its 32-byte unit u at (u ^ (i & 3)).  A half-warp's 8-byte stores cover four rows x 32 bytes: with
                // 32-byte units they fill the 32 banks; with the 16-byte swizzle rows 2i and 2i + 1 met in the same ones (B64 T1024 H12:
                // 372 us with them, 359 us without).
                unsigned char* stage = gs + G_WAQ;
                const int i = 16 * wg + (lane >> 2);  // rows i, i + 8
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t x[16];
                    tmem_ld_frag4(tlane + C_S + 64 * ((vv + 1) & 3) + 32 * half, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            *reinterpret_cast<uint2*>(stage + half * 8192 + (i + 8 * h) * 128 + ((j ^ (i & 3)) << 5) + (lane & 3) * 8) =
                                make_uint2(x[4 * j + 2 * h], x[4 * j + 2 * h + 1]);
                }
                fence_async_smem();
                group_bar(grp);
                if (wg == 0 && elect_one()) {
                    const int rec_row = (int)(((long long)d.bh * nchunks + cc + 1) * (CK_FLOATS / N));  // a record is 80 rows of 64 floats
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                                 ::"l"(&maps.ck), "r"(0), "r"(rec_row), "r"(smem_u32(stage)) : "memory");
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                                 ::"l"(&maps.ck), "r"(32), "r"(rec_row), "r"(smem_u32(stage + 8192)) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                __syncwarp();
            } else if (sdst) {
                // final state: exact, straight from registers (32-byte stores: whole sectors of the lane's 256-byte row)
                float* d = sdst + (AFF ? 32 * (wg & 1) + lane : 16 * wg + (lane & 15)) * N;
#pragma unroll
                for (int qt = 0; qt < 4; ++qt) {
                    uint32_t sv[16];
                    tmem_ld16(tlane + C_S + 64 * ((vv + 1) & 3) + 16 * qt, sv);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) sv[e] = __float_as_uint(__uint_as_float(sv[e]) * STATE_UNSCALE);  // S = 2^64 S~
                    if (AFF || lane < 16) {
#pragma unroll
                        for (int q8 = 0; q8 < 2; ++q8)
                            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(d + 16 * qt + 8 * q8), "r"(sv[8 * q8]), "r"(sv[8 * q8 + 1]),
                                         "r"(sv[8 * q8 + 2]), "r"(sv[8 * q8 + 3]), "r"(sv[8 * q8 + 4]), "r"(sv[8 * q8 + 5]), "r"(sv[8 * q8 + 6]), "r"(sv[8 * q8 + 7]) : "memory");
                    }
                }
                if (cc + 1 < nchunks) {  // the rest of this chain is another CTA's: hand the state over
                    __threadfence();
                    group_bar(grp);
                    if (gt == 0) publish_handoff(ws.flags + blockIdx.x);
                }
            }
        };
        // Scan and operand tiles: a thread has two adjacent time steps x 4 adjacent key channels (quad), so that the running sum takes
        // three shuffle rounds of 4 channels instead of four of 8 (a shuffle is a pass through the shared-memory pipe that this kernel
        // is short of).  Slot 0 is the earlier or the later one (`late`) of the two steps, such that the eight lanes of a quarter-warp store to
        // eight rows, every residue of the row mod 8 once and, with the quad's parity, all eight 16-byte units of the MN-major rows: neither
        // the raw loads nor the tile stores have bank conflicts.  Lane bits 0, 1, 3: pair of time steps; bits 2, 4: quad.
        // (One step x 8 channels: 359 us at B64 T1024 H12, 1904 us at B8 T16384 H40 without checkpoints; this: 354 and 1886 us.)
        const int late = ((lane >> 1) ^ (lane >> 2) ^ (lane >> 3)) & 1;
        const int quad = 4 * wg + ((lane >> 2) & 1) + ((lane >> 3) & 2), row0 = 2 * ((lane & 3) + ((lane >> 1) & 4)) + late;  // slot 1: row0 ^ 1
        const int j0 = 4 * quad;
        const float late0 = late ? 0.f : -1.f, late1 = late ? -1.f : 0.f;
        if (wg == 2 && grp < work.n && elect_one()) load_raw(0);
        __syncwarp();
        if (AFF && wg >= 2) {
            const uint32_t zeros[16] = {};
            tmem_st16(tlane + C_V + 16 * grp, zeros);
            tmem_st_wait();
        }
        // Iteration k: read the results of own chunk k - 1, write the operand tiles of chunk k (whose scan is in registers),
        // start its score product; then scan chunk k + 1 while the score, inverse and chain warps finish chunk k.  (k = -1 only
        // scans, the last one only reads results: one copy of each piece of code.)
        F2 o[4][2][2], fwv[2];  // [slot][channel pair] of wq, wa, kwi, bwi; kwf, bwf are formed from kwi, bwi and fw when the tiles are written
        uint32_t v[4], v2[AFF ? 4 : 1];  // (AFF: values 32 wg + .. and 32 wg + 16 + .., warps 0 and 1)
                                // V^T: values 16 wg + lane / 4 (+ 8) x time steps 2 (lane % 4), + 1; then time steps 8 ..
        for (int k = -1, v0 = grp - G; ; v0 += G, ++k) {
            if (k >= 0) {
                // ---------------- results of the previous own chunk (its operand tiles are free afterwards) --
                if (k > 0) read_results(k - 1);
                if (v0 >= work.n) {
                    if (!LN && !AFF && k > 0) {
                        fence_async_smem();
                        group_bar(grp);
                        store_y(k - 1);
                    }
                    break;
                }
                // ---------------- operand tiles -----------------------------------------------------------
                {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int row = row0 ^ e, mo = (quad >> 3) * 2048 + row * 128 + ((((quad >> 1) & 3) ^ (row & 3)) << 5) + (quad & 1) * 16;
                        F2 kf[2], bf[2];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {  // k P_L / P_t first, then 2^-64
                            kf[i] = mul2(mul2(o[2][e][i], fwv[i]), f2(STATE_SCALE, STATE_SCALE));
                            bf[i] = mul2(mul2(o[3][e][i], fwv[i]), f2(STATE_SCALE, STATE_SCALE));
                        }
                        *reinterpret_cast<float4*>(gs + G_KWF + mo) = quad4<RND>(kf);
                        *reinterpret_cast<float4*>(gs + G_BWF + mo) = quad4<RND>(bf);
                    }
                    uint32_t vf[8];  // bf16 values are exact in TF32
#pragma unroll
                    for (int i = 0; i < 4; ++i) { vf[2 * i] = v[i] << 16; vf[2 * i + 1] = v[i] & 0xffff0000u; }
                    if (!AFF || wg < 2) tmem_st_frag(tlane + C_V + 16 * grp, vf);
                    if (AFF && wg < 2) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) { vf[2 * i] = v2[AFF ? i : 0] << 16; vf[2 * i + 1] = v2[AFF ? i : 0] & 0xffff0000u; }
                        tmem_st_frag(tlane + (16u << 16) + C_V + 16 * grp, vf);
                    }
                    if (LN) {  // the epilogue's v: as the raw tile had it
                        const int t = (lane & 7) + 8 * (lane >> 4), unit = 2 * wg + ((lane >> 3) & 1);
                        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                                     ::"r"(smem_u32(gs + G_V + t * 128 + ((unit ^ (t & 7)) << 4))), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
                    }
                    if (!(lane & 8)) {  // the decay blocks' entries, one per lane (see S_CUT): channel j0 + (lane & 3)
                        const F2 p2 = lane & 2 ? fwv[1] : fwv[0];
                        const float pl = (lane & 1 ? p2.y : p2.x) * (STATE_SCALE * (1.f + S_CUT));  // where P_L underflows, so does S~ P_L
                        const uint32_t dither = ((__float_as_uint(o[2][0][0].x) ^ __float_as_uint(o[3][0][0].x)) * 0x9e3779b1u) >> 19;
                        *reinterpret_cast<uint32_t*>(gs + G_DF + quad * 128 + ((quad & 1) * 4 + (lane & 3)) * 16 + (lane & 3) * 4) =
                            (__float_as_uint(pl) + dither) & 0xffffe000u;
                    }
                    if (k > 0 && p.ckpt) {  // the state's staging tiles are the next two operand tiles: wait until the bulk stores have read them
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        group_bar(grp);
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int at = kchunk(row0 ^ e, quad, 2048);
                        *reinterpret_cast<float4*>(gs + G_WAQ + at) = quad4<false>(o[1][e]);
                        if (!AFF) *reinterpret_cast<float4*>(gs + G_WAQ + 4096 + at) = quad4<false>(o[0][e]);
                        const int ak = kchunk(kb_row(row0 ^ e), quad, 2048);
                        *reinterpret_cast<float4*>(gs + G_KB + ak) = quad4<RND>(o[2][e]);
                        *reinterpret_cast<float4*>(gs + G_KB + 4096 + ak) = quad4<RND>(o[3][e]);
                    }
                }
                tmem_st_wait();  // V
                if (ctrl->desc[grp][k & 3].flags & SEG_FIRST) load_state(ctrl->desc[grp][k & 3], wg);
                fence_async_smem();
                tc_fence_before();
                group_bar(grp);
                tc_fence_after();
                if (LN && wg == 2 && elect_one() && !ctrl->abort) {
                    expect_bytes(&ctrl->gate[grp], RAW_TILE);
                    load_tile(maps.g, G_GRAW, ctrl->desc[grp][k & 3], &ctrl->gate[grp]);
                }
                __syncwarp();
                if (gt == 127 && v0 + 2 * G < work.n) {  // read after this group's next barrier
                    ChunkDesc d = ctrl->desc[grp][(k + 1) & 3];
                    d.c += G;
                    if (d.c < d.c_end) {
                        d.flags = d.c + 1 == d.c_end ? SEG_LAST : 0;
                        ctrl->desc[grp][(k + 2) & 3] = d;
                    } else {
                        describe(grp, k + 2);
                    }
                }
                __syncwarp();
                // ---------------- the four score matrices as one product ---------------------------------
                if (!LN && !AFF && k > 0) store_y(k - 1);
                if (wg == 0 && elect_one()) {
                    const uint64_t dA = desc_kmajor(smem_u32(gs + G_WAQ), 2048), dB = desc_kmajor(smem_u32(gs + G_KB), 2048);
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) mma_ss(tmem + C_XY + 32 * grp, dA + (uint64_t)(ks * 16), dB + (uint64_t)(ks * 16), idesc(32, false), ks > 0);
                    tc_commit(&ctrl->score[grp]);
                }
                __syncwarp();
            }
            // ---------------- decay scan of the next own chunk, into registers -----------------------
            // The three transcendentals per element go to the special-function unit: with the matrix products on tcgen05 the FMA
            // pipe and the issue slots are what this kernel runs out of, not MUFU throughput.
            if (v0 + G < work.n) {
                mbar_wait<true>(&ctrl->raw[grp], (k + 1) & 1, ctrl, p.status);
                F2 cum[2][2], q[2][2], kk[2][2], a[2][2], b[2][2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = row0 ^ e;
                    const unsigned char* raw = gs + G_RAW + row * ROWB + (((quad >> 1) ^ (row & 7)) << 4) + (quad & 1) * 8;
                    load4f2(raw + 1 * RAW_TILE, cum[e]);
                    if (!AFF) load4f2(raw + 0 * RAW_TILE, q[e]);
                    load4f2(raw + 2 * RAW_TILE, kk[e]);
                    load4f2(raw + 3 * RAW_TILE, a[e]);
                    load4f2(raw + 4 * RAW_TILE, b[e]);
                }
                {
                    const int t = 8 * (lane >> 4) + (lane & 7), unit = (AFF ? 4 * (wg & 1) : 2 * wg) + ((lane >> 3) & 1);
                    const uint32_t at = smem_u32(gs + G_RAW + 5 * RAW_TILE + t * ROWB);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at + ((unit ^ (t & 7)) << 4)) : "memory");
                    if (AFF)
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v2[0]), "=r"(v2[AFF ? 1 : 0]), "=r"(v2[AFF ? 2 : 0]), "=r"(v2[AFF ? 3 : 0]) : "r"(at + (((unit + 2) ^ (t & 7)) << 4)) : "memory");
                }
                if (LN) {  // bonus dot sum_j r_j k_j bonus_j of these time steps: 4 channels here, the rest by shuffle and in the epilogue
                    const float4 bo = __ldg(reinterpret_cast<const float4*>(p.params + (2 * p.H + ctrl->desc[grp][(k + 1) & 3].hi) * N + j0));
                    float dot[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const F2 acc = fma2(mul2(q[e][1], kk[e][1]), f2(bo.z, bo.w), mul2(mul2(q[e][0], kk[e][0]), f2(bo.x, bo.y)));
                        dot[e] = acc.x + acc.y;
                    }
                    float first = late ? dot[1] : dot[0], second = late ? dot[0] : dot[1];  // (lanes of the other quads have them in the other slot)
                    first += __shfl_xor_sync(0xffffffffu, first, 4);
                    second += __shfl_xor_sync(0xffffffffu, second, 4);
                    first += __shfl_xor_sync(0xffffffffu, first, 16);
                    second += __shfl_xor_sync(0xffffffffu, second, 16);
                    if (!(lane & 0x14)) *reinterpret_cast<float2*>(&ctrl->bdot[grp][(k + 1) & 1][wg][row0 & 14]) = make_float2(first, second);
                }
                // log2 of the per-step decay: -exp(w) * log2(e); running sum along the 16 time rows
                constexpr float LOG2E = 1.4426950408889634f, FLOOR = MIN_STEP_LOG_DECAY * LOG2E;  // the per-step floor in log2 units
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        F2 x = mul2(cum[e][i], f2(LOG2E, LOG2E));
                        x = mul2(f2(ex2_approx(x.x), ex2_approx(x.y)), f2(-LOG2E, -LOG2E));
                        cum[e][i] = f2(fmaxf(x.x, FLOOR), fmaxf(x.y, FLOOR));
                        // a row beyond the end of the sequence: no decay, the state passes through
                        if (TAIL && ctrl->desc[grp][(k + 1) & 3].c + 1 == nchunks && (row0 ^ e) >= tail) cum[e][i] = f2(0.f, 0.f);
                    }
                F2 sum[2];  // through the later step of the pair
#pragma unroll
                for (int i = 0; i < 2; ++i) sum[i] = add2(cum[0][i], cum[1][i]);
#pragma unroll
                for (int d = 1; d < 4; d <<= 1)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const F2 up = f2(__shfl_up_sync(0xffffffffu, sum[i].x, d, 4), __shfl_up_sync(0xffffffffu, sum[i].y, d, 4));
                        if ((lane & 3) >= d) sum[i] = add2(sum[i], up);
                    }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int src = (lane & 0x14) | 3;
                    const F2 low = f2(__shfl_sync(0xffffffffu, sum[i].x, src), __shfl_sync(0xffffffffu, sum[i].y, src));
                    if (lane & 8) sum[i] = add2(sum[i], low);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    // P~_t = 2^64 P_t and its reciprocal (see ANCHOR_LN): both finite for cum >= -179 (2^-115 ~ e^-80)
                    const F2 sa = add2(sum[i], f2(ANCHOR_LOG2, ANCHOR_LOG2));
                    // P~_L = 2^64 P_L (P_L itself may lie below fp32's normal range)
                    const int src = (lane & 0x14) | 11;
                    fwv[i] = f2(ex2_approx(fmaxf(__shfl_sync(0xffffffffu, sa.x, src), -115.f)), ex2_approx(fmaxf(__shfl_sync(0xffffffffu, sa.y, src), -115.f)));
                    const F2 c[2] = {fma2(cum[1][i], f2(late0, late0), sa), fma2(cum[0][i], f2(late1, late1), sa)};  // less the later step's, in the earlier one
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const F2 cp = fma2(cum[e][i], f2(-1.f, -1.f), c[e]);  // without this step's own decay
                        const float cx = fmaxf(c[e].x, -115.f), cy = fmaxf(c[e].y, -115.f);
                        const F2 incl = f2(ex2_approx(cx), ex2_approx(cy));
                        const F2 inv = f2(ex2_approx(-cx), ex2_approx(-cy));
                        const F2 non = f2(ex2_approx(fmaxf(cp.x, -115.f)), ex2_approx(fmaxf(cp.y, -115.f)));
                        if (!AFF) o[0][e][i] = rnd2<RND>(mul2(q[e][i], incl));   // wq (rounded here already: writing the tiles is on the way to the chain, this is not)
                        o[1][e][i] = rnd2<RND>(mul2(a[e][i], non));    // wa
                        o[2][e][i] = mul2(kk[e][i], inv);   // kwi
                        o[3][e][i] = mul2(b[e][i], inv);    // bwi
                    }
                }
            }
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // y's tile has been read (its issuer only)
            group_bar(grp);  // the raw tiles have been read
            if (wg == 2 && v0 + 2 * G < work.n && elect_one()) load_raw(k + 2);
            __syncwarp();
        }
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory must outlive the last copies
    }

    if (ctrl->abort && elect_one()) {
        const bool prep = warp < 4 * G;  // of a group, warp 2's thread issues the loads
        abort_drain(ctrl, warp, prep && (warp & 3) == 2 ? &ctrl->raw[warp >> 2] : LN && prep && (warp & 3) == 3 ? &ctrl->gate[warp >> 2] : nullptr, p.status);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS) : "memory");
    }
}

// Tensor map over the checkpoint buffer seen as an fp32 matrix [records * 80 rows][64 floats]; box = 64 rows x
// 32 floats (128 bytes) with the 128-byte swizzle of 32-byte units.  Encoded through the runtime's driver-entry-point query
// (the library does not link against libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static bool encode_checkpoint_map(CUtensorMap* m, float* base, long long records) {
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)(records * (CK_FLOATS / N))};
    const cuuint64_t strides[1] = {(cuuint64_t)(N * sizeof(float))};
    const cuuint32_t box[2] = {32, (cuuint32_t)N};
    const cuuint32_t es[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int G, bool RND, bool LN, bool TAIL, bool AFF = false> static int launch_tt(const FwdParams& p, cudaStream_t stream) {
    auto kern = wkv7_fwd_tc_kernel<G, RND, LN, TAIL, AFF>;
    const int smem = G * (LN ? G_BYTES_LN : G_BYTES_PLAIN) + (int)sizeof(Ctrl) + 1024;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return kLaunchFailed;
    FwdMaps maps;
    memset(&maps, 0, sizeof(maps));
    if (p.ckpt && !encode_checkpoint_map(&maps.ck, p.ckpt, p.B * p.H * ((p.T + L - 1) / L))) return kLaunchFailed;
    const void* ins[8] = {p.y, p.r, p.w, p.k, p.a, p.b, p.v, p.g};
    CUtensorMap* const ms[8] = {&maps.y, &maps.in[0], &maps.in[1], &maps.in[2], &maps.in[3], &maps.in[4], &maps.in[5], &maps.g};
    for (int i = 0; i < (LN ? 8 : 7); ++i)
        if (ins[i] && !encode_bthn_map(ms[i], const_cast<void*>(ins[i]), p.B, p.T, p.H, p.st)) return kLaunchFailed;
    const WorkSplit ws = plan_work(p.B * p.H, (p.T + L - 1) / L, 1, p.sT ? p.flags : nullptr);
    if (ws.flags && cudaMemsetAsync(ws.flags, 0, ws.ctas * sizeof(unsigned), stream) != cudaSuccess) return kLaunchFailed;
    kern<<<(unsigned)ws.ctas, 128 * (G + 2), smem, stream>>>(p, ws, maps);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

template <int G, bool RND, bool LN> static int launch_t(const FwdParams& p, cudaStream_t stream) {
    return p.T % L ? launch_tt<G, RND, LN, true>(p, stream) : launch_tt<G, RND, LN, false>(p, stream);
}

// Exercises the bounded wait and the abort path with the kernel's own mbar_wait: one CTA of four warps;
// warp 0 waits (polling) and warp 1 waits (suspended) on mbarriers that nothing ever arrives on, with a
// short limit; warps 2 and 3 then wait on a third barrier with the full limit and must fall through at
// once because the CTA has aborted.  Leaves kDeviceTimeout in the status word and writes, per warp, the
// cycles its wait took.  No tensor memory, no tcgen05: nothing here can fault or hang.
__global__ void __launch_bounds__(128) bounded_wait_selftest_kernel(long long limit, int* status, long long* cycles) {
    __shared__ Ctrl ctrl;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        for (int g = 0; g < 3; ++g) mbar_init(&ctrl.full[g], 1);
        ctrl.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // clock reads that cannot be scheduled across the barrier / the wait: they take a value produced there as input
    auto clock_after = [](int dep) { long long t; asm volatile("mov.u64 %0, %%clock64;" : "=l"(t) : "r"(dep) : "memory"); return t; };
    const long long t0 = clock_after(__syncthreads_or(0));
    if (warp == 0) mbar_wait<false>(&ctrl.full[0], 0, &ctrl, status, limit);
    else if (warp == 1) mbar_wait<true>(&ctrl.full[1], 0, &ctrl, status, limit);
    const long long t1 = clock_after(__syncthreads_or(0));
    if (warp >= 2) mbar_wait<true>(&ctrl.full[2], 0, &ctrl, status);  // full limit, but the abort flag is up
    const long long t2 = clock_after(ctrl.abort);
    if ((tid & 31) == 0) cycles[warp] = warp < 2 ? t1 - t0 : t2 - t1;
}

}  // namespace tc

int launch_bounded_wait_selftest(long long limit_cycles, int* status, long long* cycles, cudaStream_t stream) {
    tc::bounded_wait_selftest_kernel<<<1, 128, 0, stream>>>(limit_cycles, status, cycles);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

template <bool LN> static int launch_ln(const FwdParams& p, int groups, cudaStream_t stream) {
    switch (groups) {
        case 2: return tc::launch_t<2, true, LN>(p, stream);
        case 3: return tc::launch_t<3, true, LN>(p, stream);
        case 4: return tc::launch_t<4, true, LN>(p, stream);
        case -2: return tc::launch_t<2, false, LN>(p, stream);
        case -3: return tc::launch_t<3, false, LN>(p, stream);
        case -4: return tc::launch_t<4, false, LN>(p, stream);
        default: return kBadShape;
    }
}

int launch_fwd_tc(const FwdParams& p, int groups, bool ln, cudaStream_t stream) {
    if (p.sM) return p.T % L ? tc::launch_tt<4, true, false, true, true>(p, stream) : tc::launch_tt<4, true, false, false, true>(p, stream);
    return ln ? launch_ln<true>(p, groups, stream) : launch_ln<false>(p, groups, stream);
}

}  // namespace wkv7
