// WKV7 forward on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory), bf16 IO.
//
// Same mathematics as wkv7_fwd.cu (the reference's forward_kernel, wind_rwkv/rwkv7/attn.cu:11-106, and
// with LN = true its fused GroupNorm + bonus + gate variant, wind_rwkv/rwkv7/attn_ln.cu:106-212),
// different machine mapping.  One CTA per SM walks its share of the chunks (WorkSplit: whole chains and at most two pieces of
// cut ones).  The 64x64 state S[value][key] lives in tensor memory and is never held in registers: per 16-step chunk two
// elected threads issue 24 tcgen05.mma instructions (M = 64 value rows, TF32 operands, fp32 accumulate)
//     ahead   [X | Yp] = V^T [AK;QK]^T,  S' = V^T kwf        needs no state: issued while the chunk before it drains; A = V^T from
//                                                            tensor memory, S' in the next of three state buffers
//     hop 1   [X | Yp] += S [wa;wq]^T                        A = S straight from tensor memory
//             S' += S diag(fw)                               eight N = 8 products apply the decay; issued beside hop 1
//     hop 2   S' += X (AI^T bwf),  Y = Yp + X (QB AI)^T      A = X from tensor memory
// with kwf = kwi*fw, bwf = bwi*fw, so the column scaling of the state never touches a CUDA core.  U = X AI^T itself is never
// formed: AI^T bwf and QB AI come from two small products off the chain.  An accumulator that the next product reads as its A
// operand needs an explicit completion wait (tcgen05.commit -> mbarrier); only same-accumulator products of one thread are ordered by the
// tensor pipe.
// What bounds it: the instructions of its 24 warps, 3500 a chunk, at 60 % of the issue slots, with some 1000 shared-memory wavefronts of loads
// and stores and 360 of operand reads beside them; a group's loop (scan, loads, operand tiles, the scores' product) is 4400 cycles for every
// third chunk, the chain itself some 1000.  1400 cycles a chunk without checkpoints (B8 T8192 H40: 795 us, 881 before the slots, the
// readers and the helper below), 1850 with (B64 T1024 H12: 332 us, 3.3 TB/s of it written).  With them, 7 % more instructions at 52 % of the
// issue slots, and the raw tiles come late out of a DRAM that is at 4.8 TB/s: 4.6 warps per issue wait for loads instead of 2.9.  It is not the
// writes alone: of 369 us with the L2 flushed, the records' matrices left out (a fifth of 1 GB) save 16, the states 57, both 86.
//
// Warp roles (768 threads).  A chunk's operand tiles, scores and results lie in one of S slots of shared and tensor memory, a place
// apart from the warps that fill it: chunk c has slot c % S from its tiles until its results have been read.  (With a slot per preparation
// group, four of them, a chunk's way through its slot, 5200 cycles, was what a chunk cost four times over.)
// PREP groups of four warps prepare every PREP-th chunk each (scan, operand tiles); READERS groups of four warps take the results out (output
// tiles, checkpoint states, attn_ln's epilogue).  Eight service warps serve all chunks, each a stage of their way to the chain (a warp takes
// some 500 to 800 cycles per stage, so that a stage shared with another one makes chunks wait): 16, 17 read the scores back from their quarter of
// tensor memory, mask them and write AK, AB, QK, QB; 18, 23 invert (I - AB) and form QB AI (even and odd chunks); 20, 21 form AI^T bwf; 19
// issues the two hops of the chain and 22, its helper, what does not stand behind the first hop.  The kernel's hot code has to stay
// small: its warps run different parts of it at the same time, and while the compiler unrolled the loops of the chain and its
// helper (9 KB more) and waits were twice as long, B64 T1024 H12 without checkpoints took 292 us where it took 273 afterwards.
// (Not better: the scores by mma.sync in the preparation warps - every operand is read four times, 1.2 times slower; forming the
// inverse's two 8x8 blocks in lanes 0-15 only, 1 % slower; waits with a time hint; the raw tiles' loads by the readers - a load takes its
// thread some 300 cycles, and the readers became the longest loop; the loads after the next tiles instead of before them.)
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
// [64 rows][32 floats] halves, conflict-free 8-byte stores) and two
// threads issue a tensor-map bulk store each (cp.async.bulk.tensor.2d, shared -> global), which undo the
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

// a chunk's shared memory, a slot of S (byte offsets; tensor-core tiles first, all 1024-byte aligned)
constexpr int G_WAQ = 0;       // [wa;wq]   32 rows x 64, K-major            8192
constexpr int G_KB = 8192;     // [kwi;bwi] 32 rows x 64, K-major            8192 (directly after WAQ: the M = 64 score
                               //                                                 product reads rows 32..63 from here, unused);
                               // time step s of every eight in row kb_row(s): the score product's columns then come back as
                               // 8x4 blocks with a column per lane, which stmatrix can store
constexpr int G_ABT = G_KB;           // AB transposed, fp32 [16][ABS], once the score product has read [kwi;bwi]   1280
constexpr int G_QBU = G_KB + 2048;    // QB AI, 16 x 16, K-major, likewise                                          1024
constexpr int G_KWF = 16384;   // kwf [time][key]    MN-major                4096
constexpr int G_BWF = 20480;   // bwf [time][key]    MN-major                4096
constexpr int G_SC = 24576;    // [AK;QK]  32 rows x 16, K-major             2048
constexpr int G_AI = 26624;    // AI^T     16 x 16, K-major                  1024
constexpr int G_QB = 27648;    // QB       16 x 16, K-major                  1024
static_assert(G_AI == G_SC + 2048 && G_QB == G_AI + 1024, "[AK;QK], AI^T, QB must be contiguous: they leave as one bulk copy");
constexpr int G_DF = 28672;    // eight 8x8 diagonal blocks of fw, K-major   2048
constexpr int G_BYTES = 30720;
static_assert(G_BYTES % 1024 == 0, "tile alignment");
// behind the slots: the raw tiles' ring, the output tiles and the readers' staging
// preparation groups and reader groups, four warps each, four groups in all; attn_ln's readers have its epilogue to do
template <bool LN> constexpr int PREP = LN ? 2 : 3;
template <bool LN> constexpr int READERS = 4 - PREP<LN>;
constexpr int THREADS_TC = 128 * 6;      // these and eight service warps
constexpr int RAW_BYTES = 6 * RAW_TILE;  // q, w, k, a, b, v of a chunk
constexpr int Y_BYTES = RAW_TILE;        // an output tile [time][value], bf16, 128-byte swizzle; two of them
constexpr int STAGE_BYTES = N * N * 4;   // a checkpoint state on its way out
// attn_ln's epilogue
constexpr int LN_YS = 68;                  // row stride (floats) of the fp32 [time][value] staging of Y
constexpr int LN_PART = L * LN_YS * 4;     // byte offset of the per-warp partial sums [4][16][2] behind it
constexpr int LN_V = LN_PART + 512;        // V [time][value], bf16, 16-byte units XOR-ed with the row
constexpr int LN_BYTES = LN_V + RAW_TILE;
constexpr int R = 4;                     // raw tiles in flight
template <int S, bool LN> constexpr int AT_RAW = S * G_BYTES;
template <int S, bool LN> constexpr int AT_Y = AT_RAW<S, LN> + R * RAW_BYTES;
template <int S, bool LN> constexpr int AT_STAGE = AT_Y<S, LN> + 2 * Y_BYTES;
template <int S, bool LN> constexpr int AT_LN = AT_STAGE<S, LN> + READERS<LN> * STAGE_BYTES;
template <int S, bool LN> constexpr int AT_CTRL = AT_LN<S, LN> + (LN ? READERS<LN> * LN_BYTES : 0);

// tensor-memory columns (32-bit each, 128 lanes; the M = 64 products use lanes 0-15 of each 32-lane quarter)
constexpr int STATES = 3;    // state buffers of 64 columns: chunk c reads c % 3 and writes (c + 1) % 3
constexpr int C_S = 0;
constexpr int C_INIT = 192;  // start state of the next segment (written by the group that prepares its first chunk)
constexpr int C_XY = 256;    // + 32 * slot: X (16) | Y (16) of the slot's chunk; before that its score products,
                             // [AK|AB] in lanes 0-15, [QK|QB] in lanes 32-47 (columns permuted, see G_KB)
constexpr int C_V = 416;     // + 16 * slot: V^T [value][time] of the slot's chunk

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

// One chunk of the CTA's work list, as its preparation group and the readers need it.
struct ChunkDesc {
    long long off;   // element offset of (batch, time 0, head) in the inputs
    int bh, c;       // chain and chunk within it
    int c_end;       // end of the segment (the chunks of this chain that follow one another in the list)
    int flags;
    int bi, hi;      // batch entry, head
    int prev_first;  // SEG_FIRST: list position of the previous segment's first chunk if that lies less than S back, else -1
};
enum : int { SEG_FIRST = 1, SEG_LAST = 2 };  // first / last chunk of a segment
// A descriptor is written when its chunk's loads are about to be issued and read last by the readers; RING of them outlast that
// (loads run R chunks ahead of a scan, which is at most S + PREP chunks ahead of the readers).
constexpr int RING = 16;

struct Ctrl {
    uint64_t full[5], done[5], score[5], read[5], mats[5], inv[5], rec[5], raw[12], hop, go[2];
    uint32_t tiles[5];         // warps that have written their part of a slot's operand tiles, counted on over all chunks
    uint32_t tmem_base;
    volatile int abort;
    ChunkDesc desc[RING];      // where the chunk at list position v lies: v % RING
    float bdot[RING][4][L];    // attn_ln: per-warp partial bonus dots [list position % RING][warp][time]
    // abort path only, a set per warp: completion of its products, and what its waits take in place of the abort flag
    uint64_t drain[THREADS_TC / 32];
    volatile int never_set[THREADS_TC / 32];
};

// Bounded wait for the phase with the given parity.  Returns at once when the CTA has aborted.
// SLEEP: 40 ns between polls, so that the many warps that wait for the chain do not take issue slots from the warps that work; the
// chain's own short waits poll.  (0, 16 and 100 ns make no difference: try_wait itself suspends a warp for a while.)
template <bool SLEEP>
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, Ctrl* ctrl, int* status, long long limit = WAIT_LIMIT) {
    // Written out, since it stands at some twenty places of code that has to stay small; the status word is written when the CTA ends.
    if (SLEEP)
        asm volatile("{\n.reg .pred P;\n.reg .b32 s, t;\nmov.u32 s, %%clock;\n"
                     "WAIT: mbarrier.try_wait.parity.shared::cta.b64 P, [%0], %1;\n@P bra DONE;\n"
                     "ld.volatile.shared.u32 t, [%2];\nsetp.ne.u32 P, t, 0;\n@P bra DONE;\nnanosleep.u32 40;\n"
                     "mov.u32 t, %%clock;\nsub.u32 t, t, s;\nsetp.lt.u32 P, t, %3;\n@P bra WAIT;\n"
                     "st.volatile.shared.u32 [%2], 1;\nDONE:\n}\n" ::"r"(smem_u32(bar)), "r"(parity), "r"(smem_u32((const void*)&ctrl->abort)), "r"((uint32_t)limit) : "memory");
    else
        asm volatile("{\n.reg .pred P;\n.reg .b32 s, t;\nmov.u32 s, %%clock;\n"
                     "WAIT: mbarrier.try_wait.parity.shared::cta.b64 P, [%0], %1;\n@P bra DONE;\n"
                     "ld.volatile.shared.u32 t, [%2];\nsetp.ne.u32 P, t, 0;\n@P bra DONE;\n"
                     "mov.u32 t, %%clock;\nsub.u32 t, t, s;\nsetp.lt.u32 P, t, %3;\n@P bra WAIT;\n"
                     "st.volatile.shared.u32 [%2], 1;\nDONE:\n}\n" ::"r"(smem_u32(bar)), "r"(parity), "r"(smem_u32((const void*)&ctrl->abort)), "r"((uint32_t)limit) : "memory");
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
// loads that this warp may have in flight, so that neither tensor memory nor shared memory is released under them.
// (`loaded`: the last list position that it has loaded, `every` positions after the one before; at most four of them are on their way.)
__device__ __forceinline__ void abort_drain(Ctrl* ctrl, int warp, int loaded, int every, int barriers, int* status) {
    volatile int* never_set = &ctrl->never_set[warp];
    *never_set = 0;
    mbar_init(&ctrl->drain[warp], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
    tc_commit(&ctrl->drain[warp]);
    const uint32_t since = clock();  // the kernel's own limit: products may stand behind a warp that still waits for a hand-off
    while (!mbar_test(&ctrl->drain[warp], 0) && !*never_set)
        if ((uint32_t)clock() - since > (uint32_t)WAIT_LIMIT) give_up(never_set, status);
    for (int i = 0, v = loaded; i < 4 && v >= 0; ++i, v -= every) {
        *never_set = 0;  // (a wait that has run out must not spoil the next one)
        mbar_wait_bounded<true>(&ctrl->raw[v % barriers], (v / barriers) & 1, never_set, status);
    }
}
// named barrier of a preparation or reader group (the id in a register: a switch over immediate ids costs instruction-cache space)
__device__ __forceinline__ void group_bar(int grp) { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); }
__device__ __forceinline__ void readers_ready() { asm volatile("bar.sync 5, 512;" ::: "memory"); }  // readers and groups

// shared-memory matrix descriptors (sm_100 version field set) in two words: the upper one is a constant, byte offsets / 16 are added to the
// lower one (64-bit arithmetic on them cost the issuing threads half of their instructions)
__device__ __forceinline__ uint32_t desc_kmajor(uint32_t saddr) { return ((saddr >> 4) & 0x3fff) | ((128 >> 4) << 16); }
__host__ __device__ constexpr uint32_t kmajor(uint32_t sbo) { return (sbo >> 4) | (1u << 14); }
__device__ __forceinline__ uint32_t desc_mnmajor(uint32_t saddr) { return ((saddr >> 4) & 0x3fff) | ((2048 >> 4) << 16); }  // 128-byte swizzle with 32-byte base
constexpr uint32_t MNMAJOR = (512 >> 4) | (1u << 14) | (1u << 29);
// instruction descriptor: fp32 accumulate, TF32 operands
__host__ __device__ constexpr uint32_t idesc(int n, bool b_mn, int m = 64) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint32_t a, uint32_t a_hi, uint32_t b, uint32_t b_hi, uint32_t id, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %2};\nmov.b64 db, {%3, %4};\nsetp.ne.b32 p, %6, 0;\ntcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %5, p;\n}\n"
                 ::"r"(d), "r"(a), "r"(a_hi), "r"(b), "r"(b_hi), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t b_hi, uint32_t id, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\n.reg .b64 db;\nmov.b64 db, {%2, %3};\nsetp.ne.b32 p, %5, 0;\ntcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], db, %4, p;\n}\n"
                 ::"r"(d), "r"(a), "r"(b), "r"(b_hi), "r"(id), "r"(acc) : "memory");
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

// the same for what nothing but the tensor core reads: it does not look at the 13 bits below
__device__ __forceinline__ float rnd_op(float x) { return __uint_as_float(__float_as_uint(x) + 0x1000u); }
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
    return R ? make_float4(rnd_op(f[0].x), rnd_op(f[0].y), rnd_op(f[1].x), rnd_op(f[1].y)) : make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
}
template <bool R> __device__ __forceinline__ F2 rnd2(F2 a) { return R ? f2(rnd_op(a.x), rnd_op(a.y)) : a; }
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

// A warp's 16 values x 16 time steps of an accumulator (the layout of tmem_ld_frag) as bf16 into a [time][value] tile: 128-byte rows, 16-byte
// units XOR-ed with the row.
__device__ __forceinline__ void store_transposed(unsigned char* tile, const uint32_t* x, int wg, int lane) {
    uint32_t h[4];  // 8x8 blocks: values 0-7 | 8-15 of time steps 0-7, then of time steps 8-15
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = pack_bf16x2_rn(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1]));
    const int t = (lane & 7) + 8 * (lane >> 4), unit = 2 * wg + ((lane >> 3) & 1);  // row address of block lane / 8
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                 ::"r"(smem_u32(tile + t * ROWB + ((unit ^ (t & 7)) << 4))), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
}

// AFF: the segments of a sequence cut in time as affine maps, S -> S M + R (wkv7_time_split.cu).  The state has 128 rows, R in lanes 0-63 and
// M in lanes 64-127 of tensor memory (M = 128 products; V^T has zeros there): one walk over the chunks instead of two, and without the
// output's products, tiles and stores.  R starts from zero (a sequence's first segment: from s0), M from the identity; they leave
// through sT and sM.
// TAIL: the sequence length is not a multiple of 16 (a build of its own, so that whole-chunk sequences carry none of
// the row tests in their register budget).

// A place in a ring of M, and the parity of the phase that its barrier is in, advanced without divisions: those were 40 % of the time of
// the thread that issues the chain.
template <int M> struct Place {
    int i;
    uint32_t parity;
    __device__ __forceinline__ void advance(int by) {  // by <= M
        i += by;
        if (i >= M) { i -= M; parity ^= 1; }
    }
};
struct alignas(64) FwdMaps { CUtensorMap ck, y, in[6]; };  // checkpoint states; output; q, w, k, a, b, v

template <int S, bool RND, bool LN, bool TAIL, bool AFF>
__global__ void __launch_bounds__(THREADS_TC, 1) wkv7_fwd_tc_kernel(FwdParams p, WorkSplit ws, const __grid_constant__ FwdMaps maps) {
    using IoT = __nv_bfloat16;
    constexpr int PREP = tc::PREP<LN>, READERS = tc::READERS<LN>, RB = R * PREP;  // raw tiles; their barriers: each is waited on by one group, which sees all of its phases
    constexpr int NCOLS = 512, M = AFF ? 128 : 64, NX = AFF ? 16 : 32;  // rows of the state; columns X | Yp or X alone
    static_assert(!(AFF && LN), "the maps have no output");
    static_assert(STATES * 64 <= C_INIT && C_INIT + 64 <= C_XY && C_XY + 32 * S <= C_V && C_V + 16 * S <= NCOLS, "tensor memory columns");
    static_assert(S >= 3 && S <= 5 && R + PREP + S < RING && PREP <= S && (READERS == 1 || S % READERS == 0), "descriptors, see RING");
    // Register reallocation.  setmaxnreg.inc blocks, without a bound, until the CTA's
    // register pool can satisfy it, and the pool is what the CTA was launched with: 768 threads x 80
    // registers (65536 / 768 rounded down to a multiple of 8; build.py checks that ptxas reports 80).
    // The raised and lowered counts must therefore fit into that pool exactly or with room to spare.
    constexpr int LAUNCH_REGS = 80, PREP_REGS = 96, SERVICE_REGS = 48;
    static_assert(128 * 4 * PREP_REGS + 256 * SERVICE_REGS <= THREADS_TC * LAUNCH_REGS, "setmaxnreg would never be satisfied");
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* sm = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(sm + AT_CTRL<S, LN>);
    constexpr int Z0 = G_QB, Z1 = AT_Y<S, LN>;  // affine maps only (which have neither): zeros, 256 bytes each
    static_assert(Z0 < G_DF && Z1 > S * G_BYTES && Z1 < 1 << 18, "descriptors have positive strides of 14 bits in 16 bytes");

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // provably warp-uniform
    const int nchunks = ws.per_chain;  // the last chunk may be partial: its missing rows read as zeros
    const WorkRange work(ws, blockIdx.x);
    const int tail = TAIL ? (int)(p.T - (long long)(nchunks - 1) * L) : L;  // time steps of the last chunk (1..16)

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&ctrl->full[s], 2 + 1 + 4);
            mbar_init(&ctrl->mats[s], AFF ? 1 : 2);
            mbar_init(&ctrl->inv[s], 1);
            mbar_init(&ctrl->rec[s], 1);
            mbar_init(&ctrl->done[s], 1);
            mbar_init(&ctrl->score[s], 1);
            mbar_init(&ctrl->read[s], 4);
        }
        for (int r = 0; r < RB; ++r) mbar_init(&ctrl->raw[r], 4);
        mbar_init(&ctrl->hop, 2);
        mbar_init(&ctrl->go[0], 2);
        mbar_init(&ctrl->go[1], 2);
        for (int s = 0; s < S; ++s) ctrl->tiles[s] = 0;
        ctrl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto describe = [&](int v, int at) {
        ChunkDesc d;
        work.locate(v, nchunks, d.bh, d.c);
        d.bi = (int)((unsigned)d.bh / (unsigned)p.H);
        d.hi = d.bh - d.bi * (int)p.H;
        d.off = d.bi * p.st.b + d.hi * p.st.h;
        d.c_end = v < work.h ? work.h : nchunks;  // the start piece is chunks 0 .. h - 1 of its chain
        d.flags = (work.starts_segment(v, d.c) ? SEG_FIRST : 0) | (d.c + 1 == d.c_end ? SEG_LAST : 0);
        d.prev_first = -1;
        if (d.flags & SEG_FIRST)
            for (int u = v - 1; u >= 0 && u > v - S; --u) {
                int ub, uc;
                work.locate(u, nchunks, ub, uc);
                if (work.starts_segment(u, uc)) { d.prev_first = u; break; }
            }
        ctrl->desc[at] = d;
    };
    if (tid < RING) describe(min(tid, work.n - 1), tid);  // (those that are not due yet get values of a chunk that exists: an aborted CTA may look at them)
    // the off-diagonal zeros of the decay blocks are written once
    for (int i = tid; i < S * (2048 / 16); i += THREADS_TC)
        *reinterpret_cast<uint4*>(sm + (i / 128) * G_BYTES + G_DF + (i % 128) * 16) = make_uint4(0, 0, 0, 0);
    if (AFF && tid < 32)  // zeros before and after them: products of 16 columns (the least with 128 rows) take a block and one of these
        *reinterpret_cast<uint4*>(sm + (tid & 16 ? Z1 : Z0) + (tid & 15) * 16) = make_uint4(0, 0, 0, 0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctrl->tmem_base)), "r"(NCOLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctrl->tmem_base;
    stream_wait();

    // Start state of a segment -> tensor memory and its checkpoint: warp wq of the group owns lanes 32 wq .. 32 wq + 31, of
    // which lanes 0-15 hold value rows 16 wq .. 16 wq + 15.  A chain's first chunk starts from s0 (or zeros); a chain that
    // the list cuts starts from the state that the CTA before this one left in sT (see WorkSplit).
    auto load_state = [&](const ChunkDesc& d, int wq) {
        if (__any_sync(0xffffffffu, ctrl->abort)) return;
        const int sbh = d.bh, sc = d.c;
        const uint32_t ta = tmem + C_INIT;
        if (d.prev_first >= 0) {  // its start state has been used, by products that read it where this one is written
            mbar_wait<true>(&ctrl->done[d.prev_first % S], (d.prev_first / S) & 1, ctrl, p.status);
            tc_fence_after();
        }
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

    // the list position at which the segment after the one that begins at c begins
    auto next_segment = [&](int c) { return c < work.h ? work.h : c < work.n - work.t ? min(c + nchunks, work.n - work.t) : work.n; };
    int loaded = -1;  // list position of the last chunk whose raw tiles this warp has had a share in loading
    if (warp >= 16) {
        // ------------------------------ service warps -----------------------------------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SERVICE_REGS));
        constexpr int W0 = 16;
        const int q = warp & 3;  // (of the score and fold warps:) tensor-memory lanes 0-15 or 32-47
        const uint32_t tq = tmem + ((uint32_t)(32 * q) << 16);
        if (warp == W0 + 3) {
          if (elect_one()) {
            const uint32_t sb = smem_u32(sm), dK = desc_kmajor(sb), dMN = desc_mnmajor(sb);  // of the first slot's beginning
            int seg_first = 0;  // list position at which the next segment begins
            Place<S> at{0, 0};
            uint32_t Sa = tmem + C_S, Sn = Sa + 64, Sf = Sa + 128;  // state that the current chunk reads, the one it writes, the third one
#pragma unroll 1
            for (int c = 0; c < work.n; ++c, at.advance(1)) {  // position in the CTA's list
                const uint32_t XY = tmem + C_XY + 32 * at.i, off = at.i * (G_BYTES >> 4), dWAQ = dK + off + (G_WAQ >> 4), dQBU = dK + off + (G_QBU >> 4), dBWU = dMN + off + (G_BWF >> 4);
                uint32_t A = Sa;
                if (c == seg_first) {
                    A = tmem + C_INIT;
                    seg_first = next_segment(c);
                }
                // the V parts are in place, and the state, this chunk's A operand, is there.  (One barrier for both, and one
                // for hop 1 and the decay: every wait of this thread is some 200 cycles of the chain, also where nothing is left to wait for.)
                mbar_wait<false>(&ctrl->go[c & 1], (c >> 1) & 1, ctrl, p.status);
                tc_fence_after();
                // hop 1
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) mma_ts(XY, A + 8 * ks, dWAQ + ks * 16, kmajor(2048), idesc(NX, false, M), 1);
                tc_commit(&ctrl->hop);
                mbar_wait<false>(&ctrl->hop, c & 1, ctrl, p.status);
                tc_fence_after();
                // hop 2: the X part of the state update and of Y
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) mma_ts(Sn, XY + 8 * ks, dBWU + ks * 64, MNMAJOR, idesc(64, true, M), 1);
#pragma unroll
                for (int ks = 0; ks < (AFF ? 0 : 2); ++ks) mma_ts(XY + 16, XY + 8 * ks, dQBU + ks * 16, kmajor(512), idesc(16, false, M), 1);
                tc_commit(&ctrl->go[(c + 1) & 1]);
                tc_commit(&ctrl->done[at.i]);
                const uint32_t t = Sa;
                Sa = Sn; Sn = Sf; Sf = t;
            }
          }
        } else if (warp == W0 + 6) {
            // ---- the chain's helper
            // The products of the chain that do not depend on its first hop: a thread takes some 25 cycles for each that it issues, and with all 24
            // of a chunk in one thread that was what the chain waited for.
            if (elect_one()) {
                const uint32_t sb = smem_u32(sm), dK = desc_kmajor(sb), dMN = desc_mnmajor(sb);
                int seg_first = 0;
                const int release_at = max(0, work.n - S);
                Place<S> at{0, 0};
                uint32_t Sa = tmem + C_S, Sn = Sa + 64, Sf = Sa + 128;
#pragma unroll 1
                for (int c = 0; c < work.n; ++c, at.advance(1)) {
                    if (c == release_at) stream_release();
                    const uint32_t XY = tmem + C_XY + 32 * at.i, V = tmem + C_V + 16 * at.i, off = at.i * (G_BYTES >> 4), dSC = dK + off + (G_SC >> 4), dKWF = dMN + off + (G_KWF >> 4), dDF = dK + off + (G_DF >> 4);
                    uint32_t A = Sa;
                    if (c == seg_first) {
                        A = tmem + C_INIT;
                        seg_first = next_segment(c);
                    }
                    // The V parts, X | Yp and S', need no state: they are issued while the chunk before drains.  When the chunk is full, its
                    // slot's last results have been read, so X | Y is free, and so has been the state of three chunks before, whose buffer was
                    // last read as an operand by the chunk before the last, which is done.
                    mbar_wait<false>(&ctrl->full[at.i], at.parity, ctrl, p.status);
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) mma_ts(XY, V + 8 * ks, dSC + ks * 16, kmajor(512), idesc(NX, false, M), ks > 0);
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) mma_ts(Sn, V + 8 * ks, dKWF + ks * 64, MNMAJOR, idesc(64, true, M), ks > 0);
                    tc_commit(&ctrl->go[c & 1]);  // (the chain may be a chunk behind here)
                    if (c == 0) mbar_arrive(&ctrl->go[0]);
                    // the decay of the old state goes into the other buffer beside hop 1
                    if (c > 0) mbar_wait<false>(&ctrl->done[at.i > 0 ? at.i - 1 : S - 1], at.i > 0 ? at.parity : at.parity ^ 1, ctrl, p.status);
                    tc_fence_after();
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        if (!AFF) {
                            mma_ts(Sn + 8 * b, A + 8 * b, dDF + b * 16, kmajor(256), idesc(8, false), 1);
                        } else {  // rows 0-7 and 8-15 of the operand: the block and zeros, or zeros and the block
                            const uint32_t blk = sb + at.i * G_BYTES + G_DF + 256 * b;
                            mma_ts(Sn + 16 * (b >> 1), A + 8 * b, desc_kmajor(b & 1 ? sb + Z0 : blk), kmajor(b & 1 ? blk - (sb + Z0) : sb + Z1 - blk), idesc(16, false, M), 1);
                        }
                    }
                    // (The tensor pipe does not keep the order of what different warps issue, also behind a fence: the decay must have
                    // been added, not only issued, when hop 2 adds to the same state.)
                    tc_commit(&ctrl->hop);
                    const uint32_t t = Sa;
                    Sa = Sn; Sn = Sf; Sf = t;
                }
            }
        } else if (AFF && warp == W0 + 1) {
            // (QK and QB are for the output)
        } else if (warp == W0 || warp == W0 + 1) {
            // ---- score warps: warp W0 reads [AK|AB], warp W0 + 1 reads [QK|QB]
            Place<S> at{0, 0};
#pragma unroll 1
            for (int c = 0; c < work.n; ++c, at.advance(1)) {
                const int s = at.i;
                unsigned char* gs = sm + s * G_BYTES;
                mbar_wait<true>(&ctrl->score[s], at.parity, ctrl, p.status);
                tc_fence_after();
                uint32_t x[16];
                tmem_ld_frag4(tq + C_XY + 32 * s, x);
                tmem_ld_wait();
                tc_fence_before();
                // the previous chunk's matrices have left for its checkpoint record
                if (p.ckpt && c >= S) mbar_wait<true>(&ctrl->rec[s], at.parity ^ 1, ctrl, p.status);
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
                if (lane == 0) mbar_arrive(&ctrl->mats[s]);
            }
        } else if (warp == W0 + 2 || warp == W0 + 7) {
            // ---- inverse warps (even and odd chunks; the matrices become ready in the order of the chunks, so a warp never sees a
            // barrier two phases behind)
            Place<S> at{warp == W0 + 7 ? 1 : 0, 0};
#pragma unroll 1
            for (int c = at.i; c < work.n; c += 2, at.advance(2)) {
                const int s = at.i;
                unsigned char* gs = sm + s * G_BYTES;
                mbar_wait<true>(&ctrl->mats[s], at.parity, ctrl, p.status);
                tri_inverse_tc(reinterpret_cast<float*>(gs + G_ABT), gs + G_AI, lane);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->inv[s]);
                if (!AFF) {  // QB AI (see the fold warps)
                    const int g8 = lane >> 2, t4 = lane & 3;
                    const uint32_t tile = (lane >> 4) * 512 + ((lane >> 3) & 1) * 128 + (lane & 7) * 16;  // A operands: 8x4 blocks (rows 0-7 | 8-15) x (4 columns | the next 4)
                    float acc[2][4] = {};
#pragma unroll
                    for (int kb = 0; kb < 2; ++kb) {
                        uint32_t a[4], ai[4];
                        ldmatrix4(ai, smem_u32(gs + G_AI) + tile + kb * 256);
                        ldmatrix4(a, smem_u32(gs + G_QB) + tile + kb * 256);
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt) mma_tf32_raw(acc[nt], a[0], a[2], a[1], a[3], ai[2 * nt], ai[2 * nt + 1]);  // B = AI^T by rows
                    }
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            *reinterpret_cast<float2*>(gs + G_QBU + kchunk(g8 + 8 * h, 2 * nt + (t4 >> 1), 512) + (t4 & 1) * 8) = make_float2(rnd_op(acc[nt][2 * h]), rnd_op(acc[nt][2 * h + 1]));
                    fence_async_smem();
                }
                __syncwarp();
                if (elect_one()) {
                    mbar_arrive(&ctrl->full[s]);
                    // The chunk's four 16x16 matrices go into its checkpoint record: the three tiles [AK;QK], AI^T, QB are
                    // contiguous in shared memory and are stored as they are, by one bulk copy.
                    if (p.ckpt) {
                        const ChunkDesc& d = ctrl->desc[c % RING];
                        float* ckm = p.ckpt + ((long long)d.bh * nchunks + d.c) * CK_FLOATS + CK_MATS;
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                     ::"l"(__cvta_generic_to_global(ckm)), "r"(smem_u32(gs + G_SC)), "n"(4 * L * L * 4) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        mbar_arrive(&ctrl->rec[s]);
                    }
                }
                __syncwarp();
            }
        } else {
            // ---- fold warps: U = X AI^T, so U bwf = X (AI^T bwf) and U QB^T = X (QB AI)^T: one dependent tensor-core round trip per chunk
            // less for the chain.  Warps W0 + 4, W0 + 5 form 32 key columns of AI^T bwf each, in the place of bwf; the inverse warps QB AI.
            // (mma.sync: as tcgen05 products they read 104 wavefronts of operands instead of 64, 64 rows of A for 32 or 16 used ones, and
            // the results came back through tensor memory.)
            const int g8 = lane >> 2, t4 = lane & 3;
            const uint32_t at = (lane >> 4) * 512 + ((lane >> 3) & 1) * 128 + (lane & 7) * 16;  // A operands: 8x4 blocks (rows 0-7 | 8-15) x (4 columns | the next 4)
            Place<S> place{0, 0};
#pragma unroll 1
            for (int c = 0; c < work.n; ++c, place.advance(1)) {
                const int s = place.i;
                unsigned char* gs = sm + s * G_BYTES;
                mbar_wait<true>(&ctrl->inv[s], place.parity, ctrl, p.status);
                uint32_t ai[2][4];
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) ldmatrix4(ai[kb], smem_u32(gs + G_AI) + at + kb * 256);
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
                        *reinterpret_cast<float2*>(bw + (g8 + 8 * h) * 128 + ((nt ^ (g8 & 3)) << 5) + t4 * 8) = make_float2(rnd_op(acc[nt][2 * h]), rnd_op(acc[nt][2 * h + 1]));
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctrl->full[s]);
            }
        }
        __syncwarp();
    } else if (warp >= 4 * PREP) {
        // ------------------------------ readers -------------------------------------------------
        // Results of every chunk: Y^T into an output tile, the chunk-end state to the checkpoint (or the final state).  Warp wg has the
        // tensor-memory lanes of its quarter.  The tiles leave by bulk tensor stores, one issuing warp each (a store costs its thread
        // some 200 cycles): warp 1 the output, warps 0 and 2 the halves of the state.
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PREP_REGS));
        const int grp = warp >> 2, wg = warp & 3, gt = tid & 127, mine = grp - PREP;  // this group's chunks: mine, mine + READERS, ...
        const uint32_t tlane = tmem + ((uint32_t)(32 * wg) << 16);
        unsigned char* const stage = sm + AT_STAGE<S, LN> + mine * STAGE_BYTES;
        unsigned char* const epi = sm + AT_LN<S, LN> + (LN ? mine * LN_BYTES : 0);
        float* const ysf = reinterpret_cast<float*>(epi);
        float* const part = reinterpret_cast<float*>(epi + LN_PART);
        uint4 gate = make_uint4(0, 0, 0, 0);
        if (AFF) {  // V^T's rows of M are zeros
            const uint32_t zeros[16] = {};
            for (int s = 0; s < S && wg >= 2; ++s) tmem_st16(tlane + C_V + 16 * s, zeros);
            tmem_st_wait();
            tc_fence_before();
            readers_ready();
        }
        // attn_ln: thread = time step lane % 16 x 8 value channels from i0
        const int t = lane & 15, i0 = 16 * wg + 8 * (lane >> 4);
        if (mine == 0 && lane < STATES) mbar_arrive(&ctrl->full[lane]);
        Place<S> at{mine, 0};
        int buf = mine;
#pragma unroll 1
        for (int c = mine; c < work.n; c += READERS, at.advance(READERS)) {
            const int s = at.i;
            buf = buf + 1 < STATES ? buf + 1 : buf + 1 - STATES;  // chunk c leaves its state in buffer (c + 1) % STATES
            const uint32_t state = tlane + C_S + 64 * buf;
            if (READERS == 2) buf = buf + 1 < STATES ? buf + 1 : buf + 1 - STATES;
            float4 lw0, lw1, lb0, lb1;  // attn_ln: GroupNorm weight and bias of this thread's channels
            if (LN) {
                // The gate of this chunk, ahead of its completion.  (Its scores say that its descriptor is there; waited for after the
                // previous chunk's results have left, since a start state may have to come from another CTA first.)
                mbar_wait<true>(&ctrl->score[s], at.parity, ctrl, p.status);
                const ChunkDesc& d = ctrl->desc[c % RING];
                if (!TAIL || d.c + 1 < nchunks || t < tail) gate = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const IoT*>(p.g) + d.off + (long long)(d.c * L + t) * p.st.t + i0));
                const float* lnp = p.params + d.hi * N + i0;
                lw0 = __ldg(reinterpret_cast<const float4*>(lnp)); lw1 = __ldg(reinterpret_cast<const float4*>(lnp) + 1);
                lb0 = __ldg(reinterpret_cast<const float4*>(lnp + p.H * N)); lb1 = __ldg(reinterpret_cast<const float4*>(lnp + p.H * N) + 1);
            }
            mbar_wait<true>(&ctrl->done[s], at.parity, ctrl, p.status);
            tc_fence_after();
            const ChunkDesc& d = ctrl->desc[c % RING];
            const int cc = d.c;
            const bool last = d.flags & SEG_LAST, ck = p.ckpt && !last;
            float* const fin = !last ? nullptr : AFF ? (wg < 2 ? p.sT : p.sM) : p.sT;
            uint32_t yv[8], x[2][16], vv[LN ? 8 : 1];
            if (!AFF) tmem_ld_frag(tlane + C_XY + 32 * s + 16, yv);
            if (LN) tmem_ld_frag(tlane + C_V + 16 * s, vv);
            if (ck) {
                tmem_ld_frag4(state, x[0]);
                tmem_ld_frag4(state + 32, x[1]);
            }
            tmem_ld_wait();
            if (fin) {
                // final state: exact, straight from registers (32-byte stores: whole sectors of the lane's 256-byte row)
                float* dst = fin + (long long)d.bh * N * N + (AFF ? 32 * (wg & 1) + lane : 16 * wg + (lane & 15)) * N;
#pragma unroll
                for (int qt = 0; qt < 4; ++qt) {
                    uint32_t sv[16];
                    tmem_ld16(state + 16 * qt, sv);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) sv[e] = __float_as_uint(__uint_as_float(sv[e]) * STATE_UNSCALE);  // S = 2^64 S~
                    if (AFF || lane < 16) {
#pragma unroll
                        for (int q8 = 0; q8 < 2; ++q8)
                            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + 16 * qt + 8 * q8), "r"(sv[8 * q8]), "r"(sv[8 * q8 + 1]),
                                         "r"(sv[8 * q8 + 2]), "r"(sv[8 * q8 + 3]), "r"(sv[8 * q8 + 4]), "r"(sv[8 * q8 + 5]), "r"(sv[8 * q8 + 6]), "r"(sv[8 * q8 + 7]) : "memory");
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&ctrl->read[s]);  // the slot may be written again
                mbar_arrive(&ctrl->full[s + STATES < S ? s + STATES : s + STATES - S]);  // and the state buffer, by chunk c + STATES
            }
            if (fin && cc + 1 < nchunks) {  // the rest of this chain is another CTA's: hand the state over
                __threadfence();
                group_bar(grp);
                if (gt == 0) publish_handoff(ws.flags + blockIdx.x);
            }
            if (AFF) continue;
            unsigned char* const ytile = sm + AT_Y<S, LN> + (c & 1) * Y_BYTES;
            // What the previous tiles' stores have read is free after the group's next barrier: the staging tile (and attn_ln's one output
            // tile; attn has two, of which this chunk's was free at the end of the previous one).
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            auto stage_state = [&] {
                // checkpoint state: exact fp32 (the backward's tensor-core products read its upper 19 bits, its carried
                // decay term all of them), staged in the swizzled layout the tensor-map store expects: half h = columns 32h..32h+31,
                // row i at i*128 bytes, its 32-byte unit u at (u ^ (i & 3)).  A half-warp's 8-byte stores cover four rows x 32 bytes: with
                // 32-byte units they fill the 32 banks; with the 16-byte swizzle rows 2i and 2i + 1 met in the same ones (B64 T1024 H12:
                // 372 us with them, 359 us without).
                const int i = 16 * wg + (lane >> 2);  // rows i, i + 8
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            *reinterpret_cast<uint2*>(stage + half * 8192 + (i + 8 * h) * 128 + ((j ^ (i & 3)) << 5) + (lane & 3) * 8) =
                                make_uint2(x[half][4 * j + 2 * h], x[half][4 * j + 2 * h + 1]);
            };
            if (!LN && ck) {
                group_bar(grp);
                stage_state();
            }
            if (!LN) {
                // Y^T [value][time], read as accumulator fragments, goes as bf16 through a transposing matrix store into the
                // [time][value] tile (128-byte rows, 16-byte units XOR-ed with the row as the tensor map's swizzle wants), which
                // leaves by one bulk tensor store; the map clips rows beyond the end of the sequence.
                store_transposed(ytile, yv, wg, lane);
            } else {
                // attn_ln epilogue (reference: wind_rwkv/rwkv7/attn_ln.cu:176-205): GroupNorm over the head's 64
                // value channels of each time step, + bonus dot * v, * gate.  Y^T goes to shared memory as
                // fp32 [time][value]; then one thread = one time step x 8 value channels.
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    ysf[(8 * (i >> 2) + 2 * (lane & 3) + (i & 1)) * LN_YS + 16 * wg + (lane >> 2) + 8 * ((i >> 1) & 1)] = __uint_as_float(yv[i]);
                store_transposed(epi + LN_V, vv, wg, lane);  // (exact: they were bf16)
                group_bar(grp);
                if (ck) stage_state();
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
                float vval[8];
                load8<IoT>(epi + LN_V + t * ROWB + (((i0 >> 3) ^ (t & 7)) << 4), vval);
                group_bar(grp);
                {
                    float a1 = 0.f, a2 = 0.f, bd = 0.f;
#pragma unroll
                    for (int w2 = 0; w2 < 4; ++w2) {
                        const float2 pp = *reinterpret_cast<const float2*>(part + (w2 * L + t) * 2);
                        a1 += pp.x; a2 += pp.y;
                        bd += ctrl->bdot[c % RING][w2][t];
                    }
                    const float md = a1 * (1.f / N);
                    const float mu = pivot + md;
                    const float rstd = rsqrtf(fmaxf(a2 * (1.f / N) - md * md, 0.f) + p.eps);
                    const uint32_t gw[4] = {gate.x, gate.y, gate.z, gate.w};
                    float o8[8];
                    const float lw8[8] = {lw0.x, lw0.y, lw0.z, lw0.w, lw1.x, lw1.y, lw1.z, lw1.w}, lb8[8] = {lb0.x, lb0.y, lb0.z, lb0.w, lb1.x, lb1.y, lb1.z, lb1.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float gv = __uint_as_float(i & 1 ? gw[i / 2] & 0xffff0000u : gw[i / 2] << 16);
                        o8[i] = ((yv8[i] - mu) * rstd * lw8[i] + lb8[i] + bd * vval[i]) * gv;
                    }
                    uint4 pk;
                    pk.x = pack_bf16x2_rn(o8[0], o8[1]); pk.y = pack_bf16x2_rn(o8[2], o8[3]);
                    pk.z = pack_bf16x2_rn(o8[4], o8[5]); pk.w = pack_bf16x2_rn(o8[6], o8[7]);
                    *reinterpret_cast<uint4*>(ytile + t * 128 + (((i0 >> 3) ^ (t & 7)) << 4)) = pk;
                }
            }
            fence_async_smem();
            group_bar(grp);
            if (wg == 1) {
                if (elect_one()) {
                    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                                 ::"l"(&maps.y), "r"(0), "r"(d.hi), "r"(cc * L), "r"(d.bi), "r"(smem_u32(ytile)) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else if (wg != 3 && ck) {
                if (elect_one()) {
                    const int rec_row = (int)(((long long)d.bh * nchunks + cc + 1) * (CK_FLOATS / N));  // a record is 80 rows of 64 floats
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                                 ::"l"(&maps.ck), "r"(16 * wg), "r"(rec_row), "r"(smem_u32(stage + 4096 * wg)) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            __syncwarp();
        }
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory must outlive the last copies
    } else {
        // ------------------------------ preparation groups --------------------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PREP_REGS));
        const int grp = warp >> 2, wg = warp & 3, gt = tid & 127;
        const uint32_t tlane = tmem + ((uint32_t)(32 * wg) << 16);
        // This warp's share of the raw tiles of the chunk at list position v, by bulk tensor loads (16 rows of 128 bytes, 16-byte units XOR-ed with the row;
        // rows beyond the end of the sequence arrive as zeros): a load costs its thread some 200 cycles.
        auto load_raw = [&](int v) {
            if (__any_sync(0xffffffffu, ctrl->abort)) return;  // (the last one's wait may have given up)
            loaded = v;
            if (elect_one()) {
                const ChunkDesc& d = ctrl->desc[v % RING];
                uint64_t* bar = &ctrl->raw[v % RB];
                const int first = AFF ? 1 : 0, i0 = wg == 0 ? 0 : wg == 1 ? 1 : wg == 2 ? 3 : 5, i1 = wg == 0 ? 1 : wg == 1 ? 3 : wg == 2 ? 5 : 6;  // warp 0 has the scores' product to issue, 3 the descriptors
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"((i1 - max(i0, first)) * RAW_TILE) : "memory");
#pragma unroll 1
                for (int i = max(i0, first); i < i1; ++i)
                    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                                 ::"r"(smem_u32(sm + AT_RAW<S, LN> + (v % R) * RAW_BYTES + i * RAW_TILE)), "l"(&maps.in[i]), "r"(smem_u32(bar)), "r"(0), "r"(d.hi), "r"(d.c * L), "r"(d.bi) : "memory");
            }
            __syncwarp();
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
#pragma unroll 1
        for (int v = (grp + R) % PREP; v < R && v < work.n; v += PREP) load_raw(v);
        if (AFF) readers_ready();
        // Iteration at chunk c: write its operand tiles (its scan is in registers) into its slot, start its score product; then scan the
        // group's next chunk while the service warps and the chain work on this one.  (The first iteration only scans: one copy of
        // each piece of code.)
        F2 o[4][2][2], fwv[2];  // [step][channel pair] of wq, wa, kwi, bwi; kwf, bwf are formed from kwi, bwi and fw when the tiles are written
        uint32_t v[4], v2[AFF ? 4 : 1];  // (AFF: values 32 wg + .. and 32 wg + 16 + .., warps 0 and 1)
                                // V^T: values 16 wg + lane / 4 (+ 8) x time steps 2 (lane % 4), + 1; then time steps 8 ..
        Place<S> at{grp, 0};
        Place<RB> rawat{grp, 0};
#pragma unroll 1
        for (int c = grp - PREP; c < work.n; c += PREP) {
            if (c >= 0) {
                const int s = at.i;
                unsigned char* gs = sm + s * G_BYTES;
                if (c >= S) mbar_wait<true>(&ctrl->read[s], at.parity ^ 1, ctrl, p.status);
                at.advance(PREP);
                tc_fence_after();
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
                    if (!AFF || wg < 2) tmem_st_frag(tlane + C_V + 16 * s, vf);
                    if (AFF && wg < 2) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) { vf[2 * i] = v2[AFF ? i : 0] << 16; vf[2 * i + 1] = v2[AFF ? i : 0] & 0xffff0000u; }
                        tmem_st_frag(tlane + (16u << 16) + C_V + 16 * s, vf);
                    }
                    if (!(lane & 8)) {  // the decay blocks' entries, one per lane (see S_CUT): channel j0 + (lane & 3)
                        const F2 p2 = lane & 2 ? fwv[1] : fwv[0];
                        const float pl = (lane & 1 ? p2.y : p2.x) * (STATE_SCALE * (1.f + S_CUT));  // where P_L underflows, so does S~ P_L
                        const uint32_t dither = ((__float_as_uint(o[2][0][0].x) ^ __float_as_uint(o[3][0][0].x)) * 0x9e3779b1u) >> 19;
                        *reinterpret_cast<uint32_t*>(gs + G_DF + quad * 128 + ((quad & 1) * 4 + (lane & 3)) * 16 + (lane & 3) * 4) =
                            (__float_as_uint(pl) + dither) & 0xffffe000u;
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
                if (ctrl->desc[c % RING].flags & SEG_FIRST) load_state(ctrl->desc[c % RING], wg);
                fence_async_smem();
                tc_fence_before();
                __syncwarp();
                // ---------------- the four score matrices as one product, issued by the group's last warp to get here ---------
                if (elect_one()) {
                    uint32_t before;
                    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(smem_u32(&ctrl->tiles[s])) : "memory");
                    if ((before & 3) == 3) {
                        tc_fence_after();
                        fence_async_smem();
                        const uint32_t dA = desc_kmajor(smem_u32(gs + G_WAQ)), dB = desc_kmajor(smem_u32(gs + G_KB));
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks) mma_ss(tmem + C_XY + 32 * s, dA + ks * 16, kmajor(2048), dB + ks * 16, kmajor(2048), idesc(32, false), ks > 0);
                        tc_commit(&ctrl->score[s]);
                    }
                }
                __syncwarp();
            }
            // ---------------- decay scan of the group's next chunk, into registers ---------------------
            // The three transcendentals per element go to the special-function unit: with the matrix products on tcgen05 the FMA
            // pipe and the issue slots are what this kernel runs out of, not MUFU throughput.
            const int n = c + PREP;
            if (n >= work.n) break;
            {
                const unsigned char* const raw0 = sm + AT_RAW<S, LN> + (R == PREP ? grp : n % R) * RAW_BYTES;
                mbar_wait<true>(&ctrl->raw[rawat.i], rawat.parity, ctrl, p.status);
                rawat.advance(PREP);
                if (gt == 127 && n + R < work.n) {  // the descriptor of the chunk whose loads are issued below
                    ChunkDesc d = ctrl->desc[n % RING];
                    d.c += R;
                    if (d.c < d.c_end) {
                        d.flags = d.c + 1 == d.c_end ? SEG_LAST : 0;
                        ctrl->desc[(n + R) % RING] = d;
                    } else {
                        describe(n + R, (n + R) % RING);
                    }
                }
                __syncwarp();
                F2 cum[2][2], q[2][2], kk[2][2], a[2][2], b[2][2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = row0 ^ e;
                    const unsigned char* raw = raw0 + row * ROWB + (((quad >> 1) ^ (row & 7)) << 4) + (quad & 1) * 8;
                    load4f2(raw + 1 * RAW_TILE, cum[e]);
                    if (!AFF) load4f2(raw + 0 * RAW_TILE, q[e]);
                    load4f2(raw + 2 * RAW_TILE, kk[e]);
                    load4f2(raw + 3 * RAW_TILE, a[e]);
                    load4f2(raw + 4 * RAW_TILE, b[e]);
                }
                {
                    const int t = 8 * (lane >> 4) + (lane & 7), unit = (AFF ? 4 * (wg & 1) : 2 * wg) + ((lane >> 3) & 1);
                    const uint32_t at = smem_u32(raw0 + 5 * RAW_TILE + t * ROWB);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at + ((unit ^ (t & 7)) << 4)) : "memory");
                    if (AFF)
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(v2[0]), "=r"(v2[AFF ? 1 : 0]), "=r"(v2[AFF ? 2 : 0]), "=r"(v2[AFF ? 3 : 0]) : "r"(at + (((unit + 2) ^ (t & 7)) << 4)) : "memory");
                }
                if (LN) {  // bonus dot sum_j r_j k_j bonus_j of these time steps: 4 channels here, the rest by shuffle and in the epilogue
                    const float4 bo = __ldg(reinterpret_cast<const float4*>(p.params + (2 * p.H + ctrl->desc[n % RING].hi) * N + j0));
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
                    if (!(lane & 0x14)) *reinterpret_cast<float2*>(&ctrl->bdot[n % RING][wg][row0 & 14]) = make_float2(first, second);
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
                        if (TAIL && ctrl->desc[n % RING].c + 1 == nchunks && (row0 ^ e) >= tail) cum[e][i] = f2(0.f, 0.f);
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
                    // P~_t = 2^64 P_t and its reciprocal (see ANCHOR_LN): both finite, since 16 steps of FLOOR are -178.9 + 64
                    const F2 sa = add2(sum[i], f2(ANCHOR_LOG2, ANCHOR_LOG2));
                    // P~_L = 2^64 P_L (P_L itself may lie below fp32's normal range)
                    const int src = (lane & 0x14) | 11;
                    fwv[i] = f2(ex2_approx(__shfl_sync(0xffffffffu, sa.x, src)), ex2_approx(__shfl_sync(0xffffffffu, sa.y, src)));
                    const F2 c[2] = {fma2(cum[1][i], f2(late0, late0), sa), fma2(cum[0][i], f2(late1, late1), sa)};  // less the later step's, in the earlier one
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const F2 cp = fma2(cum[e][i], f2(-1.f, -1.f), c[e]);  // without this step's own decay
                        const F2 incl = f2(ex2_approx(c[e].x), ex2_approx(c[e].y));
                        const F2 inv = f2(ex2_approx(-c[e].x), ex2_approx(-c[e].y));
                        const F2 non = f2(ex2_approx(cp.x), ex2_approx(cp.y));
                        if (!AFF) o[0][e][i] = rnd2<RND>(mul2(q[e][i], incl));   // wq (rounded here already: writing the tiles is on the way to the chain, this is not)
                        o[1][e][i] = rnd2<RND>(mul2(a[e][i], non));    // wa
                        o[2][e][i] = mul2(kk[e][i], inv);   // kwi
                        o[3][e][i] = mul2(b[e][i], inv);    // bwi
                    }
                }
            }
            group_bar(grp);  // the raw tiles have been read
            if (n + R < work.n) load_raw(n + R);
        }
    }

    if (ctrl->abort && elect_one()) abort_drain(ctrl, warp, loaded, PREP, RB, p.status);
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && ctrl->abort) give_up(&ctrl->abort, p.status);
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

template <int S, bool RND, bool LN, bool TAIL, bool AFF = false> static int launch_tt(const FwdParams& p, cudaStream_t stream) {
    auto kern = wkv7_fwd_tc_kernel<S, RND, LN, TAIL, AFF>;
    constexpr int smem = AT_CTRL<S, LN> + (int)sizeof(Ctrl) + 1024;
    static_assert(smem <= 232448, "shared memory of an SM");
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return kLaunchFailed;
    FwdMaps maps;
    memset(&maps, 0, sizeof(maps));
    if (p.ckpt && !encode_checkpoint_map(&maps.ck, p.ckpt, p.B * p.H * ((p.T + L - 1) / L))) return kLaunchFailed;
    const void* ins[7] = {p.y, p.r, p.w, p.k, p.a, p.b, p.v};
    CUtensorMap* const ms[7] = {&maps.y, &maps.in[0], &maps.in[1], &maps.in[2], &maps.in[3], &maps.in[4], &maps.in[5]};
    for (int i = 0; i < 7; ++i)
        if (ins[i] && !encode_bthn_map(ms[i], const_cast<void*>(ins[i]), p.B, p.T, p.H, p.st)) return kLaunchFailed;
    const WorkSplit ws = plan_work(p.B * p.H, (p.T + L - 1) / L, 1, p.sT ? p.flags : nullptr);
    if (ws.flags && cudaMemsetAsync(ws.flags, 0, ws.ctas * sizeof(unsigned), stream) != cudaSuccess) return kLaunchFailed;
    return launch(kern, dim3((unsigned)ws.ctas), THREADS_TC, smem, stream, p, ws, maps) ? kOk : kLaunchFailed;
}

template <int S, bool RND, bool LN> static int launch_t(const FwdParams& p, cudaStream_t stream) {
    return p.T % L ? launch_tt<S, RND, LN, true>(p, stream) : launch_tt<S, RND, LN, false>(p, stream);
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
    if (tid == 0 && ctrl.abort) give_up(&ctrl.abort, status);  // as the forward does when its CTA ends
}

}  // namespace tc

int launch_bounded_wait_selftest(long long limit_cycles, int* status, long long* cycles, cudaStream_t stream) {
    tc::bounded_wait_selftest_kernel<<<1, 128, 0, stream>>>(limit_cycles, status, cycles);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

// impl as wkv7_set_fwd_impl has it: its size selects attn's slots, its sign whether operands are rounded.  Five slots are the default because
// they are faster at every size: with three / four / five, L2 flushed, B64 T1024 H12 340 / 301 / 283 us, with checkpoints 387 / 371 / 369;
// B8 T8192 H40 1002 / 868 / 809; B3 T1003 H16 72 / 64 / 61.  attn_ln has room for four beside its epilogue's tiles.
int launch_fwd_tc(const FwdParams& p, int impl, bool ln, cudaStream_t stream) {
    if (p.sM) return p.T % L ? tc::launch_tt<5, true, false, true, true>(p, stream) : tc::launch_tt<5, true, false, false, true>(p, stream);
    if (ln) return impl > 0 ? tc::launch_t<4, true, true>(p, stream) : tc::launch_t<4, false, true>(p, stream);
    switch (impl) {
        case 2: return tc::launch_t<3, true, false>(p, stream);
        case 3: return tc::launch_t<4, true, false>(p, stream);
        case 4: return tc::launch_t<5, true, false>(p, stream);
        case -2: return tc::launch_t<3, false, false>(p, stream);
        case -3: return tc::launch_t<4, false, false>(p, stream);
        case -4: return tc::launch_t<5, false, false>(p, stream);
        default: return kBadShape;
    }
}

}  // namespace wkv7
