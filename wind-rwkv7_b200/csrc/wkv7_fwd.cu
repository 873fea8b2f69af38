// WKV7 forward for sm_100a: one CTA per (batch, head) chain, 4 warps, chunks of 16 time steps.
//
// Replaces the reference's forward_kernel (wind_rwkv/rwkv7/attn.cu:11-106) and, with LN = true,
// the fused variant (wind_rwkv/rwkv7/attn_ln.cu:106-212).  Not a translation: the whole
// state-dependent part of a chunk is computed TRANSPOSED (rows = value index), so that warp w
// owns value rows 16w..16w+15 of the state S, of X^T, U^T and Y^T, keeps S in registers across
// chunks as MMA accumulators, feeds accumulators straight back as A operands, and needs no
// cross-warp reduction.  Only the state-independent chunk preparation (decay scan, scaled
// operands, the four masked 16x16 score matrices and the triangular inverse) is shared through
// shared memory.
//
// Per chunk (rows = time, P_t = prod_{s<=t} exp(-exp(w_s)) per key channel, S0 = state at the
// chunk start, S[value][key]):
//     wq = q*P_t     wa = a*P_{t-1}     kwi = k/P_t     bwi = b/P_t     fw = P_L
// (in the code P_t is kept as 2^64 P_t and the state as 2^-64 S, which leaves every formula as it is: see ANCHOR_LN)
//     QK = tril(wq kwi^T)  QB = tril(wq bwi^T)  AK = stril(wa kwi^T)  AB = stril(wa bwi^T)
//     X = AK V + wa S0^T ;  U = (I-AB)^-1 X ;  Y = QK V + QB U + wq S0^T
//     S' = (S0 + V^T kwi + U^T bwi) * fw[None,:]
// Inputs are fetched one chunk ahead with 16-byte cp.async copies issued by all threads.
#include "wkv7_kernels.h"

namespace wkv7 {

template <typename IoT> struct FwdLayout {
    static constexpr int ROWB = N * (int)sizeof(IoT) + 16;  // padded staging row (bytes)
    static constexpr int TILEB = L * ROWB;
    static constexpr int YS = (sizeof(IoT) == 2) ? 24 : 20;  // y scratch row stride (elements)
};

template <typename IoT, bool LN> struct FwdSmem {
    using Lay = FwdLayout<IoT>;
    alignas(16) unsigned char st_in[5][Lay::TILEB];  // q, w, k, a, b of the current chunk
    alignas(16) unsigned char st_v[2][Lay::TILEB];   // v, double buffered (read late in the chunk)
    alignas(16) unsigned char st_g[LN ? 2 : 1][LN ? Lay::TILEB : 16];
    alignas(16) float wq[L * OPS], wa[L * OPS], kwi[L * OPS], bwi[L * OPS];
    alignas(16) float QK[L * SCS], QB[L * SCS], AK[L * SCS], AB[L * SCS], AI[L * SCS];
    alignas(16) float fw[N];
    alignas(16) float lnp[LN ? 3 * N : 4];
    float bdot[L];
    float red[WARPS][L][2];
    alignas(16) IoT ysc[WARPS][L * Lay::YS];
};

template <typename IoT> __device__ __forceinline__ float st_elem(const unsigned char* tile, int row, int col) {
    return to_f32<IoT>(*reinterpret_cast<const IoT*>(tile + row * FwdLayout<IoT>::ROWB + col * (int)sizeof(IoT)));
}

template <typename IoT, int PREC, bool LN>
__global__ void __launch_bounds__(THREADS) wkv7_fwd_kernel(FwdParams p) {
    using Lay = FwdLayout<IoT>;
    using Smem = FwdSmem<IoT, LN>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const long long bh = blockIdx.x;
    const long long bi = bh / p.H, hi = bh % p.H;
    const long long base = bi * p.st.b + hi * p.st.h;
    const int nchunks = (int)((p.T + L - 1) / L);  // the last chunk may be partial: its missing rows read as zeros
    const bool has_tail = (p.T % L) != 0;
    const IoT* gin[5] = {(const IoT*)p.r + base, (const IoT*)p.w + base, (const IoT*)p.k + base,
                         (const IoT*)p.a + base, (const IoT*)p.b + base};
    const IoT* gv = (const IoT*)p.v + base;
    const IoT* gg = LN ? (const IoT*)p.g + base : nullptr;
    IoT* gy = (IoT*)p.y + base;
    constexpr uint32_t ROW_BYTES = N * sizeof(IoT);

    if (LN) {
        for (int i = tid; i < 3 * N; i += THREADS) sm.lnp[i] = p.params[(long long)(i / N) * p.H * N + hi * N + (i % N)];
    }
    __syncthreads();

    // q, w, k, a, b are dead once the scan has run, so the next chunk's copies are issued right
    // after the first barrier of the iteration; v (and g) are read late and double buffered.
    constexpr int CH = ROW_BYTES / 16;
    auto issue_in = [&](int c) {
        for (int i = tid; i < 5 * L * CH; i += THREADS) {
            int ten = i / (L * CH), row = (i / CH) % L, ch = i % CH;
            const long long tt = (long long)c * L + row;
            if (has_tail) cp_async16_zfill(sm.st_in[ten] + row * Lay::ROWB + ch * 16,
                             reinterpret_cast<const unsigned char*>(gin[ten] + (tt < p.T ? tt : p.T - 1) * p.st.t) + ch * 16, tt < p.T);
            else cp_async16(sm.st_in[ten] + row * Lay::ROWB + ch * 16, reinterpret_cast<const unsigned char*>(gin[ten] + tt * p.st.t) + ch * 16);
        }
    };
    auto issue_v = [&](int c) {
        int s = c & 1;
        for (int i = tid; i < (LN ? 2 : 1) * L * CH; i += THREADS) {
            int ten = i / (L * CH), row = (i / CH) % L, ch = i % CH;
            const long long tt = (long long)c * L + row;
            const IoT* src = (ten == 0 ? gv : gg) + (tt < p.T ? tt : p.T - 1) * p.st.t;
            unsigned char* dst = (ten == 0 ? sm.st_v[s] : sm.st_g[LN ? s : 0]) + row * Lay::ROWB;
            if (has_tail) cp_async16_zfill(dst + ch * 16, reinterpret_cast<const unsigned char*>(src) + ch * 16, tt < p.T);
            else cp_async16(dst + ch * 16, reinterpret_cast<const unsigned char*>(src) + ch * 16);
        }
    };
    if (nchunks > 0) {
        issue_in(0);
        issue_v(0);
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncthreads();

    // State: warp owns value rows 16*warp + {g, g+8}; tile nt covers key columns 8nt..8nt+7,
    // thread holds columns 8nt+2*t4, +1.
    float S[8][4];
    {
        const float* s0 = p.s0 ? p.s0 + bh * N * N : nullptr;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            if (s0) {
                float2 lo = *reinterpret_cast<const float2*>(s0 + (16 * warp + g) * N + 8 * nt + 2 * t4);
                float2 hi2 = *reinterpret_cast<const float2*>(s0 + (16 * warp + g + 8) * N + 8 * nt + 2 * t4);
                // the state is carried as S~ = 2^-64 S (see ANCHOR_LN)
                S[nt][0] = lo.x * STATE_SCALE; S[nt][1] = lo.y * STATE_SCALE; S[nt][2] = hi2.x * STATE_SCALE; S[nt][3] = hi2.y * STATE_SCALE;
            } else {
                S[nt][0] = S[nt][1] = S[nt][2] = S[nt][3] = 0.f;
            }
        }
    }

    for (int c = 0; c < nchunks; ++c) {
        // ---------------- P1: decay scan and scaled operands ------------------------------------
        {
            decay_scan<IoT, PREC>(sm.st_in[0], sm.st_in[1], sm.st_in[2], sm.st_in[3], sm.st_in[4], Lay::ROWB, sm.wq, sm.wa,
                                  sm.kwi, sm.bwi, sm.fw, nullptr, nullptr, warp, lane, (int)min((long long)L, p.T - (long long)c * L));
            if (LN) {  // bonus dot  sum_j r_j k_j bonus_j  per time step: 8 threads per row
                const int row = tid >> 3, part = tid & 7;
                float acc = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int ch = part * 8 + i;
                    acc += st_elem<IoT>(sm.st_in[0], row, ch) * st_elem<IoT>(sm.st_in[2], row, ch) * sm.lnp[2 * N + ch];
                }
                acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                acc += __shfl_xor_sync(0xffffffffu, acc, 2);
                acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                if (part == 0) sm.bdot[row] = acc;
            }
        }
        __syncthreads();  // (A)
        if (c + 1 < nchunks) {
            issue_in(c + 1);
            issue_v(c + 1);
        }
        cp_async_commit();
        // ---------------- P2: masked score matrices, one per warp ------------------------------
        {
            const float* Am = (warp & 1) ? sm.wa : sm.wq;
            const float* Bm = (warp >> 1) ? sm.bwi : sm.kwi;
            float* dst = warp == 0 ? sm.QK : warp == 1 ? sm.AK : warp == 2 ? sm.QB : sm.AB;
            const bool strict = warp & 1;
            float d[2][4] = {};
#pragma unroll 2
            for (int kk = 0; kk < 8; ++kk) {
                FragA<PREC> a = fragA_mk<PREC, true>(Am, OPS, 0, 8 * kk, g, t4);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) mma<PREC>(d[nt], a, fragB_nk<PREC, true>(Bm, OPS, 8 * nt, 8 * kk, g, t4));
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int s = 8 * nt + 2 * t4;
                auto keep = [&](int tq, int ss) { return strict ? ss < tq : ss <= tq; };
                // AB only feeds the inverse and stays unrounded; the other three are MMA operands
                auto val = [&](float x) { return warp == 3 ? x : pre<PREC>(x); };
                float2 lo = make_float2(keep(g, s) ? val(d[nt][0]) : 0.f, keep(g, s + 1) ? val(d[nt][1]) : 0.f);
                float2 hi2 = make_float2(keep(g + 8, s) ? val(d[nt][2]) : 0.f, keep(g + 8, s + 1) ? val(d[nt][3]) : 0.f);
                if (warp == 3) {  // AB is kept transposed for the inverse
                    dst[s * SCS + g] = lo.x; dst[(s + 1) * SCS + g] = lo.y;
                    dst[s * SCS + g + 8] = hi2.x; dst[(s + 1) * SCS + g + 8] = hi2.y;
                } else {
                    *reinterpret_cast<float2*>(dst + g * SCS + s) = lo;
                    *reinterpret_cast<float2*>(dst + (g + 8) * SCS + s) = hi2;
                }
            }
        }
        // ---------------- P3: AI = (I - AB)^-1 by forward substitution (the warp that made AB) --
        if (warp == 3) {
            __syncwarp();
            if (lane < L) tri_inverse_column<PREC>(sm.AB, sm.AI, lane);
        }
        // ---------------- chain, part 1: needs only S and the scaled operands ------------------
        if (p.ckpt) {
            float* ck = p.ckpt + (bh * nchunks + c) * (long long)CK_FLOATS;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                // exact fp32: in the single-TF32 class the backward's tensor-core products read the upper 19 bits without a
                // conversion, and its carried decay term uses the full value
                *reinterpret_cast<float2*>(ck + (16 * warp + g) * N + 8 * nt + 2 * t4) = make_float2(S[nt][0], S[nt][1]);
                *reinterpret_cast<float2*>(ck + (16 * warp + g + 8) * N + 8 * nt + 2 * t4) = make_float2(S[nt][2], S[nt][3]);
            }
        }
        float XY[4][4] = {};  // [0..1] X^T (time blocks 0,1), [2..3] Y^T
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            FragA<PREC> a = fragA_from_acc<PREC>(S[kk]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
                mma<PREC>(XY[nt], a, fragB_nk<PREC, true>(nt < 2 ? sm.wa : sm.wq, OPS, 8 * (nt & 1), 8 * kk, g, t4));
        }
        __syncthreads();  // (B) scores and AI visible
        if (p.ckpt) {  // the chunk's four 16x16 matrices go into the checkpoint record: 8 floats per thread
            float* ck = p.ckpt + (bh * nchunks + c) * (long long)CK_FLOATS;
            const int m = tid >> 5, r = (tid & 31) >> 1, hf = tid & 1;
            float x[8];
            if (m == 3) {  // AI goes out transposed
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = sm.AI[(8 * hf + i) * SCS + r];
            } else {
                const float* src = (m == 0 ? sm.QK : m == 1 ? sm.QB : sm.AK) + r * SCS + 8 * hf;
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = src[i];
            }
            float* dst = ck + (m == 0 ? CK_SC + ck_tile_at(16 + r, 2 * hf) : m == 1 ? CK_QB + ck_tile_at(r, 2 * hf)
                                                                            : m == 2 ? CK_SC + ck_tile_at(r, 2 * hf) : CK_AI + ck_tile_at(r, 2 * hf));
            *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4*>(dst + 32) = make_float4(x[4], x[5], x[6], x[7]);
        }

        // ---------------- chain, part 2 ----------------------------------------------------------
        const unsigned char* vt = sm.st_v[c & 1];
        FragA<PREC> vf[2];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            const int tr = 8 * kk + 2 * t4, vc = 16 * warp + g;
            constexpr bool EXACT = sizeof(IoT) == 2;  // a bf16 value is a TF32 value
            vf[kk].x[0].template put<EXACT>(st_elem<IoT>(vt, tr, vc));
            vf[kk].x[1].template put<EXACT>(st_elem<IoT>(vt, tr, vc + 8));
            vf[kk].x[2].template put<EXACT>(st_elem<IoT>(vt, tr + 1, vc));
            vf[kk].x[3].template put<EXACT>(st_elem<IoT>(vt, tr + 1, vc + 8));
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int kk = 0; kk <= nt; ++kk) {
                mma<PREC>(XY[nt], vf[kk], fragB_nk<PREC, true>(sm.AK, SCS, 8 * nt, 8 * kk, g, t4));
                mma<PREC>(XY[2 + nt], vf[kk], fragB_nk<PREC, true>(sm.QK, SCS, 8 * nt, 8 * kk, g, t4));
            }
        float U[2][4] = {};
        {
            FragA<PREC> xa[2] = {fragA_from_acc<PREC>(XY[0]), fragA_from_acc<PREC>(XY[1])};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) mma<PREC>(U[nt], xa[kk], fragB_nk<PREC, true>(sm.AI, SCS, 8 * nt, 8 * kk, g, t4));
        }
        FragA<PREC> ua[2] = {fragA_from_acc<PREC>(U[0]), fragA_from_acc<PREC>(U[1])};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int kk = 0; kk <= nt; ++kk) mma<PREC>(XY[2 + nt], ua[kk], fragB_nk<PREC, true>(sm.QB, SCS, 8 * nt, 8 * kk, g, t4));

        // ---------------- output -----------------------------------------------------------------
        if (LN) {
            // GroupNorm over the head's 64 value channels of each time step: per-warp mean and
            // centred sum of squares over 16 rows, merged across warps (Chan's formula).
            float mean_w[4], m2_w[4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float s = XY[2 + nt][e] + XY[2 + nt][e + 2];
                    s += __shfl_xor_sync(0xffffffffu, s, 4);
                    s += __shfl_xor_sync(0xffffffffu, s, 8);
                    s += __shfl_xor_sync(0xffffffffu, s, 16);
                    const float mu = s * (1.f / 16.f);
                    const float d0 = XY[2 + nt][e] - mu, d1 = XY[2 + nt][e + 2] - mu;
                    float q = d0 * d0 + d1 * d1;
                    q += __shfl_xor_sync(0xffffffffu, q, 4);
                    q += __shfl_xor_sync(0xffffffffu, q, 8);
                    q += __shfl_xor_sync(0xffffffffu, q, 16);
                    mean_w[2 * nt + e] = mu;
                    m2_w[2 * nt + e] = q;
                }
            if (g == 0)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int tq = 8 * (i >> 1) + 2 * t4 + (i & 1);
                    sm.red[warp][tq][0] = mean_w[i];
                    sm.red[warp][tq][1] = m2_w[i];
                }
            __syncthreads();  // (D)
            const unsigned char* gt = sm.st_g[c & 1];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int nt = i >> 1, e = i & 1, tq = 8 * nt + 2 * t4 + e;
                float mu = 0.f, m2 = 0.f;
#pragma unroll
                for (int w2 = 0; w2 < WARPS; ++w2) mu += sm.red[w2][tq][0];
                mu *= 0.25f;
#pragma unroll
                for (int w2 = 0; w2 < WARPS; ++w2) {
                    const float dm = sm.red[w2][tq][0] - mu;
                    m2 += sm.red[w2][tq][1] + 16.f * dm * dm;
                }
                const float rstd = 1.f / sqrtf(m2 * (1.f / N) + p.eps);
                const float bd = sm.bdot[tq];
#pragma unroll
                for (int hrow = 0; hrow < 2; ++hrow) {
                    const int vc = 16 * warp + g + 8 * hrow;
                    float y = XY[2 + nt][e + 2 * hrow];
                    y = (y - mu) * rstd * sm.lnp[vc] + sm.lnp[N + vc] + bd * st_elem<IoT>(vt, tq, vc);
                    XY[2 + nt][e + 2 * hrow] = y * st_elem<IoT>(gt, tq, vc);
                }
            }
        }
        {
            IoT* sc = sm.ysc[warp];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int tq = 8 * nt + 2 * t4;
                sc[tq * Lay::YS + g] = from_f32<IoT>(XY[2 + nt][0]);
                sc[(tq + 1) * Lay::YS + g] = from_f32<IoT>(XY[2 + nt][1]);
                sc[tq * Lay::YS + g + 8] = from_f32<IoT>(XY[2 + nt][2]);
                sc[(tq + 1) * Lay::YS + g + 8] = from_f32<IoT>(XY[2 + nt][3]);
            }
            __syncwarp();
            const int row = lane >> 1, hf = lane & 1;
            const uint4* src = reinterpret_cast<const uint4*>(sc + row * Lay::YS + 8 * hf);
            uint4* dst = reinterpret_cast<uint4*>(gy + ((long long)c * L + row) * p.st.t + 16 * warp + 8 * hf);
            if ((long long)c * L + row < p.T) {
                dst[0] = src[0];
                if (sizeof(IoT) == 4) dst[1] = src[1];
            }
        }
        // ---------------- state update -----------------------------------------------------------
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                mma<PREC>(S[nt], vf[kk], fragB_kn<PREC, true>(sm.kwi, OPS, 8 * nt, 8 * kk, g, t4));
                mma<PREC>(S[nt], ua[kk], fragB_kn<PREC, true>(sm.bwi, OPS, 8 * nt, 8 * kk, g, t4));
            }
            const float2 f = *reinterpret_cast<const float2*>(sm.fw + 8 * nt + 2 * t4);  // P~_L = 2^64 P_L
            S[nt][0] = S[nt][0] * f.x * STATE_SCALE; S[nt][1] = S[nt][1] * f.y * STATE_SCALE;
            S[nt][2] = S[nt][2] * f.x * STATE_SCALE; S[nt][3] = S[nt][3] * f.y * STATE_SCALE;
        }
        cp_async_wait<0>();
        __syncthreads();  // (E) operand and score buffers are free again
    }

    if (p.sT) {
        float* sT = p.sT + bh * N * N;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            *reinterpret_cast<float2*>(sT + (16 * warp + g) * N + 8 * nt + 2 * t4) = make_float2(S[nt][0] * STATE_UNSCALE, S[nt][1] * STATE_UNSCALE);
            *reinterpret_cast<float2*>(sT + (16 * warp + g + 8) * N + 8 * nt + 2 * t4) = make_float2(S[nt][2] * STATE_UNSCALE, S[nt][3] * STATE_UNSCALE);
        }
    }
}

// ---- fp32 tensors, attn: the chain apart from what does not need the state --------------------------------------------------------------
// One CTA per chain, the mathematics of wkv7_fwd_kernel<float, 3>.  Four chain warps (16 value rows each, no exchange between them) do the
// products that the state goes through; PREP32 groups of four warps take a chunk each: fetch, scan, operands split into their two TF32
// parts (once, not at each use), the four score matrices, the inverse, the record's matrices.  SLOTS32 chunks in flight.
// Bound by the chain's products, 230 of 8 cycles a warp and chunk, and their dependences: 4900 cycles a chunk (all in one set of warps: 8900).
constexpr int SLOTS32 = 3, PREP32 = 3, THREADS32 = THREADS * (1 + PREP32);
constexpr int ROW32 = N * 4 + 16, TILE32 = L * ROW32;  // staging tiles [time][channel]
struct Fwd32Slot {
    alignas(16) unsigned char v[TILE32];
    alignas(16) float op[4][2][L * OPS];  // wq, wa, kwi, bwi: upper and lower part, column swizzle xcol<1>
    alignas(16) float QK[L * SCS], QB[L * SCS], AK[L * SCS], AB[L * SCS], AI[L * SCS];
    alignas(16) float fw[N];
};
struct Fwd32Smem {
    alignas(16) unsigned char raw[PREP32][5][TILE32];  // q, w, k, a, b
    Fwd32Slot slot[SLOTS32];
    uint64_t ready[SLOTS32], free[SLOTS32];
    volatile int abort;
};
static_assert(sizeof(Fwd32Smem) <= 232448, "one CTA per SM");

template <bool TAIL>
__global__ void __launch_bounds__(THREADS32, 1) wkv7_fwd32_kernel(FwdParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Fwd32Smem& sm = *reinterpret_cast<Fwd32Smem*>(smem_raw);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, t4 = lane & 3, w = warp & 3;
    const int bh = blockIdx.x, bi = bh / (int)p.H, hi = bh - bi * (int)p.H, nchunks = (int)((p.T + L - 1) / L);
    const long long base = bi * p.st.b + hi * p.st.h;
    if (tid == 0) {
        for (int i = 0; i < SLOTS32; ++i) {
            mbar_init(&sm.ready[i], WARPS);
            mbar_init(&sm.free[i], WARPS);
        }
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int bg = (g >> 2) & 1, bt = (t4 >> 1) & 1;  // element offsets under xcol<1> (pitch 72): row g, columns 8 kk + 2 t4, +1 | rows 2 t4 (, + 1), column 8 nb + g
    const int mkE = g * OPS + 2 * t4 + 8 * bg, mkO = mkE - 16 * bg, knE = 2 * t4 * OPS + g + 8 * bt, knO = knE - 16 * bt;
    auto mk = [&](int kk) { return (kk & 1 ? mkO : mkE) + 8 * kk; };
    auto kn = [&](int nb) { return (nb & 1 ? knO : knE) + 8 * nb; };
    auto put = [](auto& x, float h, float l) { x.h = __float_as_uint(h); x.l = __float_as_uint(l); };
    auto B_nk = [&](const float (&op)[2][L * OPS], int nt, int kk) {
        const float* q = op[0] + 8 * nt * OPS + mk(kk);
        const float2 h = *reinterpret_cast<const float2*>(q), l = *reinterpret_cast<const float2*>(q + L * OPS);
        FragB<3> f;
        put(f.x[0], h.x, l.x); put(f.x[1], h.y, l.y);
        return f;
    };
    // d += a b, the products with a lower part apart: the sums over the keys are what the chain waits for
    auto mma_split = [](float (&d)[4], float (&d2)[4], const FragA<3>& a, const FragB<3>& b) {
        mma_tf32_raw(d2, a.x[0].l, a.x[1].l, a.x[2].l, a.x[3].l, b.x[0].h, b.x[1].h);
        mma_tf32_raw(d, a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].h, b.x[1].h);
        mma_tf32_raw(d2, a.x[0].h, a.x[1].h, a.x[2].h, a.x[3].h, b.x[0].l, b.x[1].l);
    };

    if (warp >= WARPS) {
        // ---- preparation: group `grp` takes every PREP32-th chunk
        const int grp = warp / WARPS - 1, gt = tid & (THREADS - 1);
        const float* in[6] = {(const float*)p.r + base, (const float*)p.w + base, (const float*)p.k + base, (const float*)p.a + base, (const float*)p.b + base, (const float*)p.v + base};
        const int prow = gt / (N / 4), pch = 4 * (gt % (N / 4));  // a thread's 16-byte pieces: rows prow, prow + 8
        auto piece = [&](unsigned char* tile, const float* src, int c, int row) {  // rows beyond the sequence as zeros
            const long long tt = (long long)c * L + row;
            if (TAIL) cp_async16_zfill(tile + row * ROW32 + 4 * pch, src + pch + (tt < p.T ? tt : p.T - 1) * p.st.t, tt < p.T);
            else cp_async16(tile + row * ROW32 + 4 * pch, src + pch + tt * p.st.t);
        };
        auto fetch = [&](int c) {
#pragma unroll
            for (int ten = 0; ten < 5; ++ten)
#pragma unroll
                for (int r = prow; r < L; r += 8) piece(sm.raw[grp][ten], in[ten], c, r);
        };
        auto group_bar = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory"); };
        const int row = lane & 15, j0 = 16 * w + 8 * (lane >> 4), at = row * OPS + xcol<1>(row, j0), off = row * ROW32 + 4 * j0;
        const bool flip = (row >> 2) & 1;
        auto split = [&](float (&op)[2][L * OPS], const float (&x)[8]) {
            float h[8], l[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                h[i] = __uint_as_float(tf32_rna(x[i]));
                l[i] = __uint_as_float(tf32_rna(x[i] - h[i]));
            }
            store8(op[0] + at, h, flip);
            store8(op[1] + at, l, flip);
        };
        if (grp < nchunks) fetch(grp);
        for (int c = grp; c < nchunks; c += PREP32) {
            Fwd32Slot& t = sm.slot[c % SLOTS32];
            if (c >= SLOTS32) mbar_wait_bounded<true>(&sm.free[c % SLOTS32], (c / SLOTS32 - 1) & 1, &sm.abort, p.status);
#pragma unroll
            for (int r = prow; r < L; r += 8) piece(t.v, in[5], c, r);
            cp_async_commit();
            cp_async_wait<0>();
            group_bar();  // everyone's pieces have landed
            {   // the scan of decay_scan()
                const unsigned char (*raw)[TILE32] = sm.raw[grp];
                float lw[8], cum[8], x[8], o[8];
                load8<float>(raw[1] + off, lw);
                const int live = TAIL ? (int)min((long long)L, p.T - (long long)c * L) : L;
#pragma unroll
                for (int i = 0; i < 8; ++i) cum[i] = lw[i] = row < live ? fmaxf(-exp_p<3>(lw[i]), MIN_STEP_LOG_DECAY) : 0.f;
#pragma unroll
                for (int d = 1; d < 16; d <<= 1)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float up = __shfl_up_sync(0xffffffffu, cum[i], d, 16);
                        if (row >= d) cum[i] += up;
                    }
                load8<float>(raw[3] + off, x);
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
                for (int i = 0; i < 8; ++i) { o[i] = x[i] * cum[i]; cum[i] = rcp_p<3>(cum[i]); }
                split(t.op[0], o);
                load8<float>(raw[2] + off, x);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = x[i] * cum[i];
                split(t.op[2], o);
                load8<float>(raw[4] + off, x);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = x[i] * cum[i];
                split(t.op[3], o);
            }
            group_bar();  // operands visible, the raw tiles have been read
            if (c + PREP32 < nchunks) fetch(c + PREP32);
            {   // a score matrix per warp: QK, AK, QB, AB
                const float (&A)[2][L * OPS] = t.op[w & 1], (&B)[2][L * OPS] = t.op[2 + (w >> 1)];
                float* dst = w == 0 ? t.QK : w == 1 ? t.AK : w == 2 ? t.QB : t.AB;
                const bool strict = w & 1;
                float d[2][4] = {}, d2[2][4] = {};
#pragma unroll 2
                for (int kk = 0; kk < 8; ++kk) {
                    const float* q = A[0] + mk(kk);
                    FragA<3> a;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {  // rows g, g + 8
                        const float2 u = *reinterpret_cast<const float2*>(q + 8 * h * OPS), l = *reinterpret_cast<const float2*>(q + (8 * h + L) * OPS);
                        put(a.x[h], u.x, l.x); put(a.x[2 + h], u.y, l.y);
                    }
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma_split(d[nt], d2[nt], a, B_nk(B, nt, kk));
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int s = 8 * nt + 2 * t4, tq = g + 8 * h;
                        const float x = (strict ? s < tq : s <= tq) ? d[nt][2 * h] + d2[nt][2 * h] : 0.f;
                        const float y = (strict ? s + 1 < tq : s + 1 <= tq) ? d[nt][2 * h + 1] + d2[nt][2 * h + 1] : 0.f;
                        if (w == 3) {  // AB is kept transposed for the inverse
                            dst[s * SCS + tq] = x; dst[(s + 1) * SCS + tq] = y;
                        } else {
                            *reinterpret_cast<float2*>(dst + tq * SCS + s) = make_float2(x, y);
                        }
                    }
            }
            if (w == 3) {
                __syncwarp();
                if (lane < L) tri_inverse_column<3>(t.AB, t.AI, lane);
            }
            if (p.ckpt) {  // the chunk's four 16x16 matrices go into the checkpoint record: 8 floats per thread
                group_bar();
                float* ck = p.ckpt + ((long long)bh * nchunks + c) * CK_FLOATS;
                const int m = gt >> 5, r = (gt & 31) >> 1, hf = gt & 1;
                float x[8];
                if (m == 3) {  // AI goes out transposed
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = t.AI[(8 * hf + i) * SCS + r];
                } else {
                    const float* src = (m == 0 ? t.QK : m == 1 ? t.QB : t.AK) + r * SCS + 8 * hf;
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = src[i];
                }
                float* dst = ck + (m == 0 ? CK_SC + ck_tile_at(16 + r, 2 * hf) : m == 1 ? CK_QB + ck_tile_at(r, 2 * hf)
                                                                                : m == 2 ? CK_SC + ck_tile_at(r, 2 * hf) : CK_AI + ck_tile_at(r, 2 * hf));
                *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(dst + 32) = make_float4(x[4], x[5], x[6], x[7]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.ready[c % SLOTS32]);
        }
        cp_async_wait<0>();
        return;
    }
    // ---- the chain: value rows 16 w + {g, g + 8} of S, carried as S~ = 2^-64 S (see ANCHOR_LN); tile nt covers key columns 8 nt ..
    float S[8][4];
    const long long st = (long long)bh * N * N + (16 * w + g) * N + 2 * t4;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const float2 lo = p.s0 ? *reinterpret_cast<const float2*>(p.s0 + st + 8 * nt) : make_float2(0.f, 0.f);
        const float2 hi2 = p.s0 ? *reinterpret_cast<const float2*>(p.s0 + st + 8 * N + 8 * nt) : make_float2(0.f, 0.f);
        S[nt][0] = lo.x * STATE_SCALE; S[nt][1] = lo.y * STATE_SCALE; S[nt][2] = hi2.x * STATE_SCALE; S[nt][3] = hi2.y * STATE_SCALE;
    }
    float* gy = (float*)p.y + base + 16 * w + g;
    for (int c = 0; c < nchunks; ++c) {
        const int s = c % SLOTS32;
        const Fwd32Slot& t = sm.slot[s];
        if (p.ckpt) {
            float* ck = p.ckpt + ((long long)bh * nchunks + c) * CK_FLOATS + (16 * w + g) * N + 2 * t4;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                *reinterpret_cast<float2*>(ck + 8 * nt) = make_float2(S[nt][0], S[nt][1]);
                *reinterpret_cast<float2*>(ck + 8 * N + 8 * nt) = make_float2(S[nt][2], S[nt][3]);
            }
        }
        mbar_wait_bounded<false>(&sm.ready[s], (c / SLOTS32) & 1, &sm.abort, p.status);
        FragA<3> vf[2];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            const float* q = reinterpret_cast<const float*>(t.v + (8 * kk + 2 * t4) * ROW32) + 16 * w + g;
            vf[kk].x[0].set(q[0]); vf[kk].x[1].set(q[8]); vf[kk].x[2].set(q[ROW32 / 4]); vf[kk].x[3].set(q[ROW32 / 4 + 8]);
        }
        float XY[4][4] = {}, small[4][4] = {};  // [0..1] X^T (time blocks 0, 1), [2..3] Y^T
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const FragA<3> a = fragA_from_acc<3>(S[kk]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) mma_split(XY[nt], small[nt], a, B_nk(t.op[nt < 2 ? 1 : 0], nt & 1, kk));
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int kk = 0; kk <= nt; ++kk) {
                mma_split(XY[nt], small[nt], vf[kk], fragB_nk<3, true>(t.AK, SCS, 8 * nt, 8 * kk, g, t4));
                mma_split(XY[2 + nt], small[2 + nt], vf[kk], fragB_nk<3, true>(t.QK, SCS, 8 * nt, 8 * kk, g, t4));
            }
#pragma unroll
        for (int i = 0; i < 16; ++i) XY[i >> 2][i & 3] += small[i >> 2][i & 3];
        float U[2][4] = {};
        {
            const FragA<3> xa[2] = {fragA_from_acc<3>(XY[0]), fragA_from_acc<3>(XY[1])};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int kk = 0; kk <= nt; ++kk) mma<3>(U[nt], xa[kk], fragB_nk<3, true>(t.AI, SCS, 8 * nt, 8 * kk, g, t4));
        }
        const FragA<3> ua[2] = {fragA_from_acc<3>(U[0]), fragA_from_acc<3>(U[1])};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int kk = 0; kk <= nt; ++kk) mma<3>(XY[2 + nt], ua[kk], fragB_nk<3, true>(t.QB, SCS, 8 * nt, 8 * kk, g, t4));
        // ---- state update
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                for (int o = 2; o < 4; ++o) {
                    const float *q = t.op[o][0] + 8 * kk * OPS + kn(nt), *l = q + L * OPS;
                    FragB<3> b;
                    put(b.x[0], q[0], l[0]); put(b.x[1], q[OPS], l[OPS]);
                    mma<3>(S[nt], o == 2 ? vf[kk] : ua[kk], b);
                }
            const float2 f = *reinterpret_cast<const float2*>(t.fw + 8 * nt + 2 * t4);  // P~_L = 2^64 P_L
            S[nt][0] = S[nt][0] * f.x * STATE_SCALE; S[nt][1] = S[nt][1] * f.y * STATE_SCALE;
            S[nt][2] = S[nt][2] * f.x * STATE_SCALE; S[nt][3] = S[nt][3] * f.y * STATE_SCALE;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.free[s]);
        // ---- output: whole sectors of eight values
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const long long row = (long long)c * L + 8 * nt + 2 * t4 + e;
                if (!TAIL || row < p.T) { gy[row * p.st.t] = XY[2 + nt][e]; gy[row * p.st.t + 8] = XY[2 + nt][e + 2]; }
            }
    }
    if (p.sT) {
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            *reinterpret_cast<float2*>(p.sT + st + 8 * nt) = make_float2(S[nt][0] * STATE_UNSCALE, S[nt][1] * STATE_UNSCALE);
            *reinterpret_cast<float2*>(p.sT + st + 8 * N + 8 * nt) = make_float2(S[nt][2] * STATE_UNSCALE, S[nt][3] * STATE_UNSCALE);
        }
    }
}

static int launch_fwd32(const FwdParams& p, cudaStream_t stream) {
    auto kern = p.T % L ? wkv7_fwd32_kernel<true> : wkv7_fwd32_kernel<false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Fwd32Smem)) != cudaSuccess) return kLaunchFailed;
    kern<<<(unsigned)(p.B * p.H), THREADS32, sizeof(Fwd32Smem), stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

template <typename IoT, int PREC, bool LN> static int launch_fwd_t(const FwdParams& p, cudaStream_t stream) {
    using Smem = FwdSmem<IoT, LN>;
    auto kern = wkv7_fwd_kernel<IoT, PREC, LN>;
    const int smem = (int)sizeof(Smem);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return kLaunchFailed;
    kern<<<(unsigned)(p.B * p.H), THREADS, smem, stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? kOk : kLaunchFailed;
}

int launch_fwd(const FwdParams& p, int io_dtype, bool ln, cudaStream_t stream) {
    if (io_dtype == 0) return ln ? launch_fwd_t<__nv_bfloat16, 1, true>(p, stream) : launch_fwd_t<__nv_bfloat16, 1, false>(p, stream);
    if (io_dtype == 2) return ln ? launch_fwd_t<float, 1, true>(p, stream) : launch_fwd_t<float, 1, false>(p, stream);
    // Up to a CTA per SM the chain's own warps win (8 x 12 chains of 32 chunks 159 -> 93 us, 8 of 256 1196 -> 667); a second round of CTAs pays
    // for long chains (156 of 32: 209 -> 187), not for short ones, where wkv7_fwd_kernel's three CTAs an SM do (300 of 7: 69, here 72; 768 of
    // 4: 80, here 91).
    const long long chains = p.B * p.H, sms = sm_count();
    if (!ln && (chains <= sms || (chains <= 2 * sms && p.T > 31 * L))) return launch_fwd32(p, stream);
    return ln ? launch_fwd_t<float, 3, true>(p, stream) : launch_fwd_t<float, 3, false>(p, stream);
}

}  // namespace wkv7
