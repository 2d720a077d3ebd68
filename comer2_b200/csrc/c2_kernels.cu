// c2_kernels.cu -- phase-1 (fused score matrix + Viterbi DP) and DP
// finalisation kernels for sm_100a.
//
// Phase 1 replaces the reference's CalcSM_Init_SMEMUnroll2x +
// CalcSM_SSSS_CVS2S_SMEMUnroll2x_2 (src/libmycu/cusco/) and the per-diagonal
// ExecDP_Btck_Unroll32x launches (src/libmycu/cudp/CuBatchDP.cu:149-320,
// CuBatchDP_init_btck.cu:65-494).  Instead of materialising the L_q x N score
// matrix and a traceback byte per cell in HBM, one persistent warp sweeps
// a strip of 64 query rows of one (query, db profile) pair at a time, two rows to
// a lane, in chunks of 8 db columns:
//  * the chunk's scores go to a ring in shared memory: from FP32 dot products
//    against db records staged by cp.async (p1c_kernel), or from split-BF16
//    tensor-core products of packed db tiles fetched by cp.async.bulk with
//    query operands held in tensor memory (p1t_kernel);
//  * the DP then runs 8 steps of an anti-diagonal wavefront: lane t processes
//    column k - t of rows 2 t, 2 t + 1 at step k, the "up" states of its first row
//    coming from lane t - 1 by __shfl_up_sync, the "diagonal" states being the
//    step before's "up", the columns' transitions from a shared-memory ring;
//  * the strip's last row is handed to the next strip through a boundary
//    buffer (global memory, L2 resident), the warp's own or, for the longest
//    pairs of a search, whose strips several warps take, the pair's.
// p1_kernel (one row a lane, a column a step) serves the allocation-free entry.
// For the pairs that pass the phase-1 threshold, p2s_kernel stores the FP32
// scores column-major for the finalisation, statistics and MAP stages, and the
// traceback sweep (p1tc_kernel) runs the same DP on them again, storing btck
// codes.
#include <cuda_bf16.h>

#include <algorithm>

#include "c2_device.cuh"

namespace c2 {

#define FULL 0xffffffffu

__device__ __forceinline__ int corner_edge(int lq, int ld)
{
    // GetCornerMaxlen, src/libmycu/cudp/CuBatchDP_init_btck.cuh:118-127
    int m = lq > ld ? lq : ld;
    int e = (int)rintf(0.34f * (float)m);
    return e > 60 ? 60 : e;
}

__device__ __forceinline__ bool in_corner(int lq, int ld, int e, int y, int x)
{
    // CellYXinCorners, src/libmycu/cudp/CuBatchDP_init_btck.cuh:129-145
    return (lq <= y + e && x <= e + y - lq) || (ld - e + y <= x && y < e);
}

// Score of (own query row, db column) -- src/libmycu/cusco/CuBatchScoreMatrix_Init.cu:129-182,
// _ssss.cuh:48-131, _cvs2s.cuh:47-136.  The aa term uses the per-pair row
// factors Qt[a] = q(a) / (0.5 (bq(a) + bd(a))); the SS term uses the per-row
// table U[c] = sum_s p_q(s) T[idx_q(s)][c].
// The two dot products run in packed pairs of FP32 (fma.rn.f32x2: two IEEE
// multiply-adds per instruction, the two accumulators of each chain).  NR rows
// share the record's reads.
struct RowOps {
    unsigned long long Qt[NAA / 2];        // pairs (2 i, 2 i + 1)
    unsigned long long qcv[(NCV + 1) / 2]; // the last entry's partner is 0
    float cq, pq, hq;
};

__device__ __forceinline__ unsigned long long pack2(float x, float y)
{
    return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float lo2(unsigned long long a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(unsigned long long a) { return __uint_as_float((unsigned)(a >> 32)); }

// query row qr against a profile with background bd
__device__ __forceinline__ void row_ops(RowOps& R, const float* __restrict__ qr, const float* __restrict__ qbkg,
                                        const float* __restrict__ bd)
{
#pragma unroll
    for (int i = 0; i < NAA; i += 2)
        R.Qt[i / 2] = pack2(__fdividef(qr[QR_TRG + i], 0.5f * (qbkg[i] + bd[i])),
                            __fdividef(qr[QR_TRG + i + 1], 0.5f * (qbkg[i + 1] + bd[i + 1])));
#pragma unroll
    for (int i = 0; i < NCV; i += 2) R.qcv[i / 2] = pack2(qr[QR_CV + i], i + 1 < NCV ? qr[QR_CV + i + 1] : 0.f);
    R.cq = qr[QR_CN];
    R.pq = qr[QR_PRIOR];
    R.hq = qr[QR_HQ];
}

// hardware base-2 logarithm, denormal inputs flushed (the arguments here, an
// amino-acid odds sum and a CV determinant, are far above the denormal range)
constexpr float C2_LN2 = 0.693147180559945309f;
__device__ __forceinline__ float lg2_ftz(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Scores of NR consecutive rows; the SS row table U has USTR floats a column,
// the lane's first row at U[urow].  cvtab holds each CV map value CVREP times
// ([cvcard][CVREP]); a lane reads replica lane % CVREP so that lanes reading
// different entries rarely share a bank.  CVUNIF: the table's key range
// coincides with its index clamp (TcConsts).
template <int CVREP, int NR, int USTR, bool CVUNIF>
__device__ __forceinline__ void cell_scores(const RowOps* R, const float* __restrict__ rec,
                                            const float* __restrict__ U, int urow, const float* __restrict__ cvtab,
                                            const ScoreConsts& sc, int lane, float* S, float* mod_out)
{
    const ulonglong2* rp = reinterpret_cast<const ulonglong2*>(rec);
    unsigned long long s[NR], dot[NR];
#pragma unroll
    for (int e = 0; e < NR; e++) s[e] = dot[e] = 0ull;
    // aa term (two accumulators shorten the dependent FMA chain)
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const ulonglong2 v = rp[i];
#pragma unroll
        for (int e = 0; e < NR; e++) s[e] = fma2(R[e].Qt[2 * i + 1], v.y, fma2(R[e].Qt[2 * i], v.x, s[e]));
    }
    // CV term: dot product over [20,39) (39, the CV norm, meets a 0), then
    // (cq)(cd) - (dot+1/kappa0)^2
    float cd = 0.f;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const ulonglong2 v = rp[5 + i];
#pragma unroll
        for (int e = 0; e < NR; e++) dot[e] = fma2(R[e].qcv[2 * i + 1], v.y, fma2(R[e].qcv[2 * i], v.x, dot[e]));
        if (i == 4) cd = hi2(v.y);   // DR_CN = 39
    }
    const float4 v10 = *reinterpret_cast<const float4*>(rec + DR_PRIOR);   // 40 prior, 41..43 ss
    const float2 v11 = *reinterpret_cast<const float2*>(rec + DR_SSIDX);   // 44 ss idx, 45 hd
    const int pk = __float_as_int(v11.x);
    const float* __restrict__ u0 = U + (pk & 0xff) * USTR + urow;
    const float* __restrict__ u1 = U + ((pk >> 8) & 0xff) * USTR + urow;
    const float* __restrict__ u2 = U + ((pk >> 16) & 0xff) * USTR + urow;
    float w[3][NR];
    if (NR == 2) {
        const float2 a = *reinterpret_cast<const float2*>(u0), b = *reinterpret_cast<const float2*>(u1),
                     c = *reinterpret_cast<const float2*>(u2);
        w[0][0] = a.x; w[0][NR - 1] = a.y; w[1][0] = b.x; w[1][NR - 1] = b.y; w[2][0] = c.x; w[2][NR - 1] = c.y;
    } else {
        w[0][0] = *u0; w[1][0] = *u1; w[2][0] = *u2;
    }
#pragma unroll
    for (int e = 0; e < NR; e++) {
        const float s0 = lg2_ftz(lo2(s[e]) + hi2(s[e])) * C2_LN2 - sc.shift;
        const float dt = (lo2(dot[e]) + hi2(dot[e])) + sc.lokappa0;
        const float det = R[e].cq * cd - dt * dt;
        const float cvs = sc.cterm + sc.pownu0 * (lg2_ftz(det) * C2_LN2) - R[e].pq - v10.x;
        // the clamp keeps the shared-memory read in bounds for any table and argument;
        // from above before the shift is added, since the conversion saturates (a
        // determinant of 0 makes the score +inf, and 2^31 - 1 + shift is negative)
        const int ix = max(min(__float2int_rn(2.f * cvs), sc.cvhi) + sc.cvshift, 0);
        float cvm = cvtab[ix * CVREP + (lane & (CVREP - 1))];
        if (!CVUNIF) {
            cvm = (sc.cvkey_last <= cvs) ? sc.cvval_last : cvm;
            cvm = (cvs <= sc.cvkey_first) ? sc.cvval_first : cvm;
        }
        // SS term
        float ss = v10.y * w[0][e];
        ss = fmaf(v10.z, w[1][e], ss);
        ss = fmaf(v10.w, w[2][e], ss);
        if (-99.f < ss) {
            ss += R[e].hq * v11.y * 0.1111111f;
            ss -= 0.05f;
            ss *= sc.ssswgt;
        }
        const float add = fmaf(cvm, sc.cvswgt, ss);
        mod_out[e] = add - 0.5f * sc.cvswgt;   // modular score of the MAP stage
        S[e] = s0 + add;
    }
}

struct St5 { float MM, MI, IM, DN, ND; };

// Stage the records of columns [REC_CHUNK*m, REC_CHUNK*(m+1)) (clipped to L)
// into ring slots; records of consecutive columns are contiguous in HBM, so a
// chunk is one contiguous range copied by all lanes in 16-byte pieces.  The
// caller commits the group (possibly empty, so that wait_group counts stay aligned).
__device__ __forceinline__ void stage_chunk(float* rec, const float* __restrict__ dr, int m, int L, int lane)
{
    const int c0 = m * REC_CHUNK;
    const int nc = min(REC_CHUNK, L - c0);
    if (nc > 0) {
        const int n16 = nc * (DR_STRIDE / 4);
        float* dst = rec + (c0 & (REC_SLOTS - 1)) * DR_STRIDE;
        const float* src = dr + (long long)c0 * DR_STRIDE;
        for (int i = lane; i < n16; i += 32) cp_async16(dst + 4 * i, src + 4 * i);
    }
}

// Transitions of the columns of chunk m (8 columns) from their records into
// the column ring (slots from cs on; the chunk at slot 0 also into the mirror
// slots after the last chunk)
__device__ __forceinline__ void stage_trn(float* cring, const float* __restrict__ dr, int m, int cs, int L, int lane)
{
    const int c = P1_C * m + (lane >> 1);
    if (lane < 2 * P1_C && c < L) {
        const float* src = dr + (long long)c * DR_STRIDE + DR_TRN + 4 * (lane & 1);
        float* dst = cring + (cs + (lane >> 1)) * P1C_TRS + 4 * (lane & 1);
        cp_async16(dst, src);
        if (cs == 0) cp_async16(dst + P1_CMOD * P1C_TRS, src);
    }
}

__global__ void __launch_bounds__(P1_WARPS * 32, 2)
p1_kernel(P1Args a, const float* __restrict__ qbkg)
{
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int cvcard = a.sc.cvcard;
    const int card = a.sc.ssss_card;
    float* cvtab = smem;                                      // [cvcard][32]
    float* wb = smem + cvcard * 32 + wid * P1_WARP_FLOATS;
    float* ring = wb;                                         // [32][32]
    float* U = wb + 32 * 32;                                  // [card][32]
    float* rec = U + MAX_SSSS_CARD * 32;                      // [REC_SLOTS][DR_STRIDE] db records
    for (int i = threadIdx.x; i < cvcard * 32; i += blockDim.x) cvtab[i] = a.cvvals[i >> 5];
    __syncthreads();

    const long long slot = (long long)blockIdx.x * P1_WARPS + wid;
    const int Lmax = (int)(a.botstride / 10);
    float* bot0 = a.bot + slot * a.botstride;
    const int Lq = a.Lq;
    const int nstrips = (Lq + 31) >> 5;
    const ScoreConsts sc = a.sc;

    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.counter, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= a.nwork) break;
        const int p = a.order[item];
        const int L = a.plen[p];
        const long long off = a.poff[p];
        const float* __restrict__ dr = a.drec + off * DR_STRIDE;
        const float* __restrict__ bd = a.pbkg + (long long)p * NAA;
        const int edge = corner_edge(Lq, L);
        float best = 0.f;
        int brow = 0x7fffffff, bcol = 0x7fffffff;
        float* botr = bot0;
        float* botw = bot0 + 5 * Lmax;

        for (int s = 0; s < nstrips; s++) {
            const int r = s * 32 + lane;
            const bool act = r < Lq;
            const float* __restrict__ qr = a.qrec + (long long)(act ? r : Lq - 1) * QR_STRIDE;
            RowOps R;
            row_ops(R, qr, qbkg, bd);
            {
                // this strip's SS row tables (built once per query, c2_set_query)
                const float* __restrict__ us = a.qU + (long long)s * MAX_SSSS_CARD * 32 + lane;
#pragma unroll 8
                for (int c = 0; c < card; c++) U[c * 32 + lane] = __ldg(us + c * 32);
            }
            float q7[7];
#pragma unroll
            for (int i = 0; i < 7; i++) q7[i] = act ? qr[QR_TRN + i] : LOG0;
            // column -1 boundary states of this row and of the row above
            const bool z_left = (lane == 31);
            const bool z_diag = (lane == 31 || lane == 0);
            const St5 LB = z_left ? St5{0.f, 0.f, 0.f, 0.f, 0.f}
                                  : St5{0.f, qr[QR_C + 0], qr[QR_C + 1], qr[QR_C + 2], LOG0};
            const St5 DB = z_diag ? St5{0.f, 0.f, 0.f, 0.f, 0.f}
                                  : St5{0.f, qr[QR_CP + 0], qr[QR_CP + 1], qr[QR_CP + 2], LOG0};
            __syncwarp();

            St5 mine = {0.f, 0.f, 0.f, 0.f, 0.f};
            St5 upp = {0.f, 0.f, 0.f, 0.f, 0.f};
            float t7[7];
#pragma unroll
            for (int i = 0; i < 7; i++) t7[i] = LOG0;
            // strip-boundary prefetch: lane i holds column c0 + i of the row above
            float bcur[5], bnxt[5];
#pragma unroll
            for (int f = 0; f < 5; f++) {
                bcur[f] = 0.f;
                bnxt[f] = 0.f;
                if (s > 0) {
                    if (lane < L) bcur[f] = botr[f * Lmax + lane];
                    if (32 + lane < L) bnxt[f] = botr[f * Lmax + 32 + lane];
                }
            }
            const bool wr_bot = (lane == 31) && (s + 1 < nstrips);
            const int nsteps = L + 31;
            // db column records are staged into shared memory one chunk ahead
            stage_chunk(rec, dr, 0, L, lane);
            cp_async_commit();
            stage_chunk(rec, dr, 1, L, lane);
            cp_async_commit();
            for (int k = 0; k < nsteps; k++) {
                if ((k & (REC_CHUNK - 1)) == 0 && k < L) {
                    cp_async_wait_1();
                    __syncwarp();
                }
                // ---- score stage: column k for every lane's row
                float tc[7];
                if (k < L) {
                    const float4* rp = reinterpret_cast<const float4*>(rec + (k & (REC_SLOTS - 1)) * DR_STRIDE);
                    float mod, S;
                    cell_scores<32, 1, 32, false>(&R, reinterpret_cast<const float*>(rp), U, lane, cvtab, sc, lane, &S, &mod);
                    if (!act) S = -9.f;
                    ring[(k & 31) * 32 + lane] = S;
                    const float4 ta = rp[12], tb = rp[13];
                    tc[0] = ta.x; tc[1] = ta.y; tc[2] = ta.z; tc[3] = ta.w;
                    tc[4] = tb.x; tc[5] = tb.y; tc[6] = tb.z;
                    if ((k & (REC_CHUNK - 1)) == REC_CHUNK - 1) {
                        // chunk fully read by every lane: refill its slots two chunks ahead
                        __syncwarp();
                        stage_chunk(rec, dr, (k >> REC_CHUNK_LOG) + 2, L, lane);
                        cp_async_commit();
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 7; i++) tc[i] = LOG0;
                }
                // ---- DP stage: column j = k - lane
#pragma unroll
                for (int i = 0; i < 7; i++) {
                    const float x = __shfl_up_sync(FULL, t7[i], 1);
                    t7[i] = (lane == 0) ? tc[i] : x;
                }
                St5 up;
                up.MM = __shfl_up_sync(FULL, mine.MM, 1);
                up.MI = __shfl_up_sync(FULL, mine.MI, 1);
                up.IM = __shfl_up_sync(FULL, mine.IM, 1);
                up.DN = __shfl_up_sync(FULL, mine.DN, 1);
                up.ND = __shfl_up_sync(FULL, mine.ND, 1);
                {
                    const int src = k & 31;
                    const float b0 = __shfl_sync(FULL, bcur[0], src);
                    const float b1 = __shfl_sync(FULL, bcur[1], src);
                    const float b2 = __shfl_sync(FULL, bcur[2], src);
                    const float b3 = __shfl_sync(FULL, bcur[3], src);
                    const float b4 = __shfl_sync(FULL, bcur[4], src);
                    if (lane == 0) up = St5{b0, b1, b2, b3, b4};
                    if (src == 31) {
#pragma unroll
                        for (int f = 0; f < 5; f++) {
                            bcur[f] = bnxt[f];
                            const int c = k + 33 + lane;
                            bnxt[f] = (s > 0 && c < L) ? botr[f * Lmax + c] : 0.f;
                        }
                    }
                }
                const int j = k - lane;
                St5 left = mine, diag = upp;
                if (j == 0) { left = LB; diag = DB; }
                float S = -9.f;
                if (j >= 0 && j < L) {
                    S = ring[(j & 31) * 32 + lane];
                    if (in_corner(Lq, L, edge, r, j)) S = -9.f;
                }
                St5 nw;
                {
                    float v = fmaxf((diag.MI + q7[TMM]) + t7[TIM], (diag.IM + q7[TIM]) + t7[TMM]);
                    v = fmaxf(v, (diag.DN + q7[TDM]) + t7[TMM]);
                    v = fmaxf(v, (diag.ND + q7[TMM]) + t7[TDM]);
                    v = fmaxf(v, (diag.MM + q7[TMM]) + t7[TMM]);
                    nw.MM = fmaxf(v + S, 0.f);
                    nw.MI = fmaxf((up.MM + q7[TMM]) + t7[TMI], (up.MI + q7[TMM]) + t7[TII]);
                    nw.IM = fmaxf((left.MM + q7[TMI]) + t7[TMM], (left.IM + q7[TII]) + t7[TMM]);
                    nw.DN = fmaxf(up.MM + q7[TMD], up.DN + q7[TDD]);
                    nw.ND = fmaxf(left.MM + t7[TMD], left.ND + t7[TDD]);
                }
                const bool valid = act && j >= 0 && j < L;
                if (valid && nw.MM > best) { best = nw.MM; brow = r; bcol = j; }
                if (wr_bot && j >= 0 && j < L) {
                    botw[0 * Lmax + j] = nw.MM;
                    botw[1 * Lmax + j] = nw.MI;
                    botw[2 * Lmax + j] = nw.IM;
                    botw[3 * Lmax + j] = nw.DN;
                    botw[4 * Lmax + j] = nw.ND;
                }
                mine = nw;
                upp = up;
            }
            cp_async_wait_all();
            float* t = botr; botr = botw; botw = t;
            __syncwarp();
        }
        // warp arg-max: largest score, then smallest row, then smallest column
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const float ob = __shfl_xor_sync(FULL, best, o);
            const int orr = __shfl_xor_sync(FULL, brow, o);
            const int oc = __shfl_xor_sync(FULL, bcol, o);
            if (ob > best || (ob == best && (orr < brow || (orr == brow && oc < bcol)))) {
                best = ob; brow = orr; bcol = oc;
            }
        }
        if (lane == 0) {
            const unsigned xy = (best > 0.f) ? (((unsigned)bcol << 16) | ((unsigned)brow & 0xffffu)) : 0u;
            a.best[p] = best;
            a.coords[p] = xy;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Phase 1, chunked: the arithmetic of p1_kernel, scheduled in chunks of 8 db
// columns and strips of 64 query rows, two to a lane.  Per chunk the scores go
// to a shared-memory ring, then the warp advances the anti-diagonal wavefront by
// 8 steps.  Lane t holds rows 2 t and 2 t + 1 of the strip and processes column
// k - t at step k.
//
// The score ring is indexed by anti-diagonal: the scores of rows 2 t, 2 t + 1 at
// column j sit in slot (t + j) mod 40, so at step k every lane reads slot k mod
// 40 and a DP stage reads 8 consecutive slots from one base.

// Maximum of three (sm_100 three-input max.f32; exact, like two fmaxf)
__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// One lane of the wavefront DP.  Every Viterbi candidate of the reference's
// recurrence is (state + query transition) + db transition, evaluated in that
// order, with the sums that two candidates or two steps share computed once.
// Rounding to nearest is monotone, so max(a + t, b + t) = max(a, b) + t holds
// for the rounded sums as well: the candidates that share a db transition are
// reduced before it is added, with the same bits (18 adds and 7 maxima a cell
// instead of 21 and 7).
//   A = max(up.MM + qMM, up.IM + qIM, up.DN + qDM)     (db transition MM)
//   Y = up.MI + qMM    z = up.ND + qMM                 (IM; DM)
// are the up-sums of this step and the diagonal sums of the next (the diagonal
// predecessor of a cell is the up-neighbour of its left one).
struct WfLane {
    float MM, MI, IM, DN, ND;     // own state at the previous step (left)
    float A, Y, z;                // up-sums of the previous step
    float qMM, qDM, qIM, qMD, qDD, qMI, qII;
    float AB, YB, zB;             // diagonal sums of the column -1 boundary state
    float lbMM, lbIM, lbND;       // and the column -1 left state
    float best;
    int kbest;
};

__device__ __forceinline__ void wf_init(WfLane& D, const float* q7, const St5& LB, const St5& DB)
{
    D.qMM = q7[TMM]; D.qDM = q7[TDM]; D.qIM = q7[TIM];
    D.qMD = q7[TMD]; D.qDD = q7[TDD];
    D.qMI = q7[TMI]; D.qII = q7[TII];
    D.AB = max3f(DB.MM + D.qMM, DB.IM + D.qIM, DB.DN + D.qDM);
    D.YB = DB.MI + D.qMM;
    D.zB = DB.ND + D.qMM;
    D.lbMM = LB.MM;
    D.lbIM = LB.IM;
    D.lbND = LB.ND;
    D.MM = D.MI = D.IM = D.DN = D.ND = 0.f;
    D.A = D.Y = D.z = 0.f;
    D.best = 0.f;
    D.kbest = 0;
}

// Wavefront steps [k0, k0 + nst) of a strip of the traceback sweep (k0 a multiple
// of TB_C, nst <= TB_C; TB_C when !CHECK).  ring: diagonal-indexed scores, 32
// floats per slot.  tcol: ring of P1C_RING column records (TMM .. TDD, P1C_TRS
// floats apart).  bnd: row above the strip for columns [k0, k0 + TB_C).  Lane 31
// stores its cells to the strip's row (wr_row).  Each cell's traceback code goes
// to the warp's column ring btr (column j in slot j & 31, the lane's own row),
// and column k - 31, complete for every row at step k, is stored to the pair's
// code matrix bt (column-major, Lq rows; r = this lane's query row).
template <bool CHECK>
__device__ __forceinline__ void wf_steps(WfLane& D, int k0, int nst, int lane, int L, bool act,
                                         const float* __restrict__ ring, const float* __restrict__ tcol,
                                         const float* __restrict__ bnd, bool wr_row, float* row, int ldr,
                                         signed char (*btr)[33], signed char* __restrict__ bt, int Lq, int r)
{
    const float* __restrict__ rb = ring + (k0 & (P1C_RING - 1)) * 32 + lane;
    if (!CHECK) nst = TB_C;
    int ub = -1;
    // the instruction cache holds both variants of both kernels at these depths
    constexpr int UNR = CHECK ? 2 : 4;
#pragma unroll UNR
    for (int u = 0; u < nst; u++) {
        const float S = rb[u * 32];
        const float* __restrict__ tp = tcol + ((k0 + u - lane) & (P1C_RING - 1)) * P1C_TRS;
        const float4 ta = *reinterpret_cast<const float4*>(tp);       // MM MI MD IM
        const float4 tb = *reinterpret_cast<const float4*>(tp + 4);   // II DM DD
        float uMM = __shfl_up_sync(FULL, D.MM, 1);
        float uMI = __shfl_up_sync(FULL, D.MI, 1);
        float uIM = __shfl_up_sync(FULL, D.IM, 1);
        float uDN = __shfl_up_sync(FULL, D.DN, 1);
        float uND = __shfl_up_sync(FULL, D.ND, 1);
        {
            // row above the strip at column k (lane 0's column), broadcast reads
            const float4 ba = *reinterpret_cast<const float4*>(bnd + u * 4);
            const float b4 = bnd[4 * TB_C + u];
            if (lane == 0) { uMM = ba.x; uMI = ba.y; uIM = ba.z; uDN = ba.w; uND = b4; }
        }
        const int j = k0 + u - lane;
        float Ad = D.A, Yd = D.Y, zd = D.z, lMM = D.MM, lIM = D.IM, lND = D.ND;
        if (CHECK && j == 0) {
            Ad = D.AB; Yd = D.YB; zd = D.zB;
            lMM = D.lbMM; lIM = D.lbIM; lND = D.lbND;
        }
        const float X = uMM + D.qMM, Y = uMI + D.qMM, z = uND + D.qMM;
        const float A = max3f(X, uIM + D.qIM, uDN + D.qDM);
        const float v = max3f(Ad + ta.x, Yd + ta.w, zd + tb.y);
        const float nMM = fmaxf(v + S, 0.f);
        const float nMI = fmaxf(X + ta.y, Y + tb.x);
        const float nIM = fmaxf(lMM + D.qMI, lIM + D.qII) + ta.x;
        const float nDN = fmaxf(uMM + D.qMD, uDN + D.qDD);
        const float nND = fmaxf(lMM + ta.z, lND + tb.z);
        // inactive lanes (rows past the query) carry LOG0 query transitions:
        // their MM stays 0 and never beats a maximum
        const bool inm = !CHECK || (j >= 0 && j < L);
        if ((!CHECK || act) && inm && nMM > D.best) { D.best = nMM; ub = u; }
        // ExecDP_Btck's code: DIAG if MM > 0, then the first strictly larger
        // of MI (UP), IM (LEFT), DN (UP), ND (LEFT)
        if (act && inm) {
            int b = BT_STOP;
            float mx = nMM;
            if (nMM != 0.f) b = BT_DIAG;
            if (mx < nMI) { mx = nMI; b = BT_UP; }
            if (mx < nIM) { mx = nIM; b = BT_LEFT; }
            if (mx < nDN) { mx = nDN; b = BT_UP; }
            if (mx < nND) b = BT_LEFT;
            btr[j & 31][lane] = (signed char)b;
        }
        const int cfl = k0 + u - 31;
        if (act && (!CHECK || (cfl >= 0 && cfl < L))) bt[(long long)cfl * Lq + r] = btr[cfl & 31][lane];
        if (wr_row && (!CHECK || (j >= 0 && j < L))) row_put(row, ldr, j, nMM, nMI, nIM, nDN, nND);
        D.MM = nMM; D.MI = nMI; D.IM = nIM; D.DN = nDN; D.ND = nND;
        D.A = A; D.Y = Y; D.z = z;
    }
    if (ub >= 0) D.kbest = k0 + ub;
}

// Corner cells (CellYXinCorners): row r keeps S = -9 at columns j <= cA(r)
// and j >= cB(r).
__device__ __forceinline__ int corner_a(int r, int Lq, int edge) { return (Lq <= r + edge) ? edge + r - Lq : -1; }
__device__ __forceinline__ int corner_b(int r, int L, int edge) { return (r < edge) ? L - edge + r : 0x7fffffff; }

// Phase-1 work items.  A pair is swept by one warp, strip after strip, with
// the rows between the strips in the warp's own boundary buffer -- except the
// nsplit longest pairs, whose strips are items of their own (any warp may take
// them): those hand the rows on through per-pair buffers with published
// progress (pipe_wait, c2_device.cuh).  Without that a search
// with few pairs, or with pairs much longer than the mean, ends in a tail where
// a few warps walk all strips of a long pair alone: 1 x 1,237 against 4,999
// profiles took 16.3 ms, the time of its longest pair (39 strips x 2,031 steps).
// Which pairs are split: split_pairs (c2_host.cu).
// Order: strip 0 of all split pairs, then strip 1 and so on, then the whole
// pairs, all from one counter: strip s is taken after strip s - 1, by a running
// warp, and the whole pairs, the shortest last, even out the end.  (Warps that
// look whether the next strip is ready and exchange the counter only then,
// taking a whole pair otherwise, serialise on the counter: 5 times slower on
// 10,000 items.)
struct P1Item {
    int p, L;        // profile, its length
    int s0, s1;      // strips [s0, s1)
    int pi;          // split pair (index in the longest-first order), -1: whole pair
};

__device__ __forceinline__ bool p1_take(const P1Args& a, int nstrips, int lane, P1Item& it)
{
    int item = 0;
    if (lane == 0) item = atomicAdd(a.counter, 1);
    item = __shfl_sync(FULL, item, 0);
    const int nsi = a.nsplit * nstrips;
    int code = item - nsi + a.nsplit, strip = -1;   // index in the longest-first order; strip (-1: all)
    if (item < nsi) {
        strip = item / a.nsplit;
        code = item - strip * a.nsplit;
    } else if (code >= a.nwork) {
        return false;
    }
    it.p = a.order[code];
    it.L = a.plen[it.p];
    it.pi = strip < 0 ? -1 : code;
    it.s0 = strip < 0 ? 0 : strip;
    it.s1 = strip < 0 ? nstrips : strip + 1;
    return true;
}

// The rows between the strips of a pair, in the layout of the shared-memory
// row: states MM MI IM DN per column, then the ND values from 4 ldb on; ldb a
// multiple of 4 columns, the buffer 16-byte aligned.  Each half is thus one wide
// store or asynchronous copy per chunk.

// Wait (split pairs only) until columns [c0, c0 + P1_C) of the row above strip s
// are there; false: no such row
__device__ __forceinline__ bool p1_row_ready(const P1Args& a, const P1Item& it, int s, int c0, int lane, bool& broken)
{
    const bool have = s > 0 && c0 < it.L;
    if (have && it.pi >= 0)
        pipe_wait(a.sprog + (long long)(s - 1) * a.nsplit + it.pi, min(c0 + P1_C, it.L), lane, a.status, broken, a.spin);
    return have;
}

// The row above strip s, columns [c0, c0 + P1_C), into the warp's shared row by
// asynchronous copies through L2 (a split pair's row comes from another SM);
// zeros where there is none.  Commits one group.  Columns past the matrix hold
// whatever the buffer does: no cell inside the matrix reads them.
__device__ __forceinline__ void p1_row_async(const P1Args& a, const P1Item& it, int s, float* bnd,
                                             const float* __restrict__ botr, int ldb, int c0, int lane, bool& broken)
{
    if (p1_row_ready(a, it, s, c0, lane, broken)) {
        const int c = c0 + lane, c4 = c0 + 4 * (lane - P1_C);
        if (lane < P1_C) {
            if (c < it.L) cp_async16(bnd + 4 * lane, botr + 4 * c);
        } else if (lane < P1_C + P1_C / 4 && c4 < it.L) {
            cp_async16(bnd + 4 * P1_C + 4 * (lane - P1_C), botr + 4 * ldb + c4);
        }
    } else if (lane < P1_C) {
        *reinterpret_cast<float4*>(bnd + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);
        bnd[4 * P1_C + lane] = 0.f;
    }
    cp_async_commit();
}

// The strip's last row after a DP stage over [k0, k0 + P1_C): slot l of own holds
// lane 31's states at column k0 - 31 + l
__device__ __forceinline__ void p1_row_flush(const float* __restrict__ own, float* __restrict__ botw, int ldb, int k0,
                                             int L, int lane)
{
    const int c = k0 - 31 + lane;
    if (lane < P1_C && c >= 0 && c < L) {
        reinterpret_cast<float4*>(botw)[c] = *reinterpret_cast<const float4*>(own + lane * 4);
        botw[4 * ldb + c] = own[4 * P1_C + lane];
    }
}

// Strip s of a split pair has stored the columns [0, n) of its last row
__device__ __forceinline__ void p1_publish(const P1Args& a, const P1Item& it, int s, int n, int lane)
{
    __syncwarp();   // every lane's stores before lane 0's release
    if (lane == 0) pipe_st_release(a.sprog + (long long)s * a.nsplit + it.pi, n);
}

// The item's maximum over its lanes (largest score, then smallest row, then
// smallest column) to the pair's result.  Strips of a split pair combine theirs
// as a 64-bit key (score bits, complement of the cell); the strip that
// completes the pair writes the result.
__device__ __forceinline__ void p1_result(const P1Args& a, const P1Item& it, int nstrips, int lane, float b, int row,
                                          int col)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const float ob = __shfl_xor_sync(FULL, b, o);
        const int orr = __shfl_xor_sync(FULL, row, o);
        const int oc = __shfl_xor_sync(FULL, col, o);
        if (ob > b || (ob == b && (orr < row || (orr == row && oc < col)))) {
            b = ob; row = orr; col = oc;
        }
    }
    if (lane == 0) {
        bool wr = true;
        if (it.pi >= 0) {
            const unsigned cell = ((unsigned)row << 16) | ((unsigned)col & 0xffffu);
            if (b > 0.f)
                atomicMax(a.skey + it.pi,
                          ((unsigned long long)__float_as_uint(b) << 32) | (unsigned long long)(0xffffffffu - cell));
            __threadfence();
            wr = atomicAdd(a.sdone + it.pi, 1) == nstrips - 1;
            if (wr) {
                __threadfence();
                const unsigned long long key = atomicMax(a.skey + it.pi, 0ull);
                const unsigned c = 0xffffffffu - (unsigned)(key & 0xffffffffu);
                b = __uint_as_float((unsigned)(key >> 32));
                row = (int)(c >> 16);
                col = (int)(c & 0xffffu);
            }
        }
        if (wr) {
            a.best[it.p] = b;
            a.coords[it.p] = (b > 0.f) ? (((unsigned)col << 16) | ((unsigned)row & 0xffffu)) : 0u;
        }
    }
    __syncwarp();
}

// One lane of the wavefront DP with two query rows (2 t and 2 t + 1 of the
// strip): row 0 takes its "up" states from row 1 of lane t - 1 by shuffle, row
// 1 from row 0 of this lane at the same step.  Against one row a lane
// (WfLane), a step's shuffles, record reads and row-above selects serve two
// cells, and its two chains overlap; each cell's arithmetic is the same.
struct Wf2 {
    float MM[2], MI[2], IM[2], DN[2], ND[2];   // states at the previous step (left)
    float A[2], Y[2], z[2];                    // up-sums of the previous step (WfLane)
    float qMM[2], qDM[2], qIM[2], qMD[2], qDD[2], qMI[2], qII[2];
    float best;      // the lane's maximum, its row (0, 1) and step
    int brow, kbest;
};

// Diagonal sums and left states of column -1 for the lane's two rows
struct Wf2Edge {
    float A[2], Y[2], z[2], IM[2], ND[2];
};

__device__ __forceinline__ void wf2_init(Wf2& D, const float* __restrict__ qrec, int r0, int Lq)
{
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int r = r0 + e;
        const bool act = r < Lq;
        // rows past the query carry LOG0 transitions and -inf scores: their MM stays 0
        const float* qr = qrec + (long long)(act ? r : Lq - 1) * QR_STRIDE + QR_TRN;
        D.qMM[e] = act ? qr[TMM] : LOG0; D.qMI[e] = act ? qr[TMI] : LOG0; D.qMD[e] = act ? qr[TMD] : LOG0;
        D.qIM[e] = act ? qr[TIM] : LOG0; D.qII[e] = act ? qr[TII] : LOG0; D.qDM[e] = act ? qr[TDM] : LOG0;
        D.qDD[e] = act ? qr[TDD] : LOG0;
        D.MM[e] = D.MI[e] = D.IM[e] = D.DN[e] = D.ND[e] = 0.f;
        D.A[e] = D.Y[e] = D.z[e] = 0.f;
    }
    D.best = 0.f;
    D.brow = D.kbest = 0;
}

__device__ __forceinline__ void wf2_edge(Wf2Edge& E, const Wf2& D, const float* __restrict__ qrec, int r0, int Lq)
{
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int r = r0 + e, b = r & 31;
        const float* qr = qrec + (long long)min(r, Lq - 1) * QR_STRIDE;
        const bool zl = b == 31, zd = b == 31 || b == 0;
        E.IM[e] = zl ? 0.f : qr[QR_C + 1];
        E.ND[e] = zl ? 0.f : LOG0;
        const float dMI = zd ? 0.f : qr[QR_CP + 0], dIM = zd ? 0.f : qr[QR_CP + 1], dDN = zd ? 0.f : qr[QR_CP + 2];
        const float dND = zd ? 0.f : LOG0;
        E.A[e] = max3f(0.f + D.qMM[e], dIM + D.qIM[e], dDN + D.qDM[e]);
        E.Y[e] = dMI + D.qMM[e];
        E.z[e] = dND + D.qMM[e];
    }
}

// Four wavefront steps: rp the lane's scores (P1_RLD floats a step), tc its
// column records, bnd the row above (slots u0..) and P1_BND on the strip's own, j0 the lane's column at
// the first step, k0 that step.  HEAD: column 0 may be among the steps (steps
// below 32 of a strip).  Cells outside the matrix have scores of
// -inf, so their MM stays 0, and their other states reach no cell inside.
template <bool HEAD>
__device__ __forceinline__ void wf2_steps4(Wf2& D, const Wf2Edge& E, const float* __restrict__ rp,
                                           const float* __restrict__ tc, float* __restrict__ bnd, int u0, int j0, int k0,
                                           int lane, bool wr_bot)
{
    float m[2][4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const float2 S = *reinterpret_cast<const float2*>(rp + u * P1_RLD);
        const float4 ta = *reinterpret_cast<const float4*>(tc + u * P1C_TRS);       // MM MI MD IM
        const float4 tb = *reinterpret_cast<const float4*>(tc + u * P1C_TRS + 4);   // II DM DD
        float uMM = __shfl_up_sync(FULL, D.MM[1], 1);
        float uMI = __shfl_up_sync(FULL, D.MI[1], 1);
        float uIM = __shfl_up_sync(FULL, D.IM[1], 1);
        float uDN = __shfl_up_sync(FULL, D.DN[1], 1);
        float uND = __shfl_up_sync(FULL, D.ND[1], 1);
        {
            const float4 ba = *reinterpret_cast<const float4*>(bnd + 4 * (u0 + u));
            const float b4 = bnd[4 * P1_C + u0 + u];
            if (lane == 0) { uMM = ba.x; uMI = ba.y; uIM = ba.z; uDN = ba.w; uND = b4; }
        }
        const bool first = HEAD && j0 + u == 0;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float Ad = D.A[e], Yd = D.Y[e], zd = D.z[e], lMM = D.MM[e], lIM = D.IM[e], lND = D.ND[e];
            if (first) { Ad = E.A[e]; Yd = E.Y[e]; zd = E.z[e]; lMM = 0.f; lIM = E.IM[e]; lND = E.ND[e]; }
            const float X = uMM + D.qMM[e], Y = uMI + D.qMM[e];
            D.A[e] = max3f(X, uIM + D.qIM[e], uDN + D.qDM[e]);
            D.Y[e] = Y;
            D.z[e] = uND + D.qMM[e];
            const float v = max3f(Ad + ta.x, Yd + ta.w, zd + tb.y);
            const float nMM = fmaxf(v + (e ? S.y : S.x), 0.f);
            const float nMI = fmaxf(X + ta.y, Y + tb.x);
            const float nIM = fmaxf(lMM + D.qMI[e], lIM + D.qII[e]) + ta.x;
            const float nDN = fmaxf(uMM + D.qMD[e], uDN + D.qDD[e]);
            const float nND = fmaxf(lMM + ta.z, lND + tb.z);
            D.MM[e] = nMM; D.MI[e] = nMI; D.IM[e] = nIM; D.DN[e] = nDN; D.ND[e] = nND;
            m[e][u] = nMM;
            // row 1's "up" is this cell
            uMM = nMM; uMI = nMI; uIM = nIM; uDN = nDN; uND = nND;
        }
        if (wr_bot) {
            // lane 31's row 1 (column k0 + u - 31) into the strip's last row
            *reinterpret_cast<float4*>(bnd + P1_BND + 4 * (u0 + u)) = make_float4(uMM, uMI, uIM, uDN);
            bnd[P1_BND + 4 * P1_C + u0 + u] = uND;
        }
    }
    // the maximum of the eight cells first (4 three-input maxima); its cell
    // only when it reaches the lane's maximum, which a lane rarely does
    // (a compare and two selects per cell otherwise)
    const float cm = max3f(max3f(m[0][0], m[0][1], m[0][2]), max3f(m[0][3], m[1][0], m[1][1]), fmaxf(m[1][2], m[1][3]));
    if (cm >= D.best && cm > 0.f) {
        int row = 1, uu = 0;
#pragma unroll
        for (int i = 7; i >= 0; i--)
            if (m[i >> 2][i & 3] == cm) { row = i >> 2; uu = i & 3; }
        // a tie goes to the smaller row, then to the earlier column
        if (cm > D.best || row < D.brow) { D.best = cm; D.brow = row; D.kbest = k0 + uu; }
    }
}

// Phase 1 in FP32.  Per chunk of 8 columns every lane first scores its two
// rows against them (db records staged in shared memory by cp.async and read
// warp-uniformly, once for both rows; the cells are independent, so their
// chains overlap), then the warp advances the wavefront by 8 steps.  Bound by
// instruction issue: two rows a lane halve the record reads and the DP's
// shuffles, column and row-above reads per cell, and the packed dot products
// halve the multiply-adds' issue slots.
template <bool CVUNIF>
__global__ void __launch_bounds__(P1C_WARPS * 32, 1)
p1c_kernel(P1Args a, const float* __restrict__ qbkg)
{
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int cvcard = a.sc.cvcard;
    const int card = a.sc.ssss_card;
    float* cvtab = smem;                                      // [cvcard][P1C_CVREP]
    float* wb = smem + cvcard * P1C_CVREP + wid * P1C_WARP_FLOATS;
    float* ring = wb;                                         // [P1_SLOTS anti-diagonals][P1_RLD] scores
    float* cring = ring + P1_SLOTS * P1_RLD;                  // [P1_CRING][P1C_TRS] column transitions
    float* bnd = cring + P1_CRING * P1C_TRS;                  // [2][P1_BND] row above the strip, its last row
    float* U = bnd + P1_BNDS;                                  // [card][P1_ROWS] SS row table
    float* rec = U + MAX_SSSS_CARD * P1_ROWS;                 // [REC_SLOTS][DR_STRIDE] db records
    for (int i = threadIdx.x; i < cvcard * P1C_CVREP; i += blockDim.x) cvtab[i] = a.cvvals[i / P1C_CVREP];
    // (a lane may read a score slot or record that no chunk has filled yet;
    // such a value reaches no cell inside the matrix, but start from zeros)
    for (int i = lane; i < P1C_WARP_FLOATS; i += 32) wb[i] = 0.f;
    __syncthreads();

    const long long slotw = (long long)blockIdx.x * P1C_WARPS + wid;
    const int Lmax = (int)(a.botstride / 10);
    float* bot0 = a.bot + slotw * a.botstride;
    const int Lq = a.Lq;
    const int nstrips = (Lq + P1_ROWS - 1) / P1_ROWS, ns32 = (Lq + 31) >> 5;
    const ScoreConsts sc = a.sc;

    bool broken = false;   // a strip wait gave up
    for (;;) {
        P1Item it;
        if (!p1_take(a, nstrips, lane, it)) break;
        const int p = it.p, L = it.L;
        const float* __restrict__ dr = a.drec + a.poff[p] * DR_STRIDE;
        const float* __restrict__ bd = a.pbkg + (long long)p * NAA;
        const int edge = corner_edge(Lq, L);
        // rows between the strips: the warp's own buffer, or the split pair's
        const int ldb = it.pi < 0 ? Lmax : (L + 3) & ~3;
        float* botr = it.pi < 0 ? bot0 : a.sbnd + 10 * a.sboff[it.pi];
        float* botw = botr + 5 * ldb;
        if (it.s0 & 1) { float* t = botr; botr = botw; botw = t; }
        float pbest = 0.f;
        int prow = 0x7fffffff, pcol = 0x7fffffff;

        for (int s = it.s0; s < it.s1; s++) {
            __syncwarp();
            const int r0 = P1_ROWS * s + 2 * lane;   // the lane's first row
            const int kend = L + ((min(P1_ROWS, Lq - P1_ROWS * s) - 1) >> 1);   // wavefront steps
            RowOps R[2];
#pragma unroll
            for (int e = 0; e < 2; e++) row_ops(R[e], a.qrec + (long long)min(r0 + e, Lq - 1) * QR_STRIDE, qbkg, bd);
            {
                // this strip's SS row tables (built once per query in strips of
                // 32 rows, c2_set_query); lanes past the query's last 32 rows
                // repeat them (their cells never score)
                const int t = min(2 * s + (lane >> 4), ns32 - 1);
                const float* __restrict__ us = a.qU + (long long)t * MAX_SSSS_CARD * 32 + 2 * (lane & 15);
#pragma unroll 8
                for (int c = 0; c < card; c++)
                    *reinterpret_cast<float2*>(U + c * P1_ROWS + 2 * lane) =
                        __ldg(reinterpret_cast<const float2*>(us + c * 32));
            }
            // scores of -inf for the cells left of the matrix (step k < lane)
#pragma unroll 4
            for (int k = 0; k < 31; k++)
                if (k < lane)
                    *reinterpret_cast<float2*>(ring + k * P1_RLD + 2 * lane) = make_float2(-INFINITY, -INFINITY);
            Wf2 D;
            wf2_init(D, a.qrec, r0, Lq);
            // corner cells of the lane's rows: columns <= cA or >= cB
            const int cA0 = corner_a(r0, Lq, edge), cA1 = corner_a(r0 + 1, Lq, edge);
            const int cB0 = corner_b(r0, L, edge), cB1 = corner_b(r0 + 1, L, edge);
            const bool wr_bot = (lane == 31) && (s + 1 < nstrips);
            // records and transitions of the first two chunks
            stage_chunk(rec, dr, 0, L, lane);
            stage_trn(cring, dr, 0, 0, L, lane);
            cp_async_commit();
            stage_chunk(rec, dr, 1, L, lane);
            stage_trn(cring, dr, 1, P1_C, L, lane);
            cp_async_commit();
            int sg = 0;                                 // slot of the chunk's first anti-diagonal
            int cs = 0, cl = lane == 0 ? 0 : P1_CMOD - lane;
            for (int m = 0; P1_C * m < kend; m++) {
                const int k0 = P1_C * m;
                // the row above for this chunk's steps, copied during the score stage
                p1_row_async(a, it, s, bnd, botr, ldb, k0, lane, broken);
                cp_async_wait_2();   // records and transitions of chunk m have landed
                __syncwarp();
                // ---- score stage: columns [k0, k0 + 8); past the last column -inf,
                // for the lanes still to finish the matrix
                {
                    int w = sg + lane;
                    if (w >= P1_SLOTS) w -= P1_SLOTS;
                    const float* rc = rec + (k0 & (REC_SLOTS - 1)) * DR_STRIDE;
                    const bool hasc = __any_sync(FULL, cA1 >= k0 || cB0 < k0 + P1_C);
#pragma unroll 2
                    for (int u = 0; u < P1_C; u++) {
                        float S[2] = {-INFINITY, -INFINITY};
                        if (k0 + u < L) {
                            float mod[2];
                            cell_scores<P1C_CVREP, 2, P1_ROWS, CVUNIF>(R, rc + u * DR_STRIDE, U, 2 * lane, cvtab, sc, lane, S, mod);
                            if (hasc) {
                                const int c = k0 + u;
                                if (c <= cA0 || c >= cB0) S[0] = -9.f;
                                if (c <= cA1 || c >= cB1) S[1] = -9.f;
                            }
                        }
                        *reinterpret_cast<float2*>(ring + w * P1_RLD + 2 * lane) = make_float2(S[0], S[1]);
                        if (++w >= P1_SLOTS) w = 0;
                    }
                }
                cp_async_wait_all();
                __syncwarp();
                // ---- DP stage: wavefront steps [k0, k0 + 8)
                const float* rp = ring + sg * P1_RLD + 2 * lane;
                const float* tcol = cring + cl * P1C_TRS;
                if (k0 < 32) {
                    Wf2Edge E;
                    wf2_edge(E, D, a.qrec, r0, Lq);
#pragma unroll 1
                    for (int u0 = 0; u0 < P1_C; u0 += 4)
                        wf2_steps4<true>(D, E, rp + u0 * P1_RLD, tcol + u0 * P1C_TRS, bnd, u0, k0 + u0 - lane, k0 + u0,
                                         lane, wr_bot);
                } else {
                    Wf2Edge E;
#pragma unroll 1
                    for (int u0 = 0; u0 < P1_C; u0 += 4)
                        wf2_steps4<false>(D, E, rp + u0 * P1_RLD, tcol + u0 * P1C_TRS, bnd, u0, k0 + u0 - lane, k0 + u0,
                                          lane, wr_bot);
                }
                __syncwarp();
                if (s + 1 < nstrips) {
                    p1_row_flush(bnd + P1_BND, botw, ldb, k0, L, lane);
                    // columns up to k0 - 24 are there: published every other chunk
                    if (it.pi >= 0 && k0 >= 24 && ((m & 1) || k0 + P1_C >= kend))
                        p1_publish(a, it, s, min(k0 - 23, L), lane);
                }
                // next chunk; chunk m + 2's records and transitions into slots no longer read
                sg = sg + P1_C >= P1_SLOTS ? 0 : sg + P1_C;
                cs = cs + P1_C >= P1_CMOD ? 0 : cs + P1_C;
                cl = cl + P1_C >= P1_CMOD ? cl + P1_C - P1_CMOD : cl + P1_C;
                stage_chunk(rec, dr, m + 2, L, lane);
                stage_trn(cring, dr, m + 2, cs + P1_C >= P1_CMOD ? 0 : cs + P1_C, L, lane);
                cp_async_commit();
                __syncwarp();
            }
            cp_async_wait_all();
            {
                const int rr = r0 + D.brow, cc = D.kbest - lane;
                if (D.best > 0.f && (D.best > pbest || (D.best == pbest && (rr < prow || (rr == prow && cc < pcol))))) {
                    pbest = D.best; prow = rr; pcol = cc;
                }
            }
            float* t = botr; botr = botw; botw = t;
            __syncwarp();
        }
        p1_result(a, it, nstrips, lane, pbest, prow, pcol);
    }
}

// ---------------------------------------------------------------------------
// Phase-2 score matrices: the FP32 scores and modular scores of every cell of
// the candidate pairs, column-major per pair (the layout of the finalisation,
// statistics and MAP stages), by cell_scores -- the arithmetic of phase 1's
// FP32 form.  One warp per (candidate, strip) at a time, lanes own query rows,
// db records staged in shared memory as in phase 1; no dependencies between
// work items, so every resident warp works.  Where there are few candidates an
// item is a block of columns (P1Args::p2s_cols).
template <bool CVUNIF>
__global__ void __launch_bounds__(P2S_WARPS * 32)
p2s_kernel(P1Args a, const float* __restrict__ qbkg)
{
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int cvcard = a.sc.cvcard;
    const int card = a.sc.ssss_card;
    float* cvtab = smem;                                      // [cvcard][P1TC_CVREP]
    float* U = smem + cvcard * P1TC_CVREP + wid * P2S_WARP_FLOATS;   // [card][32]
    float* rec = U + MAX_SSSS_CARD * 32;                      // [REC_SLOTS][DR_STRIDE] db records
    for (int i = threadIdx.x; i < cvcard * P1TC_CVREP; i += blockDim.x) cvtab[i] = a.cvvals[i / P1TC_CVREP];
    __syncthreads();
    const int Lq = a.Lq;
    const int nstrips = (Lq + 31) >> 5;
    const int nsb = nstrips * a.p2s_blocks;
    const int nitems = a.nwork * nsb;
    const ScoreConsts sc = a.sc;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.counter + 1, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= nitems) break;
        const int cand = a.worder[item / nsb];
        const int sb = item % nsb, s = sb / a.p2s_blocks;
        const int p = a.order[cand];
        const int cb = (sb - s * a.p2s_blocks) * a.p2s_cols;   // columns [cb, L)
        const int L = min(a.plen[p], cb + a.p2s_cols);
        if (cb >= L) continue;
        const float* __restrict__ dr = a.drec + a.poff[p] * DR_STRIDE;
        const float* __restrict__ bd = a.pbkg + (long long)p * NAA;
        const long long coff = a.cand_off[cand];
        float* smt = a.smat + coff;
        float* mmt = a.mmat + coff;
        const int r = s * 32 + lane;
        const bool act = r < Lq;
        const float* __restrict__ qr = a.qrec + (long long)(act ? r : Lq - 1) * QR_STRIDE;
        RowOps R;
        row_ops(R, qr, qbkg, bd);
        __syncwarp();
        {
            // this strip's SS row tables (built once per query, c2_set_query)
            const float* __restrict__ us = a.qU + (long long)s * MAX_SSSS_CARD * 32 + lane;
#pragma unroll 8
            for (int c = 0; c < card; c++) U[c * 32 + lane] = __ldg(us + c * 32);
        }
        stage_chunk(rec, dr, cb >> REC_CHUNK_LOG, L, lane);
        cp_async_commit();
        stage_chunk(rec, dr, (cb >> REC_CHUNK_LOG) + 1, L, lane);
        cp_async_commit();
        // a staged chunk of REC_CHUNK columns at a time: its cells are
        // independent, so their chains overlap
        for (int c0 = cb; c0 < L; c0 += REC_CHUNK) {
            cp_async_wait_1();
            __syncwarp();
#pragma unroll
            for (int u = 0; u < REC_CHUNK; u++) {
                const int c = c0 + u;
                if (c < L) {
                    const float* rc = rec + (c & (REC_SLOTS - 1)) * DR_STRIDE;
                    float mod, Sc;
                    cell_scores<P1TC_CVREP, 1, 32, CVUNIF>(&R, rc, U, lane, cvtab, sc, lane, &Sc, &mod);
                    if (act) {
                        smt[(long long)c * Lq + r] = Sc;
                        mmt[(long long)c * Lq + r] = mod;
                    }
                }
            }
            __syncwarp();
            stage_chunk(rec, dr, (c0 >> REC_CHUNK_LOG) + 2, L, lane);
            cp_async_commit();
        }
        cp_async_wait_all();
        __syncwarp();
    }
}

// Traceback sweep over the candidate pairs: the FP32 Viterbi DP again, on the
// score matrices p2s_kernel wrote (ExecDP_Btck_Unroll32x, src/libmycu/cudp/
// CuBatchDP_init_btck.cu:303-360), with the btck code of every cell stored
// column-major and the strips of a pair pipelined over warps (c2_device.cuh): a
// chunk of 16 columns at a time, its scores loaded a chunk ahead into the
// anti-diagonal ring and the row above fetched just before its steps, so that a
// strip trails the one above by about 50 steps.  The arithmetic is p1c_kernel's:
// the maxima equal phase 1's in the FP32 form.
__global__ void __launch_bounds__(P1TC_WARPS * 32, 1)
p1tc_kernel(P1Args a, const float* __restrict__ qbkg)
{
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __shared__ signed char btr_all[P1TC_WARPS][32][33];
    signed char(*btr)[33] = btr_all[wid];
    float* wb = smem + wid * P1TC_WARP_FLOATS;
    float* ring = wb;                                         // [P1C_RING][32] scores
    float* trn = ring + P1C_RING * 32;                        // [P1C_RING][P1C_TRS] transitions
    float* bnd = trn + P1C_RING * P1C_TRS;                    // row above the strip, two chunks
    (void)qbkg;

    const int Lq = a.Lq;
    const int nstrips = (Lq + 31) >> 5;
    const int nitems = a.nwork * nstrips;
    bool broken = false;

    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.counter, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= nitems) break;
        const int iv = a.items[item];
        const int rank = iv / nstrips, s = iv - rank * nstrips;
        const int cand = a.worder[rank];
        const int p = a.order[cand];
        const int L = a.plen[p];
        const long long off = a.poff[p];
        const float* __restrict__ dr = a.drec + off * DR_STRIDE;
        const int edge = corner_edge(Lq, L);
        const long long coff = a.cand_off[cand];
        signed char* bt = a.btck + coff;
        const float* smt = a.smat + coff;
        const int ldr = row_ld(L);
        float* rowm = a.bnd + 5 * (nstrips * row_start(coff / Lq, cand) + (long long)s * ldr);   // this strip's last row
        const float* rowa = rowm - 5 * ldr;                                                      // the one above (s > 0)
        const int r = s * 32 + lane;
        const bool act = r < Lq;
        const float* __restrict__ qr = a.qrec + (long long)(act ? r : Lq - 1) * QR_STRIDE;
        WfLane D;
        {
            float q7[7];
#pragma unroll
            for (int i = 0; i < 7; i++) q7[i] = act ? qr[QR_TRN + i] : LOG0;
            const bool z_left = (lane == 31);
            const bool z_diag = (lane == 31 || lane == 0);
            const St5 LB = z_left ? St5{0.f, 0.f, 0.f, 0.f, 0.f}
                                  : St5{0.f, qr[QR_C + 0], qr[QR_C + 1], qr[QR_C + 2], LOG0};
            const St5 DB = z_diag ? St5{0.f, 0.f, 0.f, 0.f, 0.f}
                                  : St5{0.f, qr[QR_CP + 0], qr[QR_CP + 1], qr[QR_CP + 2], LOG0};
            wf_init(D, q7, LB, DB);
        }
        const int cA = corner_a(r, Lq, edge);
        const int cB = corner_b(r, L, edge);
        const bool wr_row = (lane == 31) && (s + 1 < nstrips);
        const int kend = L + 31;
        // scores of a chunk's columns (the lanes' rows of one column: one
        // 128-byte line) and the columns' transitions, loaded a chunk ahead
        float sc[TB_C];
        float4 tv;
        auto fetch = [&](int c0) {
#pragma unroll
            for (int u = 0; u < TB_C; u++) sc[u] = (act && c0 + u < L) ? __ldcg(smt + (long long)(c0 + u) * Lq + r) : 0.f;
            const int c = c0 + (lane >> 1);
            if (c < L) tv = __ldg(reinterpret_cast<const float4*>(dr + (long long)c * DR_STRIDE + DR_TRN) + (lane & 1));
        };
        fetch(0);
        __syncwarp();
        if (s > 0) row_issue<TB_C>(bnd, rowa, ldr, 0, L, lane);
        else
            for (int i = lane; i < 2 * ROW_BUF<TB_C>; i += 32) bnd[i] = 0.f;
        for (int k0 = 0; k0 < kend; k0 += TB_C) {
            if (k0 < L) {
                const bool hasc = __any_sync(FULL, cA >= k0 || cB < k0 + TB_C);
#pragma unroll
                for (int u = 0; u < TB_C; u++) {
                    const int c = k0 + u;
                    if (hasc && (c <= cA || c >= cB)) sc[u] = -9.f;
                    if (c < L) ring[((c + lane) & (P1C_RING - 1)) * 32 + lane] = sc[u];
                }
                const int c = k0 + (lane >> 1);
                if (c < L) *reinterpret_cast<float4*>(trn + (c & (P1C_RING - 1)) * P1C_TRS + 4 * (lane & 1)) = tv;
                fetch(k0 + TB_C);
            }
            // the row above for this chunk's steps, the next chunk's on its way
            float* rb = bnd + (k0 & TB_C ? ROW_BUF<TB_C> : 0);
            if (s > 0) {
                if (k0 < L) row_take<TB_C>(rb, rowa, ldr, k0, L, lane, a.status, broken, a.spin);
                if (k0 + TB_C < L) row_issue<TB_C>(bnd + (k0 & TB_C ? 0 : ROW_BUF<TB_C>), rowa, ldr, k0 + TB_C, L, lane);
            }
            __syncwarp();
            // ---- DP stage: wavefront steps [k0, k0 + TB_C), traceback codes stored
            if (k0 >= 32 && k0 + TB_C <= L)
                wf_steps<false>(D, k0, TB_C, lane, L, act, ring, trn, rb, wr_row, rowm, ldr, btr, bt, Lq, r);
            else
                wf_steps<true>(D, k0, min(TB_C, kend - k0), lane, L, act, ring, trn, rb, wr_row, rowm, ldr, btr, bt, Lq,
                               r);
            __syncwarp();
        }
        // the strip's maximum: largest score, then smallest row, then smallest column
        float best = D.best;
        int brow = (best > 0.f) ? r : 0x7fffffff;
        int bcol = (best > 0.f) ? D.kbest - lane : 0x7fffffff;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const float ob = __shfl_xor_sync(FULL, best, o);
            const int orr = __shfl_xor_sync(FULL, brow, o);
            const int oc = __shfl_xor_sync(FULL, bcol, o);
            if (ob > best || (ob == best && (orr < brow || (orr == brow && oc < bcol)))) {
                best = ob; brow = orr; bcol = oc;
            }
        }
        // pair maximum over strips as one 64-bit key (best >= 0 orders by its bits)
        if (lane == 0 && best > 0.f) {
            const unsigned cell = ((unsigned)brow << 16) | ((unsigned)bcol & 0xffffu);
            atomicMax(a.tbkey + cand,
                      ((unsigned long long)__float_as_uint(best) << 32) | (unsigned long long)(0xffffffffu - cell));
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Tensor-core score path (layouts in c2_device.cuh).

__device__ __forceinline__ unsigned bf16_bits(float x)
{
    return (unsigned)__bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// hi and lo BF16 parts of x: hi = bf16(x), lo = bf16(x - hi)
__device__ __forceinline__ void bf16_split(float x, unsigned& hi, unsigned& lo)
{
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    hi = (unsigned)__bfloat16_as_ushort(h);
    lo = bf16_bits(x - __bfloat162float(h));
}

// D += A * B, m16n8k16, BF16 inputs, FP32 accumulation
// first product of a chain: C = 0 (no accumulator zeroing)
__device__ __forceinline__ void mma_bf16_z(float* d, const unsigned* a, unsigned b0, unsigned b1)
{
    const float z = 0.f;
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(z));
}

__device__ __forceinline__ void mma_bf16(float* d, const unsigned* a, unsigned b0, unsigned b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the same with K = 8
__device__ __forceinline__ void mma_bf16_k8(float* d, unsigned a0, unsigned a1, unsigned b0)
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0));
}

// mbarrier and bulk (non-tensor, non-multicast) async copy helpers
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Tensor memory (TMEM) as a per-lane store of loop-invariant fragments: the
// allocating warp takes ncols columns for the CTA; warp w reads and writes
// lanes [32 (w % 4), 32 (w % 4) + 32) only (32x32b shape: thread i <-> lane
// 32 (w % 4) + i, consecutive 32-bit columns).
__device__ __forceinline__ void tmem_alloc(unsigned* dst_smem, unsigned ncols)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_st40(unsigned taddr, const unsigned* v)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr + 32),
        "r"(v[32]), "r"(v[33]), "r"(v[34]), "r"(v[35]), "r"(v[36]), "r"(v[37]), "r"(v[38]), "r"(v[39])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 40 columns into v: the loads, and the wait for them.  The wait takes v as
// operands, so no use of v can be scheduled before the loads have completed;
// nothing may touch v in between.
__device__ __forceinline__ void tmem_ld40(unsigned taddr, unsigned* v)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[32]), "=r"(v[33]), "=r"(v[34]), "=r"(v[35]), "=r"(v[36]), "=r"(v[37]), "=r"(v[38]), "=r"(v[39])
        : "r"(taddr + 32)
        : "memory");
}
__device__ __forceinline__ void tmem_ld40_wait(unsigned* v)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31]), "+r"(v[32]), "+r"(v[33]), "+r"(v[34]), "+r"(v[35]), "+r"(v[36]), "+r"(v[37]), "+r"(v[38]), "+r"(v[39])
                 :
                 : "memory");
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// one thread: expect `bytes` on the barrier and start the copy global -> shared
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Wait for phase `parity` of the barrier to complete; gives up after a bounded
// number of polls (returns false; the caller records a device status).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity)
{
    const unsigned a = smem_u32(bar);
    for (int it = 0; it < (1 << 22); it++) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Pack the db operands of one profile per CTA (4 warps over its 8-column
// tiles) and its column records.  lok: 1/kappa0 (CV column k = 19); wss: SS
// weight (SS operand and its folded columns k = 30, 31).
__global__ void __launch_bounds__(128) tc_pack_kernel(const float* __restrict__ drec, const long long* __restrict__ poff,
                                                      const int* __restrict__ plen, const long long* __restrict__ ttile,
                                                      unsigned* __restrict__ tcdb, float* __restrict__ cold, float lok,
                                                      float wss)
{
    const int p = blockIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int L = plen[p];
    const long long off = poff[p];
    const int ntiles = (L + P1_C - 1) / P1_C;
    const int g = lane >> 2, q = lane & 3;
    for (int t = wid; t < ntiles; t += 4) {
        const int col = P1_C * t + g;
        const bool valid = col < L;
        const float* rc = drec + (off + (valid ? col : 0)) * DR_STRIDE;
        const int pk = __float_as_int(rc[DR_SSIDX]);
        const int i0 = pk & 0xff, i1 = (pk >> 8) & 0xff, i2 = (pk >> 16) & 0xff;
        // words of the three operands: k 0-15 (2), then k 16-23 (1) or k 16-31 (2)
        unsigned h[3][4], l[3][4];
#pragma unroll
        for (int d = 0; d < 3; d++) {
#pragma unroll
            for (int w = 0; w < 4; w++) {
                unsigned hh[2], ll[2];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int k = 8 * w + 2 * q + e;
                    float x = 0.f;
                    if (valid) {
                        if (d == 0) x = (k < NAA) ? rc[DR_TRG + k] : 0.f;
                        else if (d == 1) x = (k < NCV) ? rc[DR_CV + k] : (k == NCV) ? lok : 0.f;
                        else if (k == i0) x = wss * rc[DR_SS];
                        else if (k == i1) x = wss * rc[DR_SS + 1];
                        else if (k == i2) x = wss * rc[DR_SS + 2];
                        else if (k == TC_SS_KMAX) x = wss * (rc[DR_HD] * 0.1111111f);
                        else if (k == TC_SS_KMAX + 1) x = -0.05f * wss;
                    }
                    bf16_split(x, hh[e], ll[e]);
                }
                h[d][w] = hh[0] | (hh[1] << 16);
                l[d][w] = ll[0] | (ll[1] << 16);
            }
        }
        uint4* out = reinterpret_cast<uint4*>(tcdb + (ttile[p] + t) * (long long)TC_TILE_WORDS) + lane;
        out[0 * 32] = make_uint4(h[0][0], h[0][1], h[0][2], l[0][2]);
        out[1 * 32] = make_uint4(l[0][0], l[0][1], h[1][0], h[1][1]);
        out[2 * 32] = make_uint4(l[1][0], l[1][1], h[1][2], l[1][2]);
        out[3 * 32] = make_uint4(h[2][0], h[2][1], h[2][2], h[2][3]);
        out[4 * 32] = make_uint4(l[2][0], l[2][1], l[2][2], l[2][3]);
    }
    for (int c = threadIdx.x; c < L; c += blockDim.x) {
        const float* rc = drec + (off + c) * DR_STRIDE;
        float* o = cold + (off + c) * P1C_TRS;
#pragma unroll
        for (int i = 0; i < 7; i++) o[i] = rc[DR_TRN + i];
        o[7] = 0.f;
        o[CO_CD] = rc[DR_CN];
        o[CO_PD2] = 2.f * rc[DR_PRIOR];
        o[10] = o[11] = 0.f;
    }
}

// Score epilogue of one cell of the tensor-core form from its three
// contractions (the CV one with 1/kappa0 folded in, the SS one the complete
// weighted SS term):
//   x   = 2 (cterm + pownu0 ln(cq cd - dot^2) - prior_q - prior_d)
//   cvm = w_cv T[shift + rint(x)] (T clamped; the key range tests when the
//         table is not uniform)
//   S   = (ln(aa) - shift) + (ss + cvm), evaluated as ln(aa) + (ss +
//         (cvm - shift)) with the table pre-shifted: a reassociation within
//         the rounding of the split-BF16 products (this form only ranks the
//         pairs; the candidates are rescored in FP32)
// (cell_scores is the FP32 form; src/libmycu/cusco/CuBatchScoreMatrix_ddms2s_h2.cu)
template <bool CVUNIF>
__device__ __forceinline__ float tc_cell(float daa, float dot, float ss, float cq, float rq2, float cd, float pd2,
                                         const float* __restrict__ cvl, const TcConsts& tc)
{
    // rq2 = c2 - 2 prior_q (per row); the table values and vfw, vlw carry the
    // -shift of the amino-acid term, so the cell is ln(daa) + (ss + cv)
    const float det = fmaf(-dot, dot, cq * cd);
    const float x = fmaf(tc.p2l, lg2_ftz(det), rq2) - pd2;
    const int ix = min(max(__float2int_rn(x), tc.ilo), tc.ihi);
    float cvm = cvl[ix * P1T_CVREP];
    if (!CVUNIF) {
        cvm = (tc.kl2 <= x) ? tc.vlw - tc.shift : cvm;
        cvm = (x <= tc.kf2) ? tc.vfw - tc.shift : cvm;
    }
    return fmaf(lg2_ftz(daa), C2_LN2, ss + cvm);
}

// Stage the column records of chunk m (8 columns, ring slots from cs on; the
// chunk at slot 0 also into the mirror slots after the last chunk)
__device__ __forceinline__ void stage_cols(float* cring, const float* __restrict__ cold, int m, int cs, int L, int lane)
{
    const int n16 = min(P1_C, L - P1_C * m) * (P1C_TRS / 4);
    if (lane < n16) {
        const float* src = cold + (long long)(P1_C * m) * P1C_TRS + 4 * lane;
        cp_async16(cring + cs * P1C_TRS + 4 * lane, src);
        if (cs == 0) cp_async16(cring + P1_CMOD * P1C_TRS + 4 * lane, src);
    }
    cp_async_commit();
}

// Phase 1 with the score contractions on the tensor cores: per chunk of 8
// columns the warp computes the 64 x 8 score tile of its strip with mma.sync
// (fragment layout: lane (g, q) holds rows g, g + 8 of each 16-row tile and
// columns 2q, 2q + 1), applies the epilogue per cell, writes the scores into
// the anti-diagonal ring, then advances the wavefront DP by 8 steps.
// CVUNIF: the CV table's key range coincides with its index clamp (TcConsts)
template <bool CVUNIF>
__global__ void __launch_bounds__(P1T_WARPS * 32, 1)
p1t_kernel(P1Args a, const float* __restrict__ qbkg)
{
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int cvcard = a.sc.cvcard;
    float* cvtab = smem;                                      // [cvcard][P1T_CVREP], x CV weight
    float* wb = smem + cvcard * P1T_CVREP + wid * P1T_WARP_FLOATS;
    float* ring = wb;                                         // [P1_SLOTS anti-diagonals][P1_RLD] scores
    float* cring = ring + P1_SLOTS * P1_RLD;                // [P1_CRING][P1C_TRS] column records
    float* bnd = cring + P1_CRING * P1C_TRS;                 // [2][P1_BND] row above the strip, its last row
    float* rqt = bnd + P1_BNDS;                               // [P1_ROWS][2] cvnorm, c2 - 2 x CV log prior
    unsigned* btile = reinterpret_cast<unsigned*>(rqt + 2 * P1_ROWS);   // [TC_TILE_WORDS] db operand tile
    unsigned long long* tbar = reinterpret_cast<unsigned long long*>(btile + TC_TILE_WORDS);
    for (int i = threadIdx.x; i < cvcard * P1T_CVREP; i += blockDim.x)
        cvtab[i] = a.cvvals[i / P1T_CVREP] * a.sc.cvswgt - a.tc.shift;
    // (a lane may read a score slot or record that no chunk has filled yet;
    // such a value reaches no cell inside the matrix, but start from zeros)
    for (int i = lane; i < P1T_WARP_FLOATS - 4; i += 32) wb[i] = 0.f;
    __shared__ unsigned tmem_base;
    if (lane == 0) {
        mbar_init(tbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the zeros above before the async proxy's writes
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // all query A fragments of the current strip live in TMEM (160 columns per
    // warp; warps w, w + 4, w + 8 share lanes)
    if (wid == 0) tmem_alloc(&tmem_base, P1T_TMEM_COLS);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tq = tmem_base + ((unsigned)(32 * (wid & 3)) << 16) + (unsigned)((wid >> 2) * P1T_TMEM_WARP);
    unsigned tph = 0;   // phase parity of the tile slot's barrier
    // a tile wait that gave up: the warp issues no further tile copies and
    // waits for none, and before it exits waits (bounded) once more for the
    // copy it gave up on, so that no copy into this CTA's shared memory is in
    // flight when the CTA ends
    bool tbroken = false;
    unsigned tpend = 0;

    const long long slotw = (long long)blockIdx.x * P1T_WARPS + wid;
    const int Lmax = (int)(a.botstride / 10);
    float* bot0 = a.bot + slotw * a.botstride;
    const int Lq = a.Lq;
    const int nstrips = (Lq + P1_ROWS - 1) / P1_ROWS;
    const TcConsts tc = a.tc;
    const int g = lane >> 2, q = lane & 3;
    // this lane's CV table replica, offset so that index 0 is the table's key 0
    const float* __restrict__ cvl = cvtab + a.sc.cvshift * P1T_CVREP + (lane & (P1T_CVREP - 1));
    // score writes: cell register i = 2 hh + e of m-tile mt (row 16 mt + 8 hh + g,
    // column 2 q + e of the chunk) goes to the anti-diagonal 8 mt + x past the
    // chunk's first, x = 2 q + e + 4 hh + g / 2: slot x & 7 of segment mt + (x >> 3)
    int woff[4];
    bool wnext[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int x = 2 * q + (i & 1) + 4 * (i >> 1) + (g >> 1);
        woff[i] = (x & 7) * P1_RLD + g + 8 * (i >> 1);
        wnext[i] = x >= 8;
    }

    bool broken = false;   // a strip wait gave up
    for (;;) {
        P1Item it;
        if (!p1_take(a, nstrips, lane, it)) break;
        const int p = it.p, L = it.L;
        const long long off = a.poff[p];
        const float* __restrict__ cold = a.cold + off * P1C_TRS;
        const unsigned* __restrict__ tb0 = a.tcdb + a.ttile[p] * (long long)TC_TILE_WORDS;
        const int edge = corner_edge(Lq, L);
        // rows between the strips: the warp's own buffer, or the split pair's
        const int ldb = it.pi < 0 ? Lmax : (L + 3) & ~3;
        float* botr = it.pi < 0 ? bot0 : a.sbnd + 10 * a.sboff[it.pi];
        float* botw = botr + 5 * ldb;
        if (it.s0 & 1) { float* t = botr; botr = botw; botw = t; }
        float pbest = 0.f;
        int prow = 0x7fffffff, pcol = 0x7fffffff;

        for (int s = it.s0; s < it.s1; s++) {
            __syncwarp();
            const int rows = min(P1_ROWS, Lq - P1_ROWS * s);   // of the query in this strip
            const int nmt = (rows + 15) >> 4;                  // m-tiles holding any
            const int kend = L + ((rows - 1) >> 1);            // wavefront steps
            // this strip's query fragments into TMEM, 40 columns per m-tile:
            // the amino-acid rows scaled for the pair (q(a) / (0.5 (bq(a) +
            // bd(a))), as row_ops' Qt) and split, then the CV and SS words
            {
                const float* __restrict__ bd = a.pbkg + (long long)p * NAA;
                float w[6];
#pragma unroll
                for (int i = 0; i < 6; i++) {
                    const int k = 8 * (i >> 1) + 2 * q + (i & 1);
                    w[i] = (k < NAA) ? __fdividef(1.f, 0.5f * (qbkg[k] + bd[k])) : 0.f;
                }
                for (int mt = 0; mt < nmt; mt++) {
                    unsigned v[40];
                    const float4* sa = reinterpret_cast<const float4*>(a.qaa) + (long long)(s * 4 + mt) * 96 + lane;
                    const uint4* sq = reinterpret_cast<const uint4*>(a.qa) + (long long)(s * 4 + mt) * 224 + lane;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const float4 x = __ldg(sa + i * 32);
                        unsigned h[4], l[4];
                        bf16_split(x.x * w[2 * i], h[0], l[0]);
                        bf16_split(x.y * w[2 * i + 1], h[1], l[1]);
                        bf16_split(x.z * w[2 * i], h[2], l[2]);
                        bf16_split(x.w * w[2 * i + 1], h[3], l[3]);
                        const int o = i < 2 ? 2 * i : 32;   // k 0-15; k 16-23
                        v[o] = h[0] | (h[1] << 16);
                        v[o + 1] = h[2] | (h[3] << 16);
                        const int ol = i < 2 ? 4 + 2 * i : 34;
                        v[ol] = l[0] | (l[1] << 16);
                        v[ol + 1] = l[2] | (l[3] << 16);
                    }
#pragma unroll
                    for (int i = 0; i < 7; i++) {
                        const uint4 x = __ldg(sq + i * 32);
                        const int o = i < 6 ? 8 + 4 * i : 36;
                        v[o] = x.x; v[o + 1] = x.y; v[o + 2] = x.z; v[o + 3] = x.w;
                    }
                    tmem_st40(tq + P1T_TMEM_MT * mt, v);
                }
                tmem_wait_st();
            }
            const int r0 = P1_ROWS * s + 2 * lane;   // the lane's first row
            {
                // the rows' score terms, and scores of -inf for the cells left
                // of the matrix (step k < lane) and the m-tiles past the query
                const float* qx0 = a.qrec + (long long)min(r0, Lq - 1) * QR_STRIDE;
                const float* qx1 = a.qrec + (long long)min(r0 + 1, Lq - 1) * QR_STRIDE;
                *reinterpret_cast<float4*>(rqt + 4 * lane) =
                    make_float4(qx0[QR_CN], tc.c2 - 2.f * qx0[QR_PRIOR], qx1[QR_CN], tc.c2 - 2.f * qx1[QR_PRIOR]);
#pragma unroll 4
                for (int k = 0; k < P1_SLOTS; k++)
                    if (k < lane || lane >= 8 * nmt)
                        *reinterpret_cast<float2*>(ring + k * P1_RLD + 2 * lane) = make_float2(-INFINITY, -INFINITY);
            }
            Wf2 D;
            wf2_init(D, a.qrec, r0, Lq);
            // corner cells of the lane's rows: columns <= cA or >= cB
            const int cA = r0 + 1 < Lq ? corner_a(r0 + 1, Lq, edge) : corner_a(r0, Lq, edge);
            const int cB = corner_b(r0, L, edge);
            const bool wr_bot = (lane == 31) && (s + 1 < nstrips);
            stage_cols(cring, cold, 0, 0, L, lane);
            stage_cols(cring, cold, 1, P1_C, L, lane);
            const int nch = (L + P1_C - 1) / P1_C;      // chunks holding columns
            // db operand tiles stream through the slot, one ahead: tile m + 1
            // loads while tile m's products, epilogue and DP steps run
            if (lane == 0 && !tbroken) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                bulk_load(btile, tb0, TC_TILE_WORDS * 4, tbar);
            }
            // ring segments (8 slots each, float offsets) of the chunk's anti-diagonals
            // 0-7, 8-15, ..; the chunk's first record slot; the lane's record slot
            int sg[5];
#pragma unroll
            for (int i = 0; i < 5; i++) sg[i] = i * P1_C * P1_RLD;
            int cs = 0, cl = lane == 0 ? 0 : P1_CMOD - lane;
            for (int m = 0; P1_C * m < kend; m++) {
                const int k0 = P1_C * m;
                // the row above for this chunk's steps, copied during the score stage
                p1_row_async(a, it, s, bnd, botr, ldb, k0, lane, broken);
                if (m < nch) {
                    cp_async_wait_2();   // column records of chunk m have landed
                    if (!tbroken && !__all_sync(FULL, mbar_wait(tbar, tph))) {
                        tbroken = true;
                        tpend = tph;
                        if (lane == 0 && a.status) atomicCAS(a.status, 0, PIPE_ERR_TIMEOUT_P1);
                    }
                    tph ^= 1u;
                    const uint4* bt = reinterpret_cast<const uint4*>(btile) + lane;
                    const uint4 b0 = bt[0], b1 = bt[32], b2 = bt[64], b3 = bt[96], b4 = bt[128];
                    // slot free once every lane holds its fragments: the next tile into it
                    __syncwarp();
                    if (m + 1 < nch) {
                        const unsigned* nx = tb0 + (long long)(m + 1) * TC_TILE_WORDS;
                        if (lane == 0 && !tbroken) {
                            // the warp's reads of the slot before the async-proxy write
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                            bulk_load(btile, nx, TC_TILE_WORDS * 4, tbar);
                        }
                        // the tile after that (20 lines) towards L2
                        if (m + 2 < nch && lane < TC_TILE_WORDS / 32)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + TC_TILE_WORDS + lane * 32));
                    }
                    // does any row of the strip have corner cells in this chunk?
                    const bool hasc = __any_sync(FULL, cA >= k0 || cB < k0 + P1_C);
                    const float* cr = cring + (cs + 2 * q) * P1C_TRS + CO_CD;
                    const float2 cp0 = *reinterpret_cast<const float2*>(cr);
                    const float2 cp1 = *reinterpret_cast<const float2*>(cr + P1C_TRS);
                    const float cd[2] = {cp0.x, cp1.x}, pd[2] = {cp0.y, cp1.y};
                    // ---- score stage: 64 x 8 tile of chunk m on the tensor cores
                    unsigned Q[40];   // k 0-15: aa hi, lo, cv hi, lo; ss hi 8, lo 8; k 16-23: aa hi 2, lo 2, cv hi 2, lo 2
                    tmem_ld40(tq, Q);
#pragma unroll
                    for (int mt = 0; mt < 4; mt++) {
                        if (mt >= nmt) break;
                        tmem_ld40_wait(Q);
                        float acc[3][4];
                        const unsigned *Ah = Q, *Al = Q + 4, *Ch = Q + 8, *Cl = Q + 12, *Sh = Q + 16, *Sl = Q + 24;
                        mma_bf16_z(acc[0], Al, b0.x, b0.y);
                        mma_bf16_z(acc[1], Cl, b1.z, b1.w);
                        mma_bf16_z(acc[2], Sl, b3.x, b3.y);
                        mma_bf16(acc[0], Ah, b1.x, b1.y);
                        mma_bf16(acc[1], Ch, b2.x, b2.y);
                        mma_bf16(acc[2], Sh, b4.x, b4.y);
                        mma_bf16(acc[0], Ah, b0.x, b0.y);
                        mma_bf16(acc[1], Ch, b1.z, b1.w);
                        mma_bf16(acc[2], Sh, b3.x, b3.y);
                        mma_bf16_k8(acc[0], Q[34], Q[35], b0.z);
                        mma_bf16_k8(acc[1], Q[38], Q[39], b2.z);
                        mma_bf16(acc[2], Sl + 4, b3.z, b3.w);
                        mma_bf16_k8(acc[0], Q[32], Q[33], b0.w);
                        mma_bf16_k8(acc[1], Q[36], Q[37], b2.w);
                        mma_bf16(acc[2], Sh + 4, b4.z, b4.w);
                        mma_bf16_k8(acc[0], Q[32], Q[33], b0.z);
                        mma_bf16_k8(acc[1], Q[36], Q[37], b2.z);
                        mma_bf16(acc[2], Sh + 4, b3.z, b3.w);
                        // the next m-tile's fragments load during the epilogue
                        if (mt + 1 < nmt) tmem_ld40(tq + P1T_TMEM_MT * (mt + 1), Q);
                        const float2 rq0 = *reinterpret_cast<const float2*>(rqt + 2 * (16 * mt + g));
                        const float2 rq1 = *reinterpret_cast<const float2*>(rqt + 2 * (16 * mt + g + 8));
                        float S[4];
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            S[i] = tc_cell<CVUNIF>(acc[0][i], acc[1][i], acc[2][i], i < 2 ? rq0.x : rq1.x,
                                                   i < 2 ? rq0.y : rq1.y, cd[i & 1], pd[i & 1], cvl, tc);
                        if (hasc) {
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const int rr = P1_ROWS * s + 16 * mt + g + 8 * (i >> 1), cc = k0 + 2 * q + (i & 1);
                                // (padding columns past L and rows past the query keep -inf)
                                if (cc < L && rr < Lq && (cc <= corner_a(rr, Lq, edge) || cc >= corner_b(rr, L, edge)))
                                    S[i] = -9.f;
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 4; i++) ring[(wnext[i] ? sg[mt + 1] : sg[mt]) + woff[i] + 16 * mt] = S[i];
                    }
                } else {
                    // past the last column: scores of -inf for the lanes still
                    // to finish the matrix (the lane's rows, anti-diagonals
                    // lane .. lane + 7 past the chunk's first)
                    int w = sg[0] / P1_RLD + lane;
#pragma unroll
                    for (int c = 0; c < P1_C; c++) {
                        if (w >= P1_SLOTS) w -= P1_SLOTS;
                        *reinterpret_cast<float2*>(ring + w * P1_RLD + 2 * lane) = make_float2(-INFINITY, -INFINITY);
                        w++;
                    }
                }
                cp_async_wait_all();
                __syncwarp();
                // ---- DP stage: wavefront steps [k0, k0 + 8)
                const float* rp = ring + sg[0] + 2 * lane;
                const float* tcol = cring + cl * P1C_TRS;
                if (k0 < 32) {
                    Wf2Edge E;
                    wf2_edge(E, D, a.qrec, r0, Lq);
#pragma unroll 1
                    for (int u0 = 0; u0 < P1_C; u0 += 4)
                        wf2_steps4<true>(D, E, rp + u0 * P1_RLD, tcol + u0 * P1C_TRS, bnd, u0, k0 + u0 - lane, k0 + u0,
                                         lane, wr_bot);
                } else {
                    Wf2Edge E;
#pragma unroll 1
                    for (int u0 = 0; u0 < P1_C; u0 += 4)
                        wf2_steps4<false>(D, E, rp + u0 * P1_RLD, tcol + u0 * P1C_TRS, bnd, u0, k0 + u0 - lane, k0 + u0,
                                          lane, wr_bot);
                }
                __syncwarp();
                if (s + 1 < nstrips) {
                    p1_row_flush(bnd + P1_BND, botw, ldb, k0, L, lane);
                    // columns up to k0 - 24 are there: published every other chunk
                    if (it.pi >= 0 && k0 >= 24 && ((m & 1) || k0 + P1_C >= kend))
                        p1_publish(a, it, s, min(k0 - 23, L), lane);
                }
                // next chunk: rotate the ring segments and record slots; chunk
                // m + 2's records into slots no longer read
                const int t0 = sg[0];
#pragma unroll
                for (int i = 0; i < 4; i++) sg[i] = sg[i + 1];
                sg[4] = t0;
                cs = cs + P1_C >= P1_CMOD ? 0 : cs + P1_C;
                cl = cl + P1_C >= P1_CMOD ? cl + P1_C - P1_CMOD : cl + P1_C;
                stage_cols(cring, cold, m + 2, cs + P1_C >= P1_CMOD ? 0 : cs + P1_C, L, lane);
                __syncwarp();
            }
            cp_async_wait_all();
            {
                const int rr = r0 + D.brow, cc = D.kbest - lane;
                if (D.best > 0.f && (D.best > pbest || (D.best == pbest && (rr < prow || (rr == prow && cc < pcol))))) {
                    pbest = D.best; prow = rr; pcol = cc;
                }
            }
            float* t = botr; botr = botw; botw = t;
            __syncwarp();
        }
        p1_result(a, it, nstrips, lane, pbest, prow, pcol);
    }
    if (tbroken) (void)mbar_wait(tbar, tpend);
    // every warp is past its last TMEM access: the allocating warp frees it
    tmem_fence_before();
    __syncthreads();
    if (wid == 0) {
        tmem_fence_after();
        tmem_dealloc(tmem_base, P1T_TMEM_COLS);
    }
}

// Warp butterfly sum as the reference's FinalizeDPPro reduction
// (src/libmycu/cudp/CuBatchDP_final.cu:254-260).
__device__ __forceinline__ float warp_butterfly(float v)
{
    v += __shfl_xor_sync(FULL, v, 16);
    v += __shfl_xor_sync(FULL, v, 8);
    v += __shfl_xor_sync(FULL, v, 4);
    v += __shfl_xor_sync(FULL, v, 2);
    v += __shfl_xor_sync(FULL, v, 1);
    return v;
}

// DP finalisation, one warp per candidate pair
// (src/libmycu/cudp/CuBatchDP_final.cu:170-290).  The walk from the maximum is a
// serial chain; the warp stages 32 x 32 windows of the codes and scores in
// shared memory for it (reading each cell from global memory took 0.3 ms on
// paths of 300 steps).
constexpr int FINW = 4;   // warps per CTA

__global__ void __launch_bounds__(FINW * 32) fin_kernel(FinArgs a)
{
    __shared__ float cache[FINW][36];
    __shared__ signed char wbt[FINW][32][33];
    __shared__ float wsm[FINW][32][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int c = blockIdx.x * FINW + wid;
    if (c >= a.ncand) return;
    const int p = a.cand_prof[c];
    const int Lq = a.Lq;
    const int L = a.plen[p];
    const signed char* bt = a.btck + a.cand_off[c];
    const float* sm = a.smat + a.cand_off[c];
    float* ch = cache[wid];
    // maximum and end cell from the traceback sweep (FP32 scores)
    const unsigned long long key = a.tbkey[c];
    const float maxsc = __uint_as_float((unsigned)(key >> 32));
    const unsigned cell = 0xffffffffu - (unsigned)(key & 0xffffffffu);
    const unsigned xx = (key != 0ull) ? (((cell & 0xffffu) << 16) | (cell >> 16)) : 0u;
    // ... which must reproduce the phase-1 maximum of this pair (exactly when
    // phase 1 used the same FP32 scores, within tol after BF16 scores)
    if (lane == 0 && a.status) {
        const float pb = a.best[p];
        const bool ok = (a.tol == 0.f) ? (maxsc == pb && xx == a.coords[p]) : (fabsf(maxsc - pb) <= a.tol * fmaxf(1.f, pb));
        if (!ok) atomicCAS(a.status, 0, 2);
    }
    int x = (int)(xx >> 16), y = (int)(xx & 0xffff);
    int psts = 0;
    int ndx = 4;          // next slot of the chunk: slots 4..35, the last four of the chunk before in 0..3
    float sum = 0.f;
    if (lane < 4) ch[lane] = 0.f;
    // the walk is bounded by the number of cells on any monotone path
    int guard = Lq + L + 2;
    int stop = 0, x0 = 0, y0 = 0;
    bool staged = false;
    while (!stop) {
        if (!staged && x >= 0 && y >= 0) {
            x0 = x;
            y0 = y;
            const int qy = y0 - lane;
            __syncwarp();
#pragma unroll 16
            for (int i = 0; i < 32; i++) {
                const int cc = x0 - i;
                signed char b = (signed char)BT_STOP;
                float v = 0.f;
                if (cc >= 0 && qy >= 0) {
                    const long long k = (long long)cc * Lq + qy;
                    b = bt[k];
                    v = sm[k];
                }
                wbt[wid][i][lane] = b;
                wsm[wid][i][lane] = v;
            }
            staged = true;
        }
        __syncwarp();
        int left = 0;     // the walk left the window
        if (lane == 0) {
            while (ndx < 36) {
                if (x < 0 || y < 0) { stop = 1; break; }
                const int dx = x0 - x, dy = y0 - y;
                if (dx >= 32 || dy >= 32) { left = 1; break; }
                if (--guard < 0) { stop = 1; break; }
                const int b = wbt[wid][dx][dy];
                if (b == BT_STOP) { stop = 1; break; }
                if (b == BT_UP) { y--; continue; }
                if (b == BT_LEFT) { x--; continue; }
                const float v = wsm[wid][dx][dy];
                ch[ndx] = v;
                if (v > 0.f) psts++;
                x--; y--;
                ndx++;
            }
        }
        __syncwarp();
        x = __shfl_sync(FULL, x, 0);
        y = __shfl_sync(FULL, y, 0);
        ndx = __shfl_sync(FULL, ndx, 0);
        stop = __shfl_sync(FULL, stop, 0);
        if (__shfl_sync(FULL, left, 0)) staged = false;
        if (stop || ndx == 36) {
            float cs = 0.f;
            if (!(ndx <= lane + 4))
                cs = ch[lane + 4] * (((ch[lane] + ch[lane + 1]) + ch[lane + 2]) + ch[lane + 3]);
            sum += warp_butterfly(cs);
            const float keep = lane < 4 ? ch[32 + lane] : 0.f;
            __syncwarp();
            if (lane < 4) ch[lane] = keep;
            ndx = 4;
            __syncwarp();
        }
    }
    if (lane == 0) {
        sum *= 0.5f;
        sum = sum < 0.f ? -sqrtf(-sum) : sqrtf(sum);
        const float sc = maxsc + sum;
        a.score[c] = sc;
        a.psts[c] = psts;
        a.beg[c] = ((unsigned)(x + 1) << 16) | ((unsigned)(y + 1) & 0xffffu);
        a.endc[c] = xx;
        a.passed[c] = (a.scorethld < maxsc && a.scorethld < sc) ? 1 : 0;
    }
}

// ---------------------------------------------------------------------------
// launchers (host)
// A kernel's largest dynamic shared memory.  The attribute is the kernel's, shared
// by all threads: set to the size at the largest CV map the layout takes, whatever
// the call's own, or a thread's launch could find a smaller one set by another in
// between.
template <typename K>
static cudaError_t set_smem_max(K* kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

size_t p1t_smem_bytes(int cvcard)
{
    return (size_t)(cvcard * P1T_CVREP + P1T_WARPS * P1T_WARP_FLOATS) * sizeof(float);
}

int p1t_blocks_per_sm(int cvcard, cudaError_t* err)
{
    int n = 0;
    const size_t sm = p1t_smem_bytes(cvcard);
    cudaError_t e = set_smem_max(p1t_kernel<true>, p1t_smem_bytes(P1T_MAX_CVCARD));
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, p1t_kernel<true>, P1T_WARPS * 32, sm);
    if (err) *err = e;
    return n;
}

cudaError_t launch_tc_pack(const float* drec, const long long* poff, const int* plen, const long long* ttile,
                           int nprof, unsigned* tcdb, float* cold, float lok, float wss, cudaStream_t st)
{
    if (nprof <= 0) return cudaSuccess;
    tc_pack_kernel<<<nprof, 128, 0, st>>>(drec, poff, plen, ttile, tcdb, cold, lok, wss);
    return cudaGetLastError();
}

size_t p1c_smem_bytes(int cvcard)
{
    return (size_t)(cvcard * P1C_CVREP + P1C_WARPS * P1C_WARP_FLOATS) * sizeof(float);
}

int p1c_blocks_per_sm(int cvcard)
{
    int n = 0;
    const size_t sm = p1c_smem_bytes(cvcard);
    if (set_smem_max(p1c_kernel<false>, p1c_smem_bytes(MAX_CVCARD)) != cudaSuccess) return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, p1c_kernel<false>, P1C_WARPS * 32, sm);
    return n;
}

size_t p1_smem_bytes(int cvcard)
{
    return (size_t)(cvcard * 32 + P1_WARPS * P1_WARP_FLOATS) * sizeof(float);
}

size_t p2s_smem_bytes(int cvcard)
{
    return (size_t)(cvcard * P1TC_CVREP + P2S_WARPS * P2S_WARP_FLOATS) * sizeof(float);
}

cudaError_t launch_p1(const P1Args& a, const float* qbkg, int which, int grid, cudaStream_t st)
{
    cudaError_t e;
    if (which == P1K_TENSOR) {
        const size_t sm = p1t_smem_bytes(a.sc.cvcard);
        auto* k = a.tc.uniform ? p1t_kernel<true> : p1t_kernel<false>;
        if ((e = set_smem_max(k, p1t_smem_bytes(P1T_MAX_CVCARD))) != cudaSuccess) return e;
        k<<<grid, P1T_WARPS * 32, sm, st>>>(a, qbkg);
        return cudaGetLastError();
    }
    if (which == P1K_CHUNKED) {
        const size_t sm = p1c_smem_bytes(a.sc.cvcard);
        auto* k = a.tc.uniform ? p1c_kernel<true> : p1c_kernel<false>;
        if ((e = set_smem_max(k, p1c_smem_bytes(MAX_CVCARD))) != cudaSuccess) return e;
        k<<<grid, P1C_WARPS * 32, sm, st>>>(a, qbkg);
        return cudaGetLastError();
    }
    const size_t sm = p1_smem_bytes(a.sc.cvcard);
    if (which == P1K_TRACEBACK) {
        // the score matrices first (their own work counter, a.counter[1]),
        // then the sweep over them
        const size_t sms = p2s_smem_bytes(a.sc.cvcard);
        auto* k2 = a.tc.uniform ? p2s_kernel<true> : p2s_kernel<false>;
        if ((e = set_smem_max(k2, p2s_smem_bytes(std::min(MAX_CVCARD, P1TC_MAX_CVCARD)))) != cudaSuccess) return e;
        int occ = 0;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k2, P2S_WARPS * 32, sms)) != cudaSuccess)
            return e;
        int dev = 0, nsm = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        const long long nit2 = (long long)a.nwork * ((a.Lq + 31) / 32), nit = nit2 * a.p2s_blocks;
        const int gs = (int)std::min<long long>((long long)std::max(occ, 1) * nsm, (nit + P2S_WARPS - 1) / P2S_WARPS);
        k2<<<gs, P2S_WARPS * 32, sms, st>>>(a, qbkg);
        // one CTA per SM, of fewer warps where there are few (candidate, strip)
        // items, so that they spread over all SMs
        const int wt = (int)std::max<long long>(1, std::min<long long>(P1TC_WARPS, (nit2 + nsm - 1) / nsm));
        const int gt = (int)std::min<long long>(nsm, (nit2 + wt - 1) / wt);
        const size_t smt = (size_t)wt * P1TC_WARP_FLOATS * sizeof(float);
        if ((e = set_smem_max(p1tc_kernel, P1TC_WARPS * P1TC_WARP_FLOATS * sizeof(float))) != cudaSuccess) return e;
        p1tc_kernel<<<gt, wt * 32, smt, st>>>(a, qbkg);
    } else {
        if ((e = set_smem_max(p1_kernel, p1_smem_bytes(MAX_CVCARD))) != cudaSuccess) return e;
        p1_kernel<<<grid, P1_WARPS * 32, sm, st>>>(a, qbkg);
    }
    return cudaGetLastError();
}

int p1_blocks_per_sm(int cvcard)
{
    int n = 0;
    const size_t sm = p1_smem_bytes(cvcard);
    if (set_smem_max(p1_kernel, p1_smem_bytes(MAX_CVCARD)) != cudaSuccess) return 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, p1_kernel, P1_WARPS * 32, sm);
    return n > 0 ? n : 1;
}

cudaError_t launch_fin(const FinArgs& a, cudaStream_t st)
{
    if (a.ncand <= 0) return cudaSuccess;
    fin_kernel<<<(a.ncand + FINW - 1) / FINW, FINW * 32, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace c2
