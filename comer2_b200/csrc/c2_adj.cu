// c2_adj.cu -- differentiable alignment: log-partition of the MAP forward
// model over (query, db profile) pairs and its adjoint.
//
// No counterpart in the reference, whose forward-backward (cumapdp/) only
// feeds the MAP alignment.  The model is the reference's MAP forward
// recursion (src/libmycu/cumapdp/CuBatchMAPDP_fwd.cu:72-478: five states,
// query and db transition log-probabilities, the column -1 states of its
// 32-row blocks, a local start term log 1 in the MM state) evaluated with
// true exponentials and logarithms (the hardware base-2 forms, relative
// error ~1e-7 at these arguments; the reference's MAP stage uses coarse
// approximations instead) over the score matrix
//     S = s0 + wss * ss + wcv * cv
// (amino-acid score, and the SS and context-vector terms before their
// weights), with seven offsets theta (MM MI MD IM II DM DD) added to the query
// transitions of every cell update.  logZ = log sum over cells exp(F.MM).
// The backward sweep is the transposed recursion (outside values B, with the
// local end term in MM), so exp(F + B - logZ) is a state posterior and every
// edge posterior exp(F(pred) + edge + B(succ) - logZ) is a derivative of
// logZ.  Gradients: dlogZ/dS per cell (the MM emission edges), dlogZ/dtheta
// (edges by the query transition they use), dlogZ/dwss and dlogZ/dwcv.
//
// Layout and schedule.  Per-cell arrays (scores, dlogZ/dS, posteriors) are
// in wavefront order (c2_adj.cuh).  Both sweeps run one strip of 32 query
// rows of one pair per warp, strips handed out by a global counter in the
// order of their dependencies (all pairs' strip 0, then strip 1, ...; the
// backward sweep from the last strip up), so a pair is swept by up to
// nstrips warps at once, each trailing the strip it depends on by about 40
// columns (row hand-off with bounded waits, c2_device.cuh).
// Memory: the forward sweep keeps the last row of every strip (5 states x L
// per strip, the rows the next strip reads) and each strip's partial log-sum,
// and, when they fit (20 bytes a cell), every forward state.  The backward
// sweep takes its strip's forward states from there, or -- checkpointing,
// when they did not fit -- recomputes them from the checkpoint row above into
// a per-warp scratch (32 rows x (L + 31) x 5 states); it then runs the
// outside recursion over the same rows (bottom row first) and forms every
// edge posterior of the strip as it goes.  When the states were kept and there is
// as much room again, the backward sweep only stores its outside values B, and
// a kernel over all cells forms the posteriors: the chain of steps, which bounds
// the sweep, is then as short as the forward one's.  With checkpointing neither F
// nor B is stored for the matrix: memory per cell is then the 3 score arrays and
// the 2 outputs.
#include <cuda_runtime.h>

#include <algorithm>

#include "c2_adj.cuh"

namespace c2 {

#define FULL 0xffffffffu
constexpr float XLOG0 = -99.f;   // the MAP model's log 0

struct X5 { float MM, MI, IM, DN, ND; };

// e^x through the hardware base-2 form (denormal results and arguments flushed:
// the terms they drop are below e^-87 of the largest term of a sum); log2 x, whose
// factor ln 2 goes into the addition of the maximum.  (States kept in base 2
// need neither factor, but are 1.44 times as large: the same time, and gradients
// up to 1.2 times as far from the 64-bit ones.)
constexpr float XLOG2E = 1.4426950408889634f, XLN2 = 0.6931471805599453f;
__device__ __forceinline__ float xexp(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * XLOG2E));
    return y;
}
__device__ __forceinline__ float xlog2(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// the larger term's exponential is ex2(0) = 1 exactly, the smaller one's
// difference exactly -|a - b|
__device__ __forceinline__ float xlse2(float a, float b)
{
    const float m = fmaxf(a, b);
    return fmaf(xlog2(1.f + xexp(-fabsf(a - b))), XLN2, m);
}

// log(e^v1 + ... + e^v5 + 1): the 1 is the local start (forward) or end (backward)
__device__ __forceinline__ float xlse5p1(float v1, float v2, float v3, float v4, float v5)
{
    float m = fmaxf(fmaxf(fmaxf(v1, v2), fmaxf(v3, v4)), fmaxf(v5, 0.f));
    return fmaf(xlog2(((xexp(v1 - m) + xexp(v2 - m)) + (xexp(v3 - m) + xexp(v4 - m))) + (xexp(v5 - m) + xexp(-m))), XLN2, m);
}

// transitions of position i of a profile whose raw rows start at t0: the
// forward recursion's (MM MD IM DM DD into i, MI II out of i) and the
// backward's (all out of i); log 0 outside [0, len)
__device__ __forceinline__ void xtrn_fwd(const float* __restrict__ t0, int i, int len, float* t7)
{
    if (i < 0 || i >= len) {
        for (int k = 0; k < 7; k++) t7[k] = XLOG0;
        return;
    }
    const float* a = t0 + (long long)i * 7;
    t7[TMM] = a[0]; t7[TMI] = a[7 + 1]; t7[TMD] = a[2];
    t7[TIM] = a[3]; t7[TII] = a[7 + 4]; t7[TDM] = a[5]; t7[TDD] = a[6];
}

__device__ __forceinline__ void xtrn_bwd(const float* __restrict__ t0, int i, int len, float* t7)
{
    if (i < 0 || i >= len) {
        for (int k = 0; k < 7; k++) t7[k] = XLOG0;
        return;
    }
    const float* b = t0 + (long long)(i + 1) * 7;
    for (int k = 0; k < 7; k++) t7[k] = b[k];
}

// ---------------------------------------------------------------------------
// score parts per cell: one warp per (pair, strip), lane = query row, the
// strip's wavefront steps in turn (coalesced stores).  The db records the lanes
// read (the 46 score fields of 32 consecutive columns per step) are staged per
// 32-column chunk in a shared ring of 64 columns, ADJ_REC floats apart: an odd
// number of 16-byte units, so that the lanes' 16-byte reads of consecutive
// columns share no bank (12 reads a cell instead of 46 single ones), and the SS
// term reads a table of the strip's rows instead of nine global entries a cell:
// 0.72 -> 0.54 ms on 256 pairs of 100..600 positions.
constexpr int ADJ_REC = 52, ADJ_RECF = 48;
constexpr int ADJ_SCORE_FLOATS = 64 * ADJ_REC + MAX_SSSS_CARD * 32;   // per warp: record ring, SS row table

__device__ __forceinline__ void adj_stage_records(float* ring, const float* __restrict__ d0, int c0, int L, int lane)
{
    const int nc = min(32, L - c0);
    for (int e = lane; e < nc * (ADJ_RECF / 4); e += 32) {
        const int c = e / (ADJ_RECF / 4), f = e - c * (ADJ_RECF / 4);
        *reinterpret_cast<float4*>(ring + ((c0 + c) & 63) * ADJ_REC + 4 * f) =
            __ldg(reinterpret_cast<const float4*>(d0 + (long long)(c0 + c) * DR_STRIDE) + f);
    }
}

__global__ void __launch_bounds__(ADJ_WARPS * 32) adj_score_kernel(AdjArgs a)
{
    extern __shared__ __align__(16) float adjsm[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* ring = adjsm + wid * ADJ_SCORE_FLOATS;
    float* U = ring + 64 * ADJ_REC;   // [card][32] SS table of the strip's rows
    const int nw = gridDim.x * ADJ_WARPS;
    const ScoreConsts& sc = a.sc;
    const int card = sc.ssss_card;
    for (int it = blockIdx.x * ADJ_WARPS + wid; it < a.nitems; it += nw) {
        const int2 ms = a.items_f[it];
        const int m = ms.x, s = ms.y;
        const int p = a.prof[m];
        const int L = a.plen[p], Lq = a.pLq[m];
        const int r = 32 * s + lane;
        const bool act = r < Lq;
        const float* qr = a.qrec + (a.qpos[m] + (act ? r : 0)) * QR_STRIDE;
        const float* bd = a.pbkg + (long long)p * NAA;
        const float* qb = a.qbkg + (long long)a.qidx[m] * NAA;
        // the query row's amino-acid odds for this pair, CV vector and SS values
        float qt[NAA], qc[NCV + 1];
#pragma unroll
        for (int k = 0; k < NAA; k++) qt[k] = __fdividef(qr[QR_TRG + k], 0.5f * (qb[k] + bd[k]));
#pragma unroll
        for (int k = 0; k < NCV; k++) qc[k] = qr[QR_CV + k];
        const float qcn = qr[QR_CN], qpr = qr[QR_PRIOR], qhq = qr[QR_HQ];
        const float q0 = qr[QR_SS], q1 = qr[QR_SS + 1], q2 = qr[QR_SS + 2];
        const int i0 = (int)(q0 * 9.999f), i1 = 10 + (int)(q1 * 9.999f), i2 = 20 + (int)(q2 * 9.999f);
        const long long cb = a.off[m] + (long long)s * (L + 31) * 32;
        const float* d0 = a.drec + a.poff[p] * DR_STRIDE;
        __syncwarp();
        for (int c = 0; c < card; c++)
            U[c * 32 + lane] = q0 * a.ssss[i0 * card + c] + q1 * a.ssss[i1 * card + c] + q2 * a.ssss[i2 * card + c];
        adj_stage_records(ring, d0, 0, L, lane);
        __syncwarp();
        for (int k = 0; k < L + 31; k++) {
            const int j = k - lane;
            if (act && j >= 0 && j < L) {
                const float4* dr = reinterpret_cast<const float4*>(ring + (j & 63) * ADJ_REC);
                float sa = 0.f;
#pragma unroll
                for (int t = 0; t < NAA / 4; t++) {
                    const float4 v = dr[t];
                    sa = fmaf(qt[4 * t], v.x, sa);
                    sa = fmaf(qt[4 * t + 1], v.y, sa);
                    sa = fmaf(qt[4 * t + 2], v.z, sa);
                    sa = fmaf(qt[4 * t + 3], v.w, sa);
                }
                const float s0 = __logf(sa) - sc.shift;
                float dot = 0.f, dcn = 0.f;
#pragma unroll
                for (int t = 0; t < 5; t++) {
                    const float4 v = dr[DR_CV / 4 + t];
                    dot = fmaf(qc[4 * t], v.x, dot);
                    dot = fmaf(qc[4 * t + 1], v.y, dot);
                    dot = fmaf(qc[4 * t + 2], v.z, dot);
                    if (t < 4) dot = fmaf(qc[4 * t + 3], v.w, dot);
                    else dcn = v.w;   // DR_CN
                }
                dot += sc.lokappa0;
                const float4 v10 = dr[DR_PRIOR / 4], v11 = dr[DR_SSIDX / 4];   // prior, SS; indices, P(H) + 0.1
                const float det = qcn * dcn - dot * dot;
                const float cvs = sc.cterm + sc.pownu0 * __logf(det) - qpr - v10.x;
                float cvm;
                if (cvs <= sc.cvkey_first) cvm = sc.cvval_first;
                else if (sc.cvkey_last <= cvs) cvm = sc.cvval_last;
                else cvm = a.cvvals[min(max(sc.cvshift + (int)rintf(2.f * cvs), 0), sc.cvcard - 1)];
                const int pk = __float_as_int(v11.x);
                float ss = 0.f;
                ss = fmaf(v10.y, U[(pk & 0xff) * 32 + lane], ss);
                ss = fmaf(v10.z, U[((pk >> 8) & 0xff) * 32 + lane], ss);
                ss = fmaf(v10.w, U[((pk >> 16) & 0xff) * 32 + lane], ss);
                if (-99.f < ss) {
                    ss += qhq * v11.y * 0.1111111f;
                    ss -= 0.05f;
                }
                const long long c = cb + (long long)k * 32 + lane;
                const float p0 = s0, pss = ss, pcv = cvm;
                a.S[c] = (p0 + a.wss * pss + a.wcv * pcv);
                a.pss[c] = pss;
                a.pcv[c] = pcv;
            }
            if ((k & 31) == 31) {
                // columns of the next chunk into the slots of the chunk before this one
                __syncwarp();
                if (k + 1 < L) adj_stage_records(ring, d0, k + 1, L, lane);
                __syncwarp();
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Row of a strip's neighbour, ADJ_RG columns at a time in two groups of the
// warp's shared buffer (row hand-off, c2_device.cuh).  Forward: row 32 s - 1
// (frow of strip s - 1); backward: row 32 s + 32 (brow of strip s + 1) by
// mirrored column.
constexpr int ADJ_RG = 8;


// The forward sweep starts a group's copy a group before its use (two buffers;
// 1.12 -> 0.85 ms on 256 pairs).
__device__ __forceinline__ void adj_row_init(const AdjArgs& a, float* rab, const float* __restrict__ row, int ldr, bool have,
                                             int L, int lane, bool& broken)
{
    if (have) {
        row_issue<ADJ_RG>(rab, row, ldr, 0, L, lane);
        row_take<ADJ_RG>(rab, row, ldr, 0, L, lane, a.status, broken, a.spin);
        if (ADJ_RG < L) row_issue<ADJ_RG>(rab + ROW_BUF<ADJ_RG>, row, ldr, ADJ_RG, L, lane);
    } else if (lane < 2 * ADJ_RG) {
        float* o = rab + (lane < ADJ_RG ? 0 : ROW_BUF<ADJ_RG>);
        *reinterpret_cast<float4*>(o + 4 * (lane % ADJ_RG)) = make_float4(0.f, XLOG0, XLOG0, XLOG0);
        o[4 * ADJ_RG + lane % ADJ_RG] = XLOG0;
    }
    __syncwarp();
}

// column k of the row for lane 0; after a group's last column the next group is
// taken and the one after it started
__device__ __forceinline__ void adj_row_step(const AdjArgs& a, float* rab, const float* __restrict__ row, int ldr, bool have,
                                             int k, int L, int lane, bool& broken, X5& up)
{
    const float* b = rab + (k & ADJ_RG ? ROW_BUF<ADJ_RG> : 0);
    const int u = k & (ADJ_RG - 1);
    const float4 ba = *reinterpret_cast<const float4*>(b + 4 * u);
    const float b4 = b[4 * ADJ_RG + u];
    if (lane == 0) up = X5{ba.x, ba.y, ba.z, ba.w, b4};
    if (u == ADJ_RG - 1 && have) {
        const int c0 = k + 1;
        if (c0 < L) row_take<ADJ_RG>(rab + (c0 & ADJ_RG ? ROW_BUF<ADJ_RG> : 0), row, ldr, c0, L, lane, a.status, broken, a.spin);
        if (c0 + ADJ_RG < L)
            row_issue<ADJ_RG>(rab + (c0 & ADJ_RG ? 0 : ROW_BUF<ADJ_RG>), row, ldr, c0 + ADJ_RG, L, lane);
    }
}

// The backward sweep, whose steps are longer than a trip through L2, fetches a
// group when it needs it, into rab[32][8] (slot c & 31); started a group earlier,
// every strip trails 8 columns further (2.0 -> 2.2 ms on 256 pairs).
__device__ __forceinline__ void adj_load_row(const AdjArgs& a, float* rab, const float* __restrict__ row, int ldr, bool have,
                                             int c0, int L, int lane, bool& broken)
{
    const int c = c0 + lane;
    float v[5] = {0.f, XLOG0, XLOG0, XLOG0, XLOG0};
    if (have && c0 < L) row_get(row, ldr, c, lane < ADJ_RG && c < L, v, lane, a.status, broken, a.spin);
    if (lane < ADJ_RG) {
        float* o = rab + (c & 31) * 8;
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
        o[4] = v[4];
    }
    __syncwarp();
}

// Transition rows of a pair's db profile (rows 0..L; row r holds the
// transitions into position r, MI and II of row r + 1 those out of position
// r) in the warp's shared ring trs[128][TRS] by sequence index q: q = row in the
// forward sweep, q = L - row in the mirrored backward sweep.  A step's lanes
// read rows q in [k - 31, k + 1]; chunks of 32 are staged two ahead.  Rows are 12
// floats apart: 16-byte reads of consecutive rows share no bank.  (Rows outside
// the profile hold what the ring does: only cells outside the matrix read them,
// and no cell inside reads those.)
constexpr int TRS = 12;
template <bool MIRROR>
__device__ __forceinline__ void adj_stage_trn(float* trs, const float* __restrict__ dt0, int q0, int L, int lane)
{
    const int nq = min(32, L + 1 - q0);
    for (int e = lane; e < nq * 7; e += 32) {
        const int q = q0 + e / 7, f = e % 7;
        const int row = MIRROR ? L - q : q;
        trs[(q & 127) * TRS + f] = __ldg(dt0 + (long long)row * 7 + f);
    }
}

// row q of a ring of N rows
template <int N = 128>
__device__ __forceinline__ void ring_row(const float* trs, int q, float* t)
{
    const float* o = trs + (q & (N - 1)) * TRS;
    const float4 a = *reinterpret_cast<const float4*>(o);
    const float4 b = *reinterpret_cast<const float4*>(o + 4);
    t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = a.w; t[4] = b.x; t[5] = b.y; t[6] = b.z;
}

// forward transitions of column j (rows j and j + 1) from the forward ring
__device__ __forceinline__ void ring_trn_fwd(const float* trs, int j, float* t7)
{
    ring_row(trs, j, t7);
    const float* b = trs + ((j + 1) & 127) * TRS;
    t7[TMI] = b[1];
    t7[TII] = b[4];
}

// Forward states of a strip's cells: [step][lane][4] MM MI IM DN, then [lane] ND
// (160 floats a step: two reads or writes a cell)
__device__ __forceinline__ void fw_st5(float* __restrict__ Fw, int k, int l, const X5& x)
{
    float* o = Fw + (long long)k * 160;
    reinterpret_cast<float4*>(o)[l] = make_float4(x.MM, x.MI, x.IM, x.DN);
    o[128 + l] = x.ND;
}
__device__ __forceinline__ X5 fw_ld5(const float* __restrict__ Fw, int k, int l)
{
    const float* o = Fw + (long long)k * 160;
    const float4 a = reinterpret_cast<const float4*>(o)[l];
    return X5{a.x, a.y, a.z, a.w, o[128 + l]};
}

// L1 prefetch of one 128-byte line (the lines a sweep reads a few steps
// ahead; the loads themselves then hit L1 instead of waiting on L2)
constexpr int ADJ_PF = 4;
__device__ __forceinline__ void pf_l1(const void* p)
{
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Forward recursion over strip s of pair m (lane = row 32 s + lane).
// RECOMP false (forward sweep): the row above comes from the strip above as
// it is swept; the strip's last row goes to frow (published for the strip
// below) and the lane's cells into the online log-sum (zm, zs).
// RECOMP true (backward sweep): the row above from the complete checkpoint,
// every state into the warp's scratch Fw (fw_st5).
template <bool RECOMP>
__device__ __forceinline__ void adj_fwd_strip(const AdjArgs& a, int m, int s, int lane, float* rab, float* trs,
                                              float* __restrict__ Fw, bool& broken, float& zm, float& zs)
{
    const int p = a.prof[m];
    const int L = a.plen[p], Lq = a.pLq[m], ns = (Lq + 31) >> 5;
    const long long cb = a.off[m] + (long long)s * (L + 31) * 32;
    const float* dt0 = a.dtrn + (a.poff[p] + p) * 7;
    const int ldr = row_ld(L);
    const float* above = a.frow + a.roff[m] + (long long)(s > 0 ? s - 1 : 0) * 5 * ldr;   // read when s > 0
    float* mine_row = a.frow + a.roff[m] + (long long)s * 5 * ldr;
    const int r = 32 * s + lane;
    const bool act = r < Lq;
    const X5 INIT = {0.f, XLOG0, XLOG0, XLOG0, XLOG0};
    float q7[7];
    xtrn_fwd(a.qtrn + (a.qpos[m] + a.qidx[m]) * 7, r, Lq, q7);
#pragma unroll
    for (int k = 0; k < 7; k++) q7[k] += a.theta[k];
    const float* cf = a.qcfx + (a.qpos[m] + (act ? r : 0)) * 6;
    const X5 LB = (lane == 31) ? INIT : X5{0.f, cf[0], cf[1], cf[2], XLOG0};
    const X5 DB = (lane == 31 || lane == 0) ? INIT : X5{0.f, cf[3], cf[4], cf[5], XLOG0};
    const bool wr_row = !RECOMP && lane == 31 && s + 1 < ns;
    X5 mine = INIT, upp = INIT;
    // the lane's score of the next step, loaded a step ahead
    float scn = (act && lane == 0 && L > 0) ? a.S[cb + lane] : XLOG0;
    __syncwarp();
    adj_stage_trn<false>(trs, dt0, 0, L, lane);
    adj_stage_trn<false>(trs, dt0, 32, L, lane);
    adj_row_init(a, rab, above, ldr, s > 0, L, lane, broken);
    for (int k = 0; k < L + 31; k++) {
        const int j = k - lane;
        float t7[7];
        ring_trn_fwd(trs, j, t7);
        X5 up;
        up.MM = __shfl_up_sync(FULL, mine.MM, 1);
        up.MI = __shfl_up_sync(FULL, mine.MI, 1);
        up.IM = __shfl_up_sync(FULL, mine.IM, 1);
        up.DN = __shfl_up_sync(FULL, mine.DN, 1);
        up.ND = __shfl_up_sync(FULL, mine.ND, 1);
        adj_row_step(a, rab, above, ldr, s > 0, k, L, lane, broken, up);
        if ((k & 31) == 31) {
            __syncwarp();
            if (k + 33 <= L) adj_stage_trn<false>(trs, dt0, k + 33, L, lane);
            __syncwarp();
        }
        X5 left = mine, diag = upp;
        if (j == 0) { left = LB; diag = DB; }
        if (lane == 0 && k + 2 * ADJ_PF < L + 31) pf_l1(a.S + cb + (long long)(k + 2 * ADJ_PF) * 32);
        const bool valid = act && j >= 0 && j < L;
        const float sc = valid ? scn : XLOG0;
        if (act && j + 1 >= 0 && j + 1 < L) scn = a.S[cb + (long long)(k + 1) * 32 + lane];
        X5 nw;
        // (a state is added last, to the sum of the step's own terms: one rounding
        // at the state's magnitude, and one addition in the chain of steps)
        nw.MM = xlse5p1(diag.MI + ((q7[TMM] + t7[TIM]) + sc), diag.IM + ((q7[TIM] + t7[TMM]) + sc),
                        diag.DN + ((q7[TDM] + t7[TMM]) + sc), diag.ND + ((q7[TMM] + t7[TDM]) + sc),
                        diag.MM + ((q7[TMM] + t7[TMM]) + sc));
        nw.MI = xlse2(up.MM + (q7[TMM] + t7[TMI]), up.MI + (q7[TMM] + t7[TII]));
        nw.IM = xlse2(left.MM + (q7[TMI] + t7[TMM]), left.IM + (q7[TII] + t7[TMM]));
        nw.DN = xlse2(up.MM + q7[TMD], up.DN + q7[TDD]);
        nw.ND = xlse2(left.MM + t7[TMD], left.ND + t7[TDD]);
        if (valid) {
            if (RECOMP || Fw) fw_st5(Fw, k, lane, nw);
            if (!RECOMP) {
                const float mx = fmaxf(zm, nw.MM);
                zs = fmaf(zs, xexp(zm - mx), xexp(nw.MM - mx));
                zm = mx;
            }
            if (wr_row) row_put(mine_row, ldr, j, nw.MM, nw.MI, nw.IM, nw.DN, nw.ND);
        }
        mine = nw;
        upp = up;
    }
}

// forward sweep: logZ partial sums per strip, checkpoint rows
__global__ void __launch_bounds__(ADJ_WARPS * 32) adj_fwd_kernel(AdjArgs a)
{
    __shared__ __align__(16) float rabs[ADJ_WARPS][2 * ROW_BUF<ADJ_RG>];
    __shared__ __align__(16) float trss[ADJ_WARPS][128 * TRS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    bool broken = false;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.counter, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= a.nitems) break;
        const int2 ms = a.items_f[item];
        const int m = ms.x, s = ms.y;
        float zm = -INFINITY, zs = 0.f;
        // the strip's forward states kept for the backward sweep when they fit
        float* Fw = a.Fall ? a.Fall + 5 * a.off[m] + (long long)s * (a.plen[a.prof[m]] + 31) * 160 : nullptr;
        adj_fwd_strip<false>(a, m, s, lane, rabs[wid], trss[wid], Fw, broken, zm, zs);
        // combine the lanes' (max, sum) pairs
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const float om = __shfl_xor_sync(FULL, zm, o), os = __shfl_xor_sync(FULL, zs, o);
            const float mx = fmaxf(zm, om);
            zs = (mx == -INFINITY) ? 0.f : zs * xexp(zm - mx) + os * xexp(om - mx);
            zm = mx;
        }
        if (lane == 0) {
            const long long o = a.soff[m] + s;
            a.zpart[2 * o] = zm;
            a.zpart[2 * o + 1] = zs;
        }
        __syncwarp();
    }
}

// logZ of each pair from its strips' partial sums, in strip order
__global__ void adj_logz_kernel(AdjArgs a)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= a.npairs) return;
    float zm = -INFINITY, zs = 0.f;
    const int ns = (a.pLq[m] + 31) >> 5;
    for (int s = 0; s < ns; s++) {
        const long long it = a.soff[m] + s;
        const float om = a.zpart[2 * it], os = a.zpart[2 * it + 1];
        const float mx = fmaxf(zm, om);
        zs = (mx == -INFINITY) ? 0.f : zs * xexp(zm - mx) + os * xexp(om - mx);
        zm = mx;
    }
    const float lz = logf(zs) + zm;
    a.logz[m] = lz;
    a.zpart[2 * a.soff[m]] = lz;   // for the backward sweep
}

// ---------------------------------------------------------------------------
// backward sweep and posteriors
__device__ __forceinline__ X5 shfl_up5(const X5& x)
{
    return X5{__shfl_up_sync(FULL, x.MM, 1), __shfl_up_sync(FULL, x.MI, 1), __shfl_up_sync(FULL, x.IM, 1),
              __shfl_up_sync(FULL, x.DN, 1), __shfl_up_sync(FULL, x.ND, 1)};
}
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// A strip's lines in up to POST_WARPS equal runs of at least 8 lines; gradient
// sums are taken over each run from its last line, and over the runs from the
// last one (in every form, so that they agree bit for bit)
constexpr int POST_WARPS = 8;
__device__ __forceinline__ int post_run(int lines) { return max(8, (lines + POST_WARPS - 1) / POST_WARPS); }

// Posteriors of a cell (array index kk) and of its incoming edges, from its
// outside values b and its forward predecessors; added to the gradient sums g.
__device__ __forceinline__ void edge_posteriors(const AdjArgs& a, long long kk, const X5& b, float ownMM, const X5& up,
                                                const X5& left, const X5& diag, const float* qf, const float* tf,
                                                float sc, float lz, float pss, float pcv, float* g)
{
    // (the predecessor's and the cell's states first: they nearly cancel)
    // MM: five emission edges
    const float eMM = b.MM - lz, eMI = b.MI - lz, eIM = b.IM - lz, eDN = b.DN - lz;
    const float m1 = xexp((diag.MI + eMM) + ((qf[TMM] + tf[TIM]) + sc));
    const float m2 = xexp((diag.IM + eMM) + ((qf[TIM] + tf[TMM]) + sc));
    const float m3 = xexp((diag.DN + eMM) + ((qf[TDM] + tf[TMM]) + sc));
    const float m4 = xexp((diag.ND + eMM) + ((qf[TMM] + tf[TDM]) + sc));
    const float m5 = xexp((diag.MM + eMM) + ((qf[TMM] + tf[TMM]) + sc));
    const float gs = (m1 + m2 + m3 + m4) + m5;
    // MI, IM, DN (ND uses no query transition)
    const float i1 = xexp((up.MM + eMI) + (qf[TMM] + tf[TMI]));
    const float i2 = xexp((up.MI + eMI) + (qf[TMM] + tf[TII]));
    const float l1 = xexp((left.MM + eIM) + (qf[TMI] + tf[TMM]));
    const float l2 = xexp((left.IM + eIM) + (qf[TII] + tf[TMM]));
    const float d1 = xexp((up.MM + eDN) + qf[TMD]);
    const float d2 = xexp((up.DN + eDN) + qf[TDD]);
    g[TMM] += m1 + m4 + m5 + i1 + i2;
    g[TIM] += m2;
    g[TDM] += m3;
    g[TMI] += l1;
    g[TII] += l2;
    g[TMD] += d1;
    g[TDD] += d2;
    g[7] += gs * pss;
    g[8] += gs * pcv;
    a.gS[kk] = gs;
    a.post[kk] = xexp(ownMM + eMM);
}

// column c of a complete row
__device__ __forceinline__ X5 row_ld5(const float* __restrict__ row, int ldr, int c)
{
    const float4 x = reinterpret_cast<const float4*>(row)[c];
    return X5{x.x, x.y, x.z, x.w, row[4 * ldr + c]};
}

// Backward sweep of a strip: lane t holds row i = 32 s + 31 - t (the strip's rows
// bottom first), mirrored column jm = k - t at step k, actual column
// ca = L - 1 - jm.  The outside values B follow the transposed recursion.  OUT:
// they are stored in Bw, in the forward states' layout.  Otherwise the posteriors
// of a cell's incoming edges exp(F(pred) + edge + B(cell) - logZ) are formed here,
// from the strip's forward states Fw and the checkpoint row above it.
template <bool OUT>
__device__ __forceinline__ void adj_bwd_strip(const AdjArgs& a, int m, int s, int lane, float* rab, float* trs,
                                              const float* __restrict__ Fw, float* __restrict__ Bw, bool& broken)
{
    const int p = a.prof[m];
    const int L = a.plen[p], Lq = a.pLq[m], ns = (Lq + 31) >> 5;
    const long long cb = a.off[m] + (long long)s * (L + 31) * 32;
    const float lz = a.zpart[2 * a.soff[m]];   // log Z
    const float* dt0 = a.dtrn + (a.poff[p] + p) * 7;
    const bool has_below = s + 1 < ns;
    const int ldr = row_ld(L);
    const float* below = a.brow + a.roff[m] + (long long)(has_below ? s + 1 : s) * 5 * ldr;   // read when has_below
    float* mine_row = a.brow + a.roff[m] + (long long)s * 5 * ldr;
    const float* fab = a.frow + a.roff[m] + (long long)(s > 0 ? s - 1 : 0) * 5 * ldr;   // row 32 s - 1 (s > 0)
    const int t = lane;
    const int lf = 31 - t;            // the lane's row within the strip
    const int i = 32 * s + lf;
    const bool act = i < Lq;
    const X5 INIT = {0.f, XLOG0, XLOG0, XLOG0, XLOG0};
    float qb[7], qf[7];
    const float* qt0 = a.qtrn + (a.qpos[m] + a.qidx[m]) * 7;
    xtrn_bwd(qt0, i, Lq, qb);
    xtrn_fwd(qt0, i, Lq, qf);
#pragma unroll
    for (int k = 0; k < 7; k++) { qb[k] += a.theta[k]; qf[k] += a.theta[k]; }
    // column -1 states of row i (the forward's left and diagonal at column 0)
    const float* cf = a.qcfx + (a.qpos[m] + (act ? i : 0)) * 6;
    const X5 LB = (lf == 31) ? INIT : X5{0.f, cf[0], cf[1], cf[2], XLOG0};
    const X5 DB = (lf == 31 || lf == 0) ? INIT : X5{0.f, cf[3], cf[4], cf[5], XLOG0};
    const bool wr_row = (t == 31) && s > 0;
    float g[9];
#pragma unroll
    for (int k = 0; k < 9; k++) g[k] = 0.f;
    int flush = (L + 30) / post_run(L + 31) * post_run(L + 31);   // first line of the current run
    float tot = 0.f;                                             // lane f < 9: the complete runs' sum of g[f]
    X5 mine = INIT, upp = INIT;
    __syncwarp();
    adj_stage_trn<true>(trs, dt0, 0, L, lane);
    adj_stage_trn<true>(trs, dt0, 32, L, lane);
    adj_load_row(a, rab, below, ldr, has_below, 0, L, lane, broken);
    // Forward states and scores of the lane's own row, one wavefront line a
    // step: at step k the lane's cell is on line kf = L + 30 - k, its left
    // neighbour on line kf - 1; the row above (lf - 1) is lane t + 1's, whose
    // line kf - 2 is the diagonal predecessor now and the one above at the next
    // step.  So a step loads one line of five states (20 loads a cell when each
    // neighbour was read from memory) and shuffles it.  Lane 31's row above is
    // the strip above's last row, the diagonal successor's score of lane 0 the
    // strip below's first.  Entries of cells outside the matrix are read but not used.
    const float* Sr = a.S + cb + lf;
    const float* Sb = a.S + cb + (long long)(L + 31) * 32;   // row 32 s + 32 (has_below), lane 0
    const int kf0 = L + 30;
    X5 Ac = INIT, Al = INIT, An = INIT, Up = INIT;
    if (!OUT) {
        Ac = fw_ld5(Fw, kf0, lf);
        Al = fw_ld5(Fw, kf0 - 1, lf);
        An = fw_ld5(Fw, kf0 - 2, lf);
    }
    X5 Ab = INIT;                              // lane 31: row 32 s - 1 at the diagonal column
    auto load_above = [&](int c) { return (!OUT && s > 0 && t == 31 && c >= 0 && c < L) ? row_ld5(fab, ldr, c) : INIT; };
    Ab = load_above(L - 1 + t - 1);            // step 0: ca - 1
    float sc0 = Sr[(long long)kf0 * 32], sc1 = 0.f, sc2 = 0.f, sb = XLOG0;   // scores at steps k, k - 1, k - 2; row below
    for (int k = 0; k < L + 31; k++) {
        const int jm = k - t;
        const int ca = L - 1 - jm;
        const int kf = L + 30 - k;
        {
            // lines of the steps to come: forward states (5), scores, SS and CV parts, row below
            const int kq = kf - ADJ_PF;
            if (kq >= 0) {
                if (!OUT && lane < 5 && kq >= 3) pf_l1(Fw + (long long)(kq - 3) * 160 + lane * 32);
                else if (lane == 5) pf_l1(a.S + cb + (long long)kq * 32);
                else if (!OUT && lane == 6) pf_l1(a.pss + cb + (long long)kq * 32);
                else if (!OUT && lane == 7) pf_l1(a.pcv + cb + (long long)kq * 32);
                else if (lane == 8 && has_below && L - k - ADJ_PF >= 0 && L - k - ADJ_PF < L)
                    pf_l1(Sb + (long long)(L - k - ADJ_PF) * 32);
            }
        }
        // loaded now for the next step: line kf - 3, the score, rows above and below
        X5 Aq = INIT;
        float scn = 0.f;
        if (!OUT && kf >= 3) Aq = fw_ld5(Fw, kf - 3, lf);
        if (kf >= 1) scn = Sr[(long long)(kf - 1) * 32];
        const X5 Abn = load_above(ca - 2);
        const float sbn = (t == 0 && has_below && ca >= 0 && ca < L) ? Sb[(long long)ca * 32] : XLOG0;   // column (ca - 1) + 1
        X5 dgl;   // diagonal predecessor: lane t + 1's line kf - 2
        dgl.MM = __shfl_down_sync(FULL, An.MM, 1);
        dgl.MI = __shfl_down_sync(FULL, An.MI, 1);
        dgl.IM = __shfl_down_sync(FULL, An.IM, 1);
        dgl.DN = __shfl_down_sync(FULL, An.DN, 1);
        dgl.ND = __shfl_down_sync(FULL, An.ND, 1);
        if (t == 31) dgl = Ab;
        const float scu = __shfl_up_sync(FULL, sc2, 1);   // score of (i + 1, ca + 1): lane t - 1 two steps ago
        // transitions out of column ca (row ca + 1, sequence index jm) and,
        // for the edge posteriors, into it (rows ca and ca + 1)
        float tb[7], tf[7];
        ring_row(trs, jm, tb);          // row ca + 1
        if (!OUT) ring_row(trs, jm + 1, tf);   // row ca
        tf[TMI] = tb[TMI];
        tf[TII] = tb[TII];
        X5 dn;
        dn.MM = __shfl_up_sync(FULL, mine.MM, 1);
        dn.MI = __shfl_up_sync(FULL, mine.MI, 1);
        dn.IM = __shfl_up_sync(FULL, mine.IM, 1);
        dn.DN = __shfl_up_sync(FULL, mine.DN, 1);
        dn.ND = __shfl_up_sync(FULL, mine.ND, 1);
        {
            const int src = k & 31;
            const float4 ba = *reinterpret_cast<const float4*>(rab + src * 8);
            const float b4 = rab[src * 8 + 4];
            if (lane == 0) dn = X5{ba.x, ba.y, ba.z, ba.w, b4};
            if ((src & (ADJ_RG - 1)) == ADJ_RG - 1) {
                __syncwarp();
                adj_load_row(a, rab, below, ldr, has_below, k + 1, L, lane, broken);
            }
            if (src == 31) {
                if (k + 33 <= L) adj_stage_trn<true>(trs, dt0, k + 33, L, lane);
                __syncwarp();
            }
        }
        X5 rt = mine, dg = upp;
        if (jm == 0) { rt = INIT; dg = INIT; }
        const bool valid = act && jm >= 0 && jm < L;
        // score of the diagonal successor (i + 1, ca + 1)
        const float sco = (valid && i + 1 < Lq && ca + 1 < L) ? (t == 0 ? sb : scu) : XLOG0;
        X5 nw;
        nw.MM = xlse5p1(dn.MI + (qb[TMM] + tb[TMI]), rt.IM + (qb[TMI] + tb[TMM]), dn.DN + qb[TMD],
                        rt.ND + tb[TMD], dg.MM + ((qb[TMM] + tb[TMM]) + sco));
        nw.MI = xlse2(dg.MM + ((qb[TMM] + tb[TIM]) + sco), dn.MI + (qb[TMM] + tb[TII]));
        nw.IM = xlse2(dg.MM + ((qb[TIM] + tb[TMM]) + sco), rt.IM + (qb[TII] + tb[TMM]));
        nw.DN = xlse2(dg.MM + ((qb[TDM] + tb[TMM]) + sco), dn.DN + qb[TDD]);
        nw.ND = xlse2(dg.MM + ((qb[TMM] + tb[TDM]) + sco), rt.ND + tb[TDD]);
        // rows past the query (the last strip's first lanes) are the matrix
        // edge for the rows above them
        if (!act) nw = INIT;
        if (OUT && valid) {
            fw_st5(Bw, kf, lf, nw);
            if (wr_row) row_put(mine_row, ldr, jm, nw.MM, nw.MI, nw.IM, nw.DN, nw.ND);
        }
        if (!OUT && valid) {
            // edge posteriors of cell (i, ca): its forward predecessors
            const X5 own = Ac, up = Up;
            X5 left = Al, diag = dgl;
            if (ca == 0) {
                left = LB;
                diag = DB;
            }
            const long long kk = cb + (long long)kf * 32 + lf;
            edge_posteriors(a, kk, nw, own.MM, up, left, diag, qf, tf, sc0, lz, a.pss[kk], a.pcv[kk], g);
            if (wr_row) row_put(mine_row, ldr, jm, nw.MM, nw.MI, nw.IM, nw.DN, nw.ND);
        }
        if (!OUT && kf == flush) {
            // a run of lines is complete (adj_post_kernel's order of summation)
#pragma unroll
            for (int f = 0; f < 9; f++) {
                const float v = warp_sum(g[f]);
                if (lane == f) tot += v;
                g[f] = 0.f;
            }
            flush -= post_run(L + 31);
        }
        mine = nw;
        upp = dn;
        Up = dgl;
        Ac = Al; Al = An; An = Aq;
        Ab = Abn;
        sc2 = sc1; sc1 = sc0; sc0 = scn;
        sb = sbn;
    }
    if (!OUT && lane < 9) a.gpart[(a.soff[m] + s) * 9 + lane] = tot;
}

// Bound by the chain of steps.  Three forms:
//  ADJ_OUT: the forward sweep kept its states (Fall) and there is room for the
//    outside values too (Ball): this sweep stores B, adj_post_kernel then forms the
//    posteriors of all cells at once.  The chain's step is ~110 instructions
//    instead of ~350.
//  ADJ_KEPT: room for Fall only.  Posteriors in the sweep, 12 warps an SM at 162
//    registers (16 at 128 were slower: 1.88 against 1.72 ms on 256 pairs of 100..600).
//  ADJ_RECOMP: Fall did not fit; the strip's forward states are computed again.
constexpr int ADJ_RECOMP = 0, ADJ_KEPT = 1, ADJ_OUT = 2;
template <int MODE>
__global__ void __launch_bounds__(ADJ_WARPS * 32, MODE == ADJ_OUT ? 5 : MODE == ADJ_KEPT ? 3 : 4) adj_bwd_kernel(AdjArgs a)
{
    __shared__ __align__(16) float rabs[ADJ_WARPS][32 * 8];
    __shared__ __align__(16) float trss[ADJ_WARPS][128 * TRS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* const scr = MODE == ADJ_RECOMP ? a.scratch + ((long long)blockIdx.x * ADJ_WARPS + wid) * a.scratch_stride : nullptr;
    bool broken = false;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.counter + 1, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= a.nitems) break;
        const int2 ms = a.items_b[item];
        const int m = ms.x, s = ms.y;
        const long long st5 = 5 * a.off[m] + (long long)s * (a.plen[a.prof[m]] + 31) * 160;   // the strip's states
        const float* Fw = nullptr;
        float* Bw = nullptr;
        if (MODE == ADJ_OUT) {
            Bw = a.Ball + st5;
        } else if (MODE == ADJ_KEPT) {
            Fw = a.Fall + st5;
        } else {
            // checkpointing: the strip's states again, from the row above
            float zm = 0.f, zs = 0.f;
            adj_fwd_strip<true>(a, m, s, lane, rabs[wid], trss[wid], scr, broken, zm, zs);
            Fw = scr;
        }
        __syncwarp();
        adj_bwd_strip<MODE == ADJ_OUT>(a, m, s, lane, rabs[wid], trss[wid], Fw, Bw, broken);
        __syncwarp();
    }
}

// Posteriors and gradient sums from stored F and B: one CTA per strip, one warp per
// run of its lines, from the last line of the run.  A line's cells lie on
// consecutive lanes; the left, upper and diagonal neighbours are on the two lines
// below it, kept in registers, the row above by shuffle.  Every line of F, B and the
// three score arrays is read once (the first two of a run twice) and the two
// outputs written: 60 bytes a cell, bound by DRAM on large batches.
__global__ void __launch_bounds__(POST_WARPS * 32) adj_post_kernel(AdjArgs a)
{
    __shared__ __align__(16) float trss[POST_WARPS][64 * TRS];
    __shared__ float gsh[POST_WARPS][9];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* trs = trss[wid];
    const int2 ms = a.items_b[blockIdx.x];
    const int m = ms.x, s = ms.y;
    const int p = a.prof[m];
    const int L = a.plen[p], Lq = a.pLq[m];
    const long long cb = a.off[m] + (long long)s * (L + 31) * 32;
    const float* Fw = a.Fall + 5 * a.off[m] + (long long)s * (L + 31) * 160;
    const float* Bw = a.Ball + 5 * a.off[m] + (long long)s * (L + 31) * 160;
    const float lz = a.zpart[2 * a.soff[m]];
    const float* dt0 = a.dtrn + (a.poff[p] + p) * 7;
    const int ldr = row_ld(L);
    const float* fab = a.frow + a.roff[m] + (long long)(s > 0 ? s - 1 : 0) * 5 * ldr;
    const int i = 32 * s + lane;
    const bool act = i < Lq;
    const X5 INIT = {0.f, XLOG0, XLOG0, XLOG0, XLOG0};
    float qf[7];
    xtrn_fwd(a.qtrn + (a.qpos[m] + a.qidx[m]) * 7, i, Lq, qf);
#pragma unroll
    for (int k = 0; k < 7; k++) qf[k] += a.theta[k];
    const float* cf = a.qcfx + (a.qpos[m] + (act ? i : 0)) * 6;
    const X5 LB = (lane == 31) ? INIT : X5{0.f, cf[0], cf[1], cf[2], XLOG0};
    const X5 DB = (lane == 31 || lane == 0) ? INIT : X5{0.f, cf[3], cf[4], cf[5], XLOG0};
    const int nl = L + 31, run = post_run(nl);
    const int k0 = wid * run, k1 = min(nl, k0 + run);
    float g[9];
#pragma unroll
    for (int f = 0; f < 9; f++) g[f] = 0.f;
    if (k0 < k1) {
        auto row_above = [&](int c) { return (s > 0 && lane == 0 && c >= 0 && c < L) ? row_ld5(fab, ldr, c) : INIT; };
        // lines k (own), k - 1 (left), and the row above at columns c and c - 1
        X5 own = fw_ld5(Fw, k1 - 1, lane);
        X5 left = k1 >= 2 ? fw_ld5(Fw, k1 - 2, lane) : INIT;
        X5 up = shfl_up5(left);
        if (lane == 0) up = row_above(k1 - 1);
        for (int ke = k1; ke > k0; ke -= 32) {
            // transition rows ke - 63 .. ke of the next 32 lines (row r at r & 63)
            __syncwarp();
            for (int e = lane; e < 64 * 7; e += 32) {
                const int row = ke - 63 + e / 7, f = e % 7;
                if (row >= 0 && row <= L) trs[(row & 63) * TRS + f] = __ldg(dt0 + (long long)row * 7 + f);
            }
            __syncwarp();
#pragma unroll 2
            for (int k = ke - 1; k >= max(k0, ke - 32); k--) {
                const int c = k - lane;
                const bool valid = act && c >= 0 && c < L;
                const long long kk = cb + (long long)k * 32 + lane;
                const X5 nx = k >= 2 ? fw_ld5(Fw, k - 2, lane) : INIT;
                const X5 b = fw_ld5(Bw, k, lane);
                const float sc = a.S[kk], ps = a.pss[kk], pc = a.pcv[kk];
                X5 dg = shfl_up5(nx);
                if (lane == 0) dg = row_above(c - 1);
                float tf[7], tn[7];
                ring_row<64>(trs, c, tf);
                ring_row<64>(trs, c + 1, tn);
                tf[TMI] = tn[TMI];
                tf[TII] = tn[TII];
                if (valid)
                    edge_posteriors(a, kk, b, own.MM, up, c == 0 ? LB : left, c == 0 ? DB : dg, qf, tf, sc, lz, ps, pc, g);
                up = dg;
                own = left;
                left = nx;
            }
        }
    }
#pragma unroll
    for (int f = 0; f < 9; f++) {
        const float v = warp_sum(g[f]);
        if (lane == 0) gsh[wid][f] = v;
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        float v = 0.f;
        for (int w = POST_WARPS - 1; w >= 0; w--) v += gsh[w][threadIdx.x];
        a.gpart[(a.soff[m] + s) * 9 + threadIdx.x] = v;
    }
}

// gradients of each pair: its strips' sums in strip order
__global__ void adj_gsum_kernel(AdjArgs a)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= a.npairs * 9) return;
    const int m = x / 9, f = x % 9;
    const int ns = (a.pLq[m] + 31) >> 5;
    float v = 0.f;
    for (int s = 0; s < ns; s++) v += a.gpart[(a.soff[m] + s) * 9 + f];
    a.grad[x] = v;
}

cudaError_t adj_occupancy(int* fwd_ctas_per_sm, int* bwd_ctas_per_sm)
{
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(fwd_ctas_per_sm, adj_fwd_kernel, ADJ_WARPS * 32, 0);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bwd_ctas_per_sm, adj_bwd_kernel<ADJ_RECOMP>, ADJ_WARPS * 32, 0);
}

cudaError_t launch_adj_fwd(const AdjArgs& a, int grid, cudaStream_t st)
{
    if (a.npairs <= 0) return cudaSuccess;
    const int sgrid = std::min((a.nitems + ADJ_WARPS - 1) / ADJ_WARPS, 1184);
    const size_t ssm = (size_t)ADJ_WARPS * ADJ_SCORE_FLOATS * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(adj_score_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm);
    if (e != cudaSuccess) return e;
    adj_score_kernel<<<sgrid, ADJ_WARPS * 32, ssm, st>>>(a);
    adj_fwd_kernel<<<grid, ADJ_WARPS * 32, 0, st>>>(a);
    adj_logz_kernel<<<(a.npairs + 127) / 128, 128, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adj_bwd(const AdjArgs& a, int grid, cudaStream_t st)
{
    if (a.npairs <= 0) return cudaSuccess;
    if (a.Ball) {
        int occ = 0, dev = 0, nsm = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, adj_bwd_kernel<ADJ_OUT>, ADJ_WARPS * 32, 0);
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        const int g = std::min(nsm * std::max(occ, 1), (a.nitems + ADJ_WARPS - 1) / ADJ_WARPS);
        adj_bwd_kernel<ADJ_OUT><<<g, ADJ_WARPS * 32, 0, st>>>(a);
        adj_post_kernel<<<a.nitems, POST_WARPS * 32, 0, st>>>(a);
    } else if (a.Fall) {
        adj_bwd_kernel<ADJ_KEPT><<<grid, ADJ_WARPS * 32, 0, st>>>(a);
    } else {
        adj_bwd_kernel<ADJ_RECOMP><<<grid, ADJ_WARPS * 32, 0, st>>>(a);
    }
    adj_gsum_kernel<<<(a.npairs * 9 + 127) / 128, 128, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace c2
