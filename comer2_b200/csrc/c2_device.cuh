// c2_device.cuh -- device-side layouts and kernel arguments of the B200
// implementation of the COMER2 search hot path.
//
// HBM layout (built by c2_upload_db / c2_set_query):
//  * db position records, DR_STRIDE floats (224 B) per position, everything a
//    score column and a DP column need, so one warp-uniform (broadcast) read
//    stream per column feeds all 32 lanes (lanes own query rows):
//      [0,20)  target probabilities          [20,39) context vector
//      39      cvnorm2 + 1 + 1/kappa0         40      CV log prior
//      [41,44) SS probabilities C,E,H         44      SS table indices, packed
//      45      P(H) + 0.1                     [48,55) DP transitions of the column
//      55      residue letter
//  * query position records, QR_STRIDE floats (256 B), the same fields for the
//    query rows plus the column -1 boundary states of the reference's DP
//    (see c2_host.cu: colm1 states).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace c2 {

constexpr int NAA = 20, NCV = 19, NSS = 3;
constexpr float LOG0 = -32768.0f;

enum : int {
    QR_TRG = 0, QR_CV = 20, QR_CN = 39, QR_PRIOR = 40, QR_SS = 41, QR_SSIDX = 44,
    QR_HQ = 47, QR_TRN = 48, QR_C = 55, QR_CP = 58, QR_STRIDE = 64
};
enum : int {
    DR_TRG = 0, DR_CV = 20, DR_CN = 39, DR_PRIOR = 40, DR_SS = 41, DR_SSIDX = 44,
    DR_HD = 45, DR_TRN = 48, DR_AA = 55, DR_STRIDE = 56
};
// DP transitions of a row/column: MM and MD, IM, DM, DD into the position,
// MI and II out of it (the reference's MMp, MIc, MDp, IMp, IIc, DMp, DDp;
// src/libmycu/cudp/CuBatchDP_init.cuh:132-155)
enum : int { TMM = 0, TMI, TMD, TIM, TII, TDM, TDD };

// btck codes (src/libmycu/cudp/CuBatchDP_com.h:99-104)
enum : int { BT_STOP = 0, BT_LEFT = 1, BT_UP = 2, BT_DIAG = 3 };

struct ScoreConsts {
    float ssswgt, cvswgt, shift;          // term weights, aa-term shift
    float lokappa0, pownu0, cterm;        // context-vector constants
    float cvkey_first, cvkey_last, cvval_first, cvval_last;
    int cvcard, cvshift, ssss_card;
    int cvhi;                             // cvcard - 1 - cvshift: largest table index before its shift
};

constexpr int P1_WARPS = 8;               // warps per CTA of the DP kernels
constexpr int MAX_SSSS_CARD = 32;
// db record staging ring of the phase-1 kernel: 2 chunks of 8 columns
constexpr int REC_CHUNK = 8, REC_CHUNK_LOG = 3, REC_SLOTS = 16;
// shared memory per warp: score ring [32][32], SS row table [32][32], record ring
constexpr int P1_WARP_FLOATS = 32 * 32 + MAX_SSSS_CARD * 32 + REC_SLOTS * DR_STRIDE;
constexpr int MAX_CVCARD = 256;
// Tensor-core (BF16 split) phase-1 kernel.  The three contractions of a cell
// score -- amino acids (K = 20), context vectors (K = 19) and the SS table
// (K = card <= 32, the db side a 3-hot vector of SS probabilities) -- run as
// mma.sync BF16 products with FP32 accumulation (K 16 + 8 for the first two,
// 16 + 16 for the third), each operand split into hi + lo BF16 parts
// (x = hi + lo + O(2^-17 x)) and hi*hi + hi*lo + lo*hi accumulated.  db
// operands (B fragments) are packed once per database in the fragment order
// of the 32 lanes, 8 db columns per tile (ceil(L / 8) tiles a profile):
//   tcdb[tile][5][lane 32][4 words]
//     0: aa hi k0-15 (2 words), aa hi k16-23, aa lo k16-23
//     1: aa lo k0-15 (2), cv hi k0-15 (2)
//     2: cv lo k0-15 (2), cv hi k16-23, cv lo k16-23
//     3: ss hi k0-15 (2), ss hi k16-31 (2)     4: ss lo, the same
// query operands (A fragments, strips of 64 rows) per query: context vectors
// and SS tables qa[strip][mtile 4][7][lane 32][4 words] (cv hi k0-15, lo k0-15; ss
// hi k0-15, hi k16-31, lo k0-15, lo k16-31; cv hi k16-23 (2), lo k16-23 (2):
// groups of 4 words, so that every fragment lands in aligned registers) and the
// unscaled amino-acid rows
// qaa[strip][mtile 4][3][lane 32][4 floats] (k0-15: 8, k16-23: 4; scaled per
// pair by 1 / (0.5 (bq + bd)) and split).
// The constant parts of the CV and SS terms ride in the spare K columns:
// CV k = 19 carries 1 (query) x 1/kappa0 (db), so the CV accumulator is the
// shifted dot product; the SS operand is weighted by the SS weight on the db
// side and k = 30, 31 carry P(H)q + 0.1 x w (P(H)d + 0.1) / 9 and 1 x -0.05 w,
// so the SS accumulator is the complete weighted SS term (the reference's
// "-99 < ss" guard always holds for tables above SS_FOLD_MIN, which the
// tensor-core form requires, with card <= 30).
// Per db position the DP and the score epilogue also read a column record
// cold[pos][P1C_TRS]: the DP transitions (TMM .. TDD, slots 0..6), cvnorm and
// 2 x CV log prior (slots 8, 9), pad.
constexpr int P1_ROWS = 64;                           // query rows per strip of the phase-1 kernels
constexpr int TC_TILE_WORDS = 5 * 32 * 4;
constexpr int TC_QA_WORDS = 4 * 7 * 32 * 4;           // per strip
constexpr int TC_QAA_FLOATS = 4 * 3 * 32 * 4;         // per strip
constexpr float SS_FOLD_MIN = -49.f;
constexpr int TC_SS_KMAX = 30;
enum : int { CO_CD = 8, CO_PD2 = 9 };
// phase-1 kernel variants of launch_p1
enum : int { P1K_STRIP = 0, P1K_CHUNKED = 1, P1K_TRACEBACK = 2, P1K_TENSOR = 3 };
// column records in shared memory, 12 floats apart (the two 16-byte reads of 8
// lanes at consecutive columns cover 32 distinct banks)
constexpr int P1C_RING = 64, P1C_TRS = 12;
constexpr int TB_C = 16;   // columns per chunk of the traceback sweep
// traceback sweep over the stored score matrices: per warp the score ring, the
// transition ring, the row above and a [32][33]-byte traceback column ring;
// 16 warps per SM.  P1TC_CVREP: CV table replicas of the phase-2 score kernel
constexpr int P1TC_WARPS = 16, P1TC_CVREP = 8;
constexpr int P1TC_WARP_FLOATS = P1C_RING * 32 + P1C_RING * P1C_TRS + 2 * 5 * TB_C;
// phase-2 score kernel: 8 warps per CTA, per warp the SS row table and the
// record staging ring; the CV table (P1TC_CVREP replicas) per CTA
constexpr int P2S_WARPS = 8;
constexpr int P2S_WARP_FLOATS = MAX_SSSS_CARD * 32 + REC_SLOTS * DR_STRIDE;

// Largest CV maps the shared-memory layouts hold (opt-in shared memory per CTA
// on sm_100: 227 KB): the phase-2 score kernel, which every search runs.  The
// tensor-core form takes maps of up to 106 entries.  The reference's cvs2s map
// has 93 entries.
constexpr int SMEM_CTA_MAX = 227 * 1024;
constexpr int P1TC_MAX_CVCARD =
    (SMEM_CTA_MAX - P2S_WARPS * P2S_WARP_FLOATS * 4) / (P1TC_CVREP * 4);
constexpr int P1T_MAX_CVCARD = 106;
// Phase-1 kernels, two query rows per lane (strips of 64 rows), the db columns
// in chunks of 8.  Per warp: score ring of 40 anti-diagonals (31 lanes of skew
// + a chunk) of 64 floats, padded to 68 so that the score writes (a lane's two
// rows, or the tensor fragments) and the wavefront's 8-byte reads are free of
// bank conflicts; column-record ring of 7 chunks and a mirror of its first
// chunk, so that the 8 records a lane reads in one DP stage never wrap; the row
// above the strip for one chunk and the strip's own last row (not in its place:
// nothing orders lane 31's write of a step before lane 0's read of it).
constexpr int P1_C = 8;
constexpr int P1_SLOTS = 40, P1_RLD = 68, P1_CMOD = 56, P1_CRING = 64;
constexpr int P1_BND = 5 * P1_C;
// (the two rows, and a gap that leaves the arrays after them where the FP32 kernel
// runs best: 14.08 ms on 1 x 400 vs 20,000 profiles, without it 14.27)
constexpr int P1_BNDS = 2 * P1_BND + 24;
constexpr int P1_WF_FLOATS = P1_SLOTS * P1_RLD + P1_CRING * P1C_TRS + P1_BNDS;
// FP32 kernel: also the SS row table of the strip and the record staging ring
constexpr int P1C_WARPS = 8, P1C_CVREP = 16;
constexpr int P1C_WARP_FLOATS = P1_WF_FLOATS + MAX_SSSS_CARD * P1_ROWS + REC_SLOTS * DR_STRIDE;
static_assert((MAX_CVCARD * P1C_CVREP + P1C_WARPS * P1C_WARP_FLOATS) * 4 <= SMEM_CTA_MAX, "FP32 phase-1 shared memory");
// tensor-core kernel: also the rows' score terms and one slot for the db
// operand tile (a bulk async copy, one mbarrier)
constexpr int P1T_WARPS = 12, P1T_CVREP = 16;
constexpr unsigned P1T_TMEM_COLS = 512;   // TMEM columns of a CTA: 3 warps x 160 per lane quarter
constexpr int P1T_TMEM_MT = 40, P1T_TMEM_WARP = 4 * P1T_TMEM_MT;
constexpr int P1T_WARP_FLOATS = P1_WF_FLOATS + 2 * P1_ROWS + TC_TILE_WORDS + 4;
static_assert((P1T_MAX_CVCARD * P1T_CVREP + P1T_WARPS * P1T_WARP_FLOATS) * 4 + 16 <= SMEM_CTA_MAX,
              "tensor-core phase-1 shared memory");
static_assert(P1T_WARP_FLOATS % 4 == 0 && P1C_WARP_FLOATS % 4 == 0, "16-byte alignment of the warps' shared memory");

// Epilogue constants of the tensor-core form: x = 2 x (CV score argument)
// = (2 pownu0 ln2) log2(det) + 2 cterm - 2 prior_q - 2 prior_d, compared
// with twice the table keys; table values pre-multiplied by the CV weight.
// uniform: the table index clamp alone reproduces the key range tests.
struct TcConsts {
    float shift, p2l, c2, kf2, kl2, vfw, vlw;
    int ilo, ihi, uniform;
};

struct P1Args {
    const float* qrec;      // [Lq][QR_STRIDE]
    int Lq;
    const float* drec;      // [npos][DR_STRIDE]
    const int* plen;        // [nprof]
    const long long* poff;  // [nprof]
    const float* pbkg;      // [nprof][20]
    int nwork;              // number of work items (profiles or candidates)
    const int* order;       // work item -> profile
    int* counter;           // work-queue head
    const float* ssss;      // [card][card]
    const float* cvvals;    // [cvcard]
    const float* qU;        // [strip][MAX_SSSS_CARD][32] SS row tables of the query rows
    ScoreConsts sc;
    float* bot;             // strip-boundary rows: per warp slot 2 x 5 x Lmax
    long long botstride;    // floats per warp slot
    // phase-1 pairs whose strips are work items of their own (the first nsplit of order)
    int nsplit;
    const long long* sboff; // sum of the lengths (rounded up to 4) before each pair of order
    float* sbnd;            // per split pair at 10 x sboff: two last-row buffers of 5 floats a column
    int* sprog;             // [nstrips][nsplit] finished columns per strip
    int* sdone;             // [nsplit] finished strips
    unsigned long long* skey;  // [nsplit] maximum so far and its cell, packed
    // phase-1 outputs (indexed by profile)
    float* best;
    unsigned* coords;
    // traceback variant: per work item k, scratch at cand_off[k]
    const long long* cand_off;  // byte offsets into btck / float offsets into smat
    signed char* btck;          // [L][Lq] per candidate (column-major)
    float* smat;                // [L][Lq] per candidate
    float* mmat;                // [L][Lq] per candidate: modular scores
    int* status;                // device error word (0 = ok)
    // strip pipeline of the traceback variant
    float* bnd;                 // last rows of the strips (row_block)
    unsigned long long* tbkey;  // [ncand] maximum of the traceback sweep and its cell, packed
    const int* worder;          // traceback sweep: rank -> candidate (longest first)
    int p2s_cols, p2s_blocks;   // phase-2 score matrices: columns per work item, items per (candidate, strip)
    const int* items;           // traceback sweep: work item -> rank * nstrips + strip
    unsigned spin;              // polls before a strip wait gives up
    // tensor-core operands (P1K_TENSOR)
    const unsigned* tcdb;       // db B fragments
    const long long* ttile;     // [nprof] first tile of each profile
    const float* cold;          // [npos][P1C_TRS] column records
    const unsigned* qa;         // query A fragments (cv, ss)
    const float* qaa;           // query amino-acid rows in fragment order
    TcConsts tc;
};

struct FinArgs {
    int Lq;
    int ncand;
    const int* cand_prof;
    const long long* cand_off;
    const int* plen;
    const signed char* btck;
    const float* smat;
    const float* best;
    const unsigned* coords;
    float scorethld;
    const unsigned long long* tbkey;  // [ncand] maxima of the traceback sweep and their cells
    float tol;                  // allowed |phase-1 maximum - traceback maximum| (0: identical)
    int* status;
    // outputs [ncand]
    float* score;
    int* psts;
    unsigned* beg;
    unsigned* endc;
    int* passed;
};

}  // namespace c2

// ---------------------------------------------------------------------------
// Phase-2 sweeps (traceback DP, MAP forward/backward/MAP DP) run one strip of
// one pair per warp: a work item is (pair m, strip s), items are handed out
// in the order of a host-built table from a global counter.  The table puts
// (m, s) after (m, s - 1) (ordered by m + K s, K = pairs started per strip
// lag), so the item a warp waits on was taken earlier by a warp that is
// running, and strips are handed out about when their predecessor is ready.  A long pair
// is thus swept by up to nstrips warps at once instead of one.
//
// Row hand-off.  Strip s writes its last row (5 states per column) to a buffer
// of its own, filled with ROW_EMPTY words before the sweep; strip s + 1 reads a
// group of columns ahead of its use and polls until none of their words is
// empty.  The data is its own flag: no fence, no separate progress word and no
// cache invalidation stand between the strips, so a hand-off costs one trip
// through L2 (with progress words, released every 8 columns and acquired by the
// strip below, the fence and the acquire took longer than the 8 columns' cells).
// A computed value is never ROW_EMPTY: the device's arithmetic yields only the
// NaN 0x7fffffff.  The copies (16 bytes each) may read words that another SM is
// writing.  What is relied on is that an aligned 4-byte word arrives whole, old or
// new; nothing is assumed about the order in which a row's words arrive: every one
// is tested, and one found empty is read again (ld.relaxed.gpu).
// Layout of a row: [ld][4] states MM MI IM DN, then [ld] ND, ld the length
// rounded up to 4; the rows of a pair's strips follow one another.
namespace c2 {
constexpr unsigned PIPE_SPIN = 1u << 22;  // default polls before a wait gives up (c2_set_wait_limit)
constexpr int PIPE_ERR_TIMEOUT = 3;       // device status of an abandoned wait
constexpr int PIPE_ERR_TIMEOUT_P1 = 4;    // ... of phase 1

__device__ __forceinline__ int pipe_ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void pipe_st_release(int* p, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Warp-uniform wait until *flag >= need (lane 0 polls).  After `spin` polls
// (at least one) it records PIPE_ERR_TIMEOUT in *status, marks the warp
// broken (no further waits) and returns; the sweep then finishes with invalid
// values -- every cell index stays inside its pair, so nothing is read or
// written out of bounds -- and the host reports the status.
__device__ __forceinline__ void pipe_wait(const int* flag, int need, int lane, int* status, bool& broken,
                                          unsigned spin)
{
    if (broken) return;
    unsigned it = 0;
    for (;;) {
        int ok = 0;
        if (lane == 0) ok = pipe_ld_acquire(flag) >= need;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) break;
        if (++it >= spin) {
            if (lane == 0 && status) atomicCAS(status, 0, PIPE_ERR_TIMEOUT_P1);
            broken = true;
            break;
        }
        __nanosleep(128);
    }
    __syncwarp();
}

constexpr unsigned ROW_EMPTY = 0xffffffffu;

// First column of pair c's rows, pos the sum of the lengths of the pairs before
// it (each row rounded up to 4 columns fits before the next pair's)
__host__ __device__ __forceinline__ long long row_start(long long pos, long long c) { return (pos + 8 * c + 3) & ~3LL; }
__host__ __device__ __forceinline__ int row_ld(int L) { return (L + 3) & ~3; }

// one thread: column c of a row
__device__ __forceinline__ void row_put(float* row, int ld, int c, float mm, float mi, float im, float dn, float nd)
{
    asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(row + 4 * c), "f"(mm), "f"(mi), "f"(im),
                 "f"(dn)
                 : "memory");
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(row + 4 * ld + c), "f"(nd) : "memory");
}

// Warp-uniform wait: poll() (lane predicate, re-reading its words) until it
// holds for every lane.  After `spin` polls it records PIPE_ERR_TIMEOUT in
// *status, marks the warp broken (no further waits) and returns; the sweep then
// finishes with invalid values -- every cell index stays inside its pair, so
// nothing is read or written out of bounds -- and the host reports the status.
template <typename F>
__device__ __forceinline__ void row_poll(F poll, int lane, int* status, bool& broken, unsigned spin)
{
    for (unsigned it = 0;;) {
        if (__all_sync(0xffffffffu, poll()) || broken) return;
        if (++it >= spin) {
            if (lane == 0 && status) atomicCAS(status, 0, PIPE_ERR_TIMEOUT);
            broken = true;
            return;
        }
        // (short sleeps first: the columns are usually a few steps away)
        __nanosleep(it < 32 ? 20 : 128);
    }
}

// asynchronous global->shared copies (cp.async, 16 B each, through L2)
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_2() { asm volatile("cp.async.wait_group 2;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The lane's column c of a row another warp writes, for lanes with want
__device__ __forceinline__ void row_get(const float* row, int ld, int c, bool want, float* v, int lane, int* status,
                                        bool& broken, unsigned spin)
{
    row_poll(
        [&]() -> bool {
            if (!want) return true;
            asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                         : "l"(row + 4 * c)
                         : "memory");
            asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v[4]) : "l"(row + 4 * ld + c) : "memory");
            bool ok = true;
#pragma unroll
            for (int f = 0; f < 5; f++) ok = ok && __float_as_uint(v[f]) != ROW_EMPTY;
            return ok;
        },
        lane, status, broken, spin);
}

// A group of G columns of the row above in shared memory: [G][4] states, then
// [G] ND.  row_issue starts its copy a group ahead of its use; row_take, just
// before the use, looks whether the copy found every column there and polls for
// the rest only otherwise: a strip that trails far enough never waits for L2.
// Columns past the matrix stay empty (no cell inside the matrix reads them).
template <int G> constexpr int ROW_BUF = 5 * G;

template <int G>
__device__ __forceinline__ void row_issue(float* buf, const float* row, int ld, int c0, int L, int lane)
{
    const int c4 = c0 + 4 * (lane - G);
    if (lane < G) {
        if (c0 + lane < L) cp_async16(buf + 4 * lane, row + 4 * (c0 + lane));
    } else if (lane < G + G / 4 && c4 < L) {
        cp_async16(buf + 4 * G + 4 * (lane - G), row + 4 * ld + c4);
    }
    cp_async_commit();
}

template <int G>
__device__ __forceinline__ void row_take(float* buf, const float* row, int ld, int c0, int L, int lane, int* status,
                                         bool& broken, unsigned spin)
{
    cp_async_wait_all();
    __syncwarp();
    const bool want = lane < G && c0 + lane < L;
    bool ok = true;
    if (want) {
        const uint4 w = *reinterpret_cast<const uint4*>(buf + 4 * lane);
        ok = w.x != ROW_EMPTY && w.y != ROW_EMPTY && w.z != ROW_EMPTY && w.w != ROW_EMPTY &&
             __float_as_uint(buf[4 * G + lane]) != ROW_EMPTY;
    }
    if (!__all_sync(0xffffffffu, ok)) {
        float v[5];
        row_get(row, ld, c0 + lane, want, v, lane, status, broken, spin);
        if (want) {
            *reinterpret_cast<float4*>(buf + 4 * lane) = make_float4(v[0], v[1], v[2], v[3]);
            buf[4 * G + lane] = v[4];
        }
    }
    __syncwarp();
}
}  // namespace c2
