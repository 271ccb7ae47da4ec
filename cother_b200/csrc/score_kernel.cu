// Batch score matrix: profile-profile + secondary structure + distance
// distribution match score (DDMS) for every (query position, database
// position) cell of a slab, in ONE kernel.
//
// The reference computes the three terms in three kernels that add into the
// output with atomics (src/libmycu/cusco/CuBatchScoreMatrix.cu:236-396:
// CalcSM_Init_SMEMUnroll2x, CalcSM_SSSS_SMEMUnroll2x,
// CalcSM_DDMS2S_SMEMUnroll2x_h2). Here one thread owns one database
// position (lane) and walks a strip of query positions, adding the terms in
// the reference's order -- (init + SS) + DDMS -- and writing each cell once.
//
// DDMS dominates the cost (~550 segment-DP steps per cell for 99-distance
// lists); it is CUDA-core ALU-bound, so the kernel is shaped for issue
// efficiency: distance lists split by parity in shared memory, the database's
// as bytes at an odd word stride (conflict-free for lanes in step), a word of
// four read at once and byte and table row combined by one dp4a; a 22x22
// pair-score table in shared memory; the segment register reached only by
// steps that can change it; and DSTSEGM as compile-time cases.
#include <cmath>
#include "cother_b200.h"
#include "common.cuh"
#include "cbmath.cuh"
#include "layout.h"
#include "score_kernel.cuh"
#include "bulkcopy.cuh"

namespace cbp {

namespace {

constexpr int kCols = 32;          // database positions per block (one per lane)
constexpr int kWarps = 4;
constexpr int kThreads = kCols * kWarps;
constexpr int kDbCopy = 112;       // bytes of a list brought in by one bulk copy (and its packed stride)
// The diagonals of the DDMS step through the lists two elements at a time,
// so a diagonal reads elements of one parity only: a database list is kept
// as its even and its odd elements, bytes, element m of a parity at byte
// m + 3 of its kHalfWords words (element 1 starts a word).
constexpr int kHalfWords = 16;
constexpr int kDbWords = 2 * kHalfWords + 1;   // an odd stride: lanes in step do not conflict
// A query list is kept as 32-bit byte offsets into the pair-score table
// (code x 88): the even elements for the upper diagonals, element m at word
// m + 3 (element 1 on 16 bytes), and for the lower diagonals the elements of
// the parity they use twice, element n at word n + 1 and at word n, so that
// element n0 + 1 starts on 8 bytes for even and for odd n0.
constexpr int kQUp = 64, kQLow = 60;
constexpr int kQWords = kQUp + 2 * kQLow;
constexpr unsigned long long kListWaitNs = 1000000000ull;   // the lists' copies: a wait gives up after 1 s

// Top-3 register of non-intersecting segments
// (src/libmycu/cusco/CuBatchScoreMatrix_ddms2s.cuh:182-251). The reference
// packs a segment's coordinates into one word [QB QE PB PE] and tests
// intersection with per-byte SIMD min/max. Here a segment is two words,
// begins (QB<<16 | PB) and ends (QE<<16 | PE), the ends with the top bit of
// each halfword set: two segments intersect when their query OR their
// database ranges overlap (ddms2s.cuh:162-173), i.e. when in either halfword
// both ends are at or past the other's begin, and with the guard bits each
// difference keeps its top bit exactly then (positions < 32768).
constexpr uint32_t kGuard = 0x80008000u;
__device__ __forceinline__ bool seg_intersect(uint32_t b1, uint32_t e1, uint32_t b2, uint32_t e2)
{
    return ((e1 - b2) & (e2 - b1) & kGuard) != 0u;
}

// Saturating add/multiply: the result clamped to [0, 1] in one FMA-pipe
// instruction.
__device__ __forceinline__ float sat_add(float a, float b)
{
    float r;
    asm("add.sat.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float sat_fma(float a, float b, float c)
{
    float r;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The third score while its entry is empty: the smallest positive float, so
// that it is also the register's threshold (every positive candidate is at
// least this).
constexpr float kTiny = 0x1p-149f;
constexpr unsigned kFull = 0xffffffffu;

// The register of one cell: the three scores in order, and the coordinates
// of the first two entries (every change of the register drops the third,
// so its coordinates are never consulted; nor are an empty entry's).
struct DdmsReg {
    float m0 = 0.0f, m1 = 0.0f, m2 = kTiny;
    uint32_t b0 = 0, e0 = kGuard, b1 = 0, e1 = kGuard;
};

// Lengths are kept in units of 2^22, as the bits of a float: see
// ddms_diagonal().
constexpr int kLenUnit = 1 << 22;

// The bits of a length, as a float, grow with it, so a saturating multiply-add
// turns them into 1 at DSTSEGM - 1 units and above and 0 below.
struct LenMask { float scale, bias; };
template <int kSeg>
__device__ __forceinline__ LenMask len_mask(int dst)
{
    if (kSeg == 6) return {0x1p126f, -2.0f};       // 5 units: 1.5 x 2^-125; 4 units: 2^-125
    if (dst == 1) return {0.0f, 1.0f};
    const float at = __int_as_float((dst - 1) * kLenUnit), below = __int_as_float((dst - 2) * kLenUnit);
    const float scale = __fdiv_rn(1.0f, at - below);   // a power of two, at most 2^127
    return {scale, -(below * scale)};
}

// The best candidate of one 4-step, offered to the register: t1..t4 are the
// running sums after the step's elements, c0..c3 the elements since the sum
// was last zero, up to the element before each (a candidate needs DSTSEGM - 1
// of them), pos the query and database index of the step's first element. All
// three cases of the reference's register are one rule: a candidate at or
// above the third score enters unless it intersects an entry of a higher
// score; entering, it removes the entries of at most its score that it
// intersects, and the third.
//
// Returns the threshold of the lane until the running segment ends: a later
// candidate of the same segment has the same begin and a larger end, so it
// intersects what this one does, and below this one's score (if it entered)
// or below that of the entry that rejected it, it changes nothing. Without
// that threshold a lane of 57 % of the warp steps has a candidate at or above
// its third entry; with it, 36 % (a CPU emulation of the warps on the lists of
// a 400-position query and 200 profiles).
template <int kSeg>
__device__ __forceinline__ float ddms_offer(DdmsReg& r, bool on, uint32_t pos, float thr, LenMask lm, int c0, int c1,
                                            int c2, int c3, float t1, float t2, float t3, float t4)
{
    // the sum where the segment is long enough, else 0
    const float v1 = t1 * sat_fma(__int_as_float(c0), lm.scale, lm.bias);
    const float v2 = t2 * sat_fma(__int_as_float(c1), lm.scale, lm.bias);
    const float v3 = t3 * sat_fma(__int_as_float(c2), lm.scale, lm.bias);
    const float v4 = t4 * sat_fma(__int_as_float(c3), lm.scale, lm.bias);
    const float s = fmaxf(fmaxf(v1, v2), fmaxf(v3, v4));
    const bool ok = on & (thr <= s);
    if (ok) {
        // ending at the first element that attains it
        const uint32_t k = (v1 == s) ? 0x80018001u : (v2 == s) ? 0x80028002u : (v3 == s) ? 0x80038003u : 0x80048004u;
        const uint32_t ce = pos + k;
        // DSTSEGM >= 5: the candidate, at least 5 long and ending at most 4
        // past the step's first element, contains it: c0 elements up to it
        uint32_t cb;
        if (kSeg != 1) {
            cb = (pos + 0x00010001u) - __umulhi((uint32_t)c0, 0x00010001u << 10);
        } else {
            const int ck = (v1 == s) ? c0 : (v2 == s) ? c1 : (v3 == s) ? c2 : c3;
            cb = (ce - kGuard) - __umulhi((uint32_t)ck, 0x00010001u << 10);
        }
        const bool x0 = seg_intersect(cb, ce, r.b0, r.e0);
        const bool x1 = seg_intersect(cb, ce, r.b1, r.e1);
        const bool g0 = r.m0 <= s, g1 = r.m1 <= s;
        const bool rej0 = x0 & !g0, rej1 = x1 & !g1;
        thr = rej0 ? r.m0 : rej1 ? r.m1 : s;
        if (!rej0 & !rej1) {
            if (x1) r.m1 = 0.0f;
            r.m2 = fmaxf(g1 ? r.m1 : s, kTiny);
            if (g0) {
                if (x0) r.m2 = kTiny;
                else { r.m1 = r.m0; r.b1 = r.b0; r.e1 = r.e0; }
                r.m0 = s; r.b0 = cb; r.e0 = ce;
            } else if (g1) {
                r.m1 = s; r.b1 = cb; r.e1 = ce;
            }
        }
    }
    return thr;
}

// One diagonal of the DDMS segment DP. Elements e = 0,1,... pair query list
// element oq+e with database list element od+e (upper diagonals: oq = 0,
// od = j; lower: oq = i, od = 0). Pair scores at even offsets within each
// 4-step are table values, odd ones the mean of their neighbours
// (src/libmycu/cusco/CuBatchScoreMatrix_ddms2s_h2.cuh:184-198); a segment
// restarts when the running sum has fallen to zero, and the best segment of
// length >= DSTSEGM ending in each 4-step is offered to the top-3 register
// (ddms2s_h2.cuh:124-176, 288-396).
//
// The pair scores come pre-scaled by 2^-7, so every running sum stays in
// [0, 1) and max(sum, 0) is one saturating add; scaling by a power of two
// commutes exactly with IEEE rounding, so the sums are the reference's
// times 2^-7, bit for bit. An odd element's mean 0.5*(a+b) is exact once a+b
// is rounded, so adding it is one saturating fma(0.5, a+b, sum). The bits of
// a sum, as an integer, are 0 when it is zero and 158 x 2^22 (the bits of
// 2^-48) at least when not: the scaled values are multiples of 2^-47 (checked
// by build_dms_table()), their means of 2^-48, and so is every sum of them. A
// length is 105 at most (a list holds 99 elements, and the last two steps end
// up to six past it), so the number of elements since the last zero, in units of
// 2^22, is min(c + 2^22, bits), one instruction (VIADDMNMX) for the two that a
// float length needs.
//
// A step can offer a candidate (DSTSEGM >= 5) only when its first sum is
// positive and c1 >= DSTSEGM - 3, which is all that every step tests; the
// masked sums and the register are in ddms_offer(), in 64 % and 36 % of the
// warp steps. What bounds the kernel is instruction issue (0.87 a cycle and
// scheduler), with the ALU pipe, which takes an instruction every other
// cycle, at 69 %: the steps' arithmetic is therefore spread over both pipes
// (sums and masks FMA, lengths ALU, table offsets the FMA pipe's dp4a).
// Measured at q400 x 1,000 profiles, 16 rows a block: 51.0 warp instructions
// a step and 77.4 ms, against 59.2 and 85.8 ms with float lengths, the masked
// sums in every step and no threshold per segment; with the masks in every
// step 82 ms, with a running maximum tested first 86 ms, with votes for the
// branches 91 ms.
//
// qw: words of elements 1.. of the query list on this diagonal, q0 its
// element 0; dw, sel: the words that hold elements 1.. of the database list
// (upper: the byte selector that aligns them), d0 its element 0; ks: the
// multipliers that pick byte 0..3 of a word and scale it to a table offset.
template <bool kUpper, int kSeg>
__device__ __forceinline__ void ddms_diagonal(
    const uint32_t* __restrict__ qw, uint32_t q0, const uint32_t* __restrict__ dw, uint32_t sel, uint32_t d0,
    const char* __restrict__ T, int lim, uint32_t pos0, int dst, LenMask lm, uint4 ks, DdmsReg& r)
{
    const int need = (kSeg == 6 ? 5 : dst - 1) * kLenUnit;
    float s0 = *reinterpret_cast<const float*>(T + (q0 + 4u * d0));
    float t = sat_add(s0, 0.0f);
    int c = t > 0.0f ? kLenUnit : 0;
    float thr = 0.0f;
    uint32_t cur = dw[0];
    auto step = [&](float s2, float s4, int x, bool on) {
        const float t1 = sat_fma(0.5f, s0 + s2, t);
        const int c1 = __viaddmin_s32(c, kLenUnit, __float_as_int(t1));
        const float t2 = sat_add(t1, s2);
        const int c2 = __viaddmin_s32(c1, kLenUnit, __float_as_int(t2));
        const float t3 = sat_fma(0.5f, s2 + s4, t2);
        const int c3 = __viaddmin_s32(c2, kLenUnit, __float_as_int(t3));
        const float t4 = sat_add(t3, s4);
        const uint32_t pos = pos0 + (uint32_t)x * 0x00010001u;
        if (kSeg != 1) {
            // a segment's first step that can offer has c1 <= DSTSEGM units:
            // its threshold is the register's
            const bool fresh = c1 <= need + kLenUnit;
            if (c1 >= need - 2 * kLenUnit)
                thr = ddms_offer<kSeg>(r, on, pos, fresh ? r.m2 : thr, lm, c, c1, c2, c3, t1, t2, t3, t4);
        } else {
            (void)ddms_offer<kSeg>(r, on, pos, r.m2, lm, c, c1, c2, c3, t1, t2, t3, t4);
        }
        s0 = s4;
        t = t4;
        c = __viaddmin_s32(c3, kLenUnit, __float_as_int(t4));
    };
    auto score = [&](uint32_t o) { return *reinterpret_cast<const float*>(T + o); };
    // two steps an iteration: four elements of each list (unrolled further,
    // or with the scores of the next iteration fetched ahead, it was slower)
#pragma unroll 1
    for (int x = 0; x < lim; x += 8) {
        uint32_t d, o0, o1, o2, o3;
        if (kUpper) {
            const uint32_t nxt = dw[(x >> 3) + 1];
            d = __byte_perm(cur, nxt, sel);
            cur = nxt;
            const uint4 o = *reinterpret_cast<const uint4*>(qw + (x >> 1));
            o0 = o.x; o1 = o.y; o2 = o.z; o3 = o.w;
        } else {
            d = dw[x >> 3];
            const uint2 a = *reinterpret_cast<const uint2*>(qw + (x >> 1));
            const uint2 b = *reinterpret_cast<const uint2*>(qw + (x >> 1) + 2);
            o0 = a.x; o1 = a.y; o2 = b.x; o3 = b.y;
        }
        const float sa = score(__dp4a(d, ks.x, o0)), sb = score(__dp4a(d, ks.y, o1));
        const float sc = score(__dp4a(d, ks.z, o2)), sd = score(__dp4a(d, ks.w, o3));
        step(sa, sb, x, true);
        step(sc, sd, x + 4, x + 4 < lim);
    }
}

// DDMS of one cell (src/libmycu/cusco/CuBatchScoreMatrix_ddms2s_h2.cuh:433-500).
// Returns the top-3 sum in the reference's scale.
template <int kSeg>
__device__ __forceinline__ float ddms_cell(const uint32_t* __restrict__ q, int len1,
                                           const uint32_t* __restrict__ d, int len2,
                                           const char* __restrict__ T, int dst, uint4 ks)
{
    const LenMask lm = len_mask<kSeg>(dst);
    DdmsReg r;
    const uint8_t* db = reinterpret_cast<const uint8_t*>(d);
    {
        const int par = ((len2 >> 2) & 1) * kHalfWords;
        for (int j = len2 >> 2; 0 <= j; j -= 2) {
            const int n0 = j >> 1;
            ddms_diagonal<true, kSeg>(q + 4, q[3], d + par + 1 + (n0 >> 2), 0x3210u + 0x1111u * (uint32_t)(n0 & 3),
                                      db[4 * par + 3 + n0], T, min(len1, len2 - j), (uint32_t)j,
                                      dst, lm, ks, r);
        }
    }
    for (int i = len1 >> 2; 0 < i; i -= 2) {
        const int n0 = i >> 1;
        const uint32_t* ql = q + kQUp + ((n0 & 1) ? kQLow + n0 : n0 + 1);   // element n0
        ddms_diagonal<false, kSeg>(ql + 1, ql[0], d + 1, 0u, db[3], T, min(len2, len1 - i),
                                   (uint32_t)i << 16, dst, lm, ks, r);
    }
    float sum = 0.0f;
    sum = sum + r.m0;
    sum = sum + r.m1;
    sum = sum + (r.m2 > kTiny ? r.m2 : 0.0f);
    return sum * 128.0f;
}

// Context-vector term of one cell (CalcCVS2ScoreSMEMUnroll2x,
// src/libmycu/cusco/CuBatchScoreMatrix_cvs2s.cuh:47-136): the log-odds of
// the two normal vectors, log det(C2 + H'H) from their dot product and
// squared norms less both log priors, translated through the map
// (SerializedCVS2Scores::GetScoreE1S1Step2Boundary,
// src/libmycu/cupro/SerializedCVS2Scores.cuh:377-410). The dot product, the
// determinant and the log-odds are fused multiply-adds and the logarithm is
// the __logf intrinsic, as in the reference's build. A log-odds that is
// not above the first key (a NaN included) takes the first score.
__device__ __forceinline__ float cvs_cell(const ScoreArgs& a, const float* __restrict__ qcv, float qprior,
                                          float qnorm2, const float (*__restrict__ dcv)[kCols], int lane,
                                          float dprior, float dnorm2)
{
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < kNCV; i++) dot = __fmaf_rn(qcv[i], dcv[i][lane], dot);
    dot = dot + a.cvs_lokappa0;
    const float qa = qnorm2 + 1.0f + a.cvs_lokappa0;
    const float da = dnorm2 + 1.0f + a.cvs_lokappa0;
    const float det = __fmaf_rn(qa, da, -(dot * dot));
    if (a.cvs_int_priors) {   // FtorRoundMAPALN0 (CuBatchScoreMatrix_cvs2s.cuh:38-41)
        qprior = (float)(int)qprior;
        dprior = (float)(int)dprior;
    }
    const float lo = __fmaf_rn(a.cvs_pownu0, __logf(det), a.cvs_cterm) - qprior - dprior;
    if (!(a.cvs_key_first < lo)) return __ldg(a.cvs_scores);
    if (a.cvs_key_last <= lo) return __ldg(a.cvs_scores + a.cvs_card - 1);
    return __ldg(a.cvs_scores + a.cvs_shift + (int)rintf(lo + lo));
}

// kRows query positions per block (8, 16 or 32; each warp takes every
// kWarps-th of them), chosen by the tuner. kDdms: with the distance term (a
// search without it needs neither its lists nor its registers). kStacked: the rows belong to
// several queries (cbp_process_batch), each with its own background; a
// separate instantiation, so that the single-query kernel is unchanged.
template <int kRows, bool kStacked, bool kDdms>
__global__ void __launch_bounds__(kThreads, 8)
score_matrix_kernel(const ScoreArgs a)
{
    __shared__ float s_dms[kDstCard * kDstCard];
    __shared__ float s_sst[kSSCard * kSSCard];
    // the distance lists: first packed at kDbCopy bytes as the bulk copies
    // leave them, then split by parity at the odd stride of kDbWords words
    __shared__ __align__(16) uint32_t s_dbe[kCols * kDbWords];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ __align__(16) uint32_t s_qe[kRows * kQWords];
    __shared__ float s_dtf[kNAA][kCols];
    __shared__ float s_dbg[kNAA][kCols];
    __shared__ float s_dss[kNSS][kCols];
    __shared__ float s_qtf[kRows][kNAA + 1];
    __shared__ float s_qss[kRows][kNSS];
    __shared__ int s_dlen[kCols];
    __shared__ int s_qlen[kRows];
    // context vectors and their log priors and squared norms (CVSWGT > 0):
    // dynamic shared memory, absent otherwise, so that more blocks fit an SM
    extern __shared__ float s_cvsdyn[];
    float (*s_dcv)[kCols] = reinterpret_cast<float (*)[kCols]>(s_cvsdyn);
    float (*s_dcvpn)[kCols] = reinterpret_cast<float (*)[kCols]>(s_cvsdyn + kNCV * kCols);
    float (*s_qcv)[kNCV + 1] = reinterpret_cast<float (*)[kNCV + 1]>(s_cvsdyn + (kNCV + 2) * kCols);
    float (*s_qcvpn)[kRows] =
        reinterpret_cast<float (*)[kRows]>(s_cvsdyn + (kNCV + 2) * kCols + kRows * (kNCV + 1));
    __shared__ int s_col[kCols];
    __shared__ __align__(16) uint32_t s_ks[4];
    if (threadIdx.x < 4) s_ks[threadIdx.x] = 4u << (8 * threadIdx.x);

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int colb = blockIdx.x * kCols;
    const int rowb = blockIdx.y * kRows;
    const long long N = a.db.N;

    if (tid < kCols) {
        const int slot = colb + tid;
        s_col[tid] = slot < a.ncols ? (a.colorder ? a.colorder[slot] : slot) : -1;
    }
    constexpr bool ddms = kDdms;
    for (int i = tid; ddms && i < kDstCard * kDstCard; i += kThreads) s_dms[i] = a.dmstab[i] * 0x1p-7f;
    for (int i = tid; i < kSSCard * kSSCard; i += kThreads) s_sst[i] = a.sstab[i];
    if (ddms && tid == 0) {
        mbar_init(&s_bar);
        mbar_init_fence();
    }
    __syncthreads();

    // the block's distance lists (DDMS only): one bulk copy per column,
    // bytes 0..111 of its 128-byte list (this GPU's memory, 128-byte
    // aligned) into s_dbe at a 112-byte stride, in flight while the
    // column fields and the query rows below are read
    if (ddms && warp == 0) {
        const int cc = s_col[lane];
        const unsigned ncopy = __popc(__ballot_sync(0xffffffffu, cc >= 0));
        if (lane == 0) mbar_expect_tx(&s_bar, ncopy * (unsigned)kDbCopy);
        __syncwarp();
        if (cc >= 0) bulk_load(reinterpret_cast<char*>(s_dbe) + lane * kDbCopy, a.db.dst + (a.col0 + cc) * kDstStride, kDbCopy, &s_bar);
    }

    // database columns of this block: lane l takes slab column s_col[l]
    const int col = s_col[lane];
    const bool cvalid = col >= 0;
    const long long gpos = a.col0 + col;
    if (cvalid) {
        const int p = a.db.pro[gpos];
        for (int k = warp; k < kNAA; k += kWarps) {
            s_dtf[k][lane] = a.db.tf[(long long)k * N + gpos];
            // one query: the denominator 0.5*(query bkg + profile bkg) of
            // the column, rounded as in the cell loop; stacked queries: the
            // profile's background alone
            const float b = a.db.bkg[(long long)k * a.db.P + p];
            s_dbg[k][lane] = kStacked ? b : 0.5f * (__ldg(a.q.bkg + k) + b);
        }
        if (warp < kNSS) s_dss[warp][lane] = a.db.ss[(long long)warp * N + gpos];
        if (warp == kNSS) s_dlen[lane] = a.db.dstlen[gpos];
    } else if (warp == kNSS) {
        s_dlen[lane] = 0;
    }
    // query rows of this block
    for (int idx = tid; idx < kRows * kNAA; idx += kThreads) {
        const int r = idx / kNAA, k = idx - r * kNAA;
        const int row = rowb + r;
        s_qtf[r][k] = row < a.Lq ? a.q.tf[(long long)k * a.q.N + row] : 0.0f;
    }
    for (int idx = tid; idx < kRows * kNSS; idx += kThreads) {
        const int r = idx / kNSS, k = idx - r * kNSS;
        const int row = rowb + r;
        s_qss[r][k] = row < a.Lq ? a.q.ss[(long long)k * a.q.N + row] : 0.0f;
    }
    if (a.cvswgt > 0.0f) {
        if (cvalid) {
            for (int k = warp; k < kNCV; k += kWarps) s_dcv[k][lane] = a.db.cv[(long long)k * N + gpos];
            if (warp == 0) {
                s_dcvpn[0][lane] = a.db.cvprior[gpos];
                s_dcvpn[1][lane] = a.db.cvnorm2[gpos];
            }
        }
        for (int idx = tid; idx < kRows * kNCV; idx += kThreads) {
            const int r = idx / kNCV, k = idx - r * kNCV;
            const int row = rowb + r;
            s_qcv[r][k] = row < a.Lq ? a.q.cv[(long long)k * a.q.N + row] : 0.0f;
        }
        if (tid < kRows) {
            const int row = rowb + tid;
            s_qcvpn[0][tid] = row < a.Lq ? a.q.cvprior[row] : 0.0f;
            s_qcvpn[1][tid] = row < a.Lq ? a.q.cvnorm2[row] : 0.0f;
        }
    }
    if (tid < kRows) s_qlen[tid] = (rowb + tid < a.Lq) ? a.q.dstlen[rowb + tid] : 0;
    // query lists as the diagonals read them: each code times 88, the byte
    // offset of its table row
    for (int idx = tid; ddms && idx < kRows * kQWords; idx += kThreads) {
        const int r = idx / kQWords, w = idx - r * kQWords;
        const int row = rowb + r;
        uint32_t v = kDstNoData;
        if (row < a.Lq) {
            int e;
            if (w < kQUp) {
                e = 2 * (w - 3);
            } else {
                const int par = (a.q.dstlen[row] >> 2) & 1;
                e = w < kQUp + kQLow ? 2 * (w - kQUp - 1) + par : 2 * (w - kQUp - kQLow) + par;
            }
            if (e >= 0 && e < kDstStride) v = a.q.dst[(long long)row * kDstStride + e];
        }
        s_qe[idx] = v * (kDstCard * 4);
    }
    if (ddms) {
        // the lists' copies: a wait that gives up flags the launch, waits
        // once more for the copies still in flight into this block's
        // shared memory, and ends the block without writing
        const bool got = mbar_wait_for(&s_bar, 0, kListWaitNs);
        if (__syncthreads_or(!got)) {
            if (tid == 0 && a.err) atomicExch(a.err, 2);
            (void)mbar_wait_for(&s_bar, 0, kListWaitNs);
            return;
        }
        // split by parity; a slot without a column and bytes past the
        // list read as no data
        constexpr int kPer = (kCols * kDbWords + kThreads - 1) / kThreads;
        const uint8_t* src = reinterpret_cast<const uint8_t*>(s_dbe);
        uint32_t w[kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const int idx = tid + k * kThreads;
            const int c = idx / kDbWords, wd = idx - c * kDbWords;
            const int par = wd >= kHalfWords ? 1 : 0;
            w[k] = 0;
            for (int y = 0; y < 4; y++) {
                const int e = 2 * (4 * (wd - par * kHalfWords) + y - 3) + par;
                uint32_t v = kDstNoData;
                if (idx < kCols * kDbWords && s_col[c] >= 0 && e >= 0 && e < kDbCopy) v = src[c * kDbCopy + e];
                w[k] |= v << (8 * y);
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const int idx = tid + k * kThreads;
            if (idx < kCols * kDbWords) s_dbe[idx] = w[k];
        }
    }
    __syncthreads();

    // no block-wide synchronisation below; a lane without a column stays
    // with its warp (the DDMS runs by warps) and writes nothing
    const uint4 ks = *reinterpret_cast<const uint4*>(s_ks);
    const int dlen = s_dlen[lane];
    const uint32_t* de = s_dbe + lane * kDbWords;
    const float dss0 = s_dss[0][lane], dss1 = s_dss[1][lane], dss2 = s_dss[2][lane];

    for (int r = warp; r < kRows; r += kWarps) {
        const int row = rowb + r;
        if (row >= a.Lq) break;

        float s = 0.0f, mod = 0.0f;
        if (cvalid) {
        // profile-profile term (CuBatchScoreMatrix_Init.cu:159-186)
        float acc = 0.0f;
        if (a.dots_in_scores) {
            acc = a.scores[(long long)row * a.ld + col];
        } else if (!kStacked) {
#pragma unroll
            for (int k = 0; k < kNAA; k++) {
                const float num = s_qtf[r][k] * s_dtf[k][lane];
                acc = acc + __fdiv_rn(num, s_dbg[k][lane]);
            }
        } else {
            // stacked queries: the background of this row's query
            const float* __restrict__ qbg = a.q.bkg + a.q.pro[row];
#pragma unroll
            for (int k = 0; k < kNAA; k++) {
                const float num = s_qtf[r][k] * s_dtf[k][lane];
                const float den = 0.5f * (__ldg(qbg + (long long)k * a.q.P) + s_dbg[k][lane]);
                acc = acc + __fdiv_rn(num, den);
            }
        }
        s = cb_logf(acc) - a.initshift;
        const float cvs = (a.cvswgt > 0.0f)
                              ? cvs_cell(a, s_qcv[r], s_qcvpn[0][r], s_qcvpn[1][r], s_dcv, lane,
                                         s_dcvpn[0][lane], s_dcvpn[1][lane])
                              : 0.0f;

        // SS term (CuBatchScoreMatrix_ssss.cu:209-279)
        if (a.ssswgt > 0.0f) {
            float ss = 0.0f;
            const float dsv[3] = {dss0, dss1, dss2};
#pragma unroll
            for (int i = 0; i < kNSS; i++) {
                const float f1 = s_qss[r][i];
                const int ri = i * 10 + (int)(f1 * 9.999f);
#pragma unroll
                for (int j = 0; j < kNSS; j++) {
                    const float f2 = dsv[j];
                    const int cj = j * 10 + (int)(f2 * 9.999f);
                    ss = __fmaf_rn(f1 * f2, s_sst[ri * kSSCard + cj], ss);
                }
            }
            if (-99.0f < ss) {
                ss = __fmaf_rn((s_qss[r][2] + 0.1f) * (dss2 + 0.1f), 0.1111111f, ss);
                ss = ss - 0.05f;
                ss = ss * a.ssswgt;
            }
            if (a.cvswgt > 0.0f) {
                // SS plus the weighted CVS term, the modular score 0.5*CVSWGT
                // lower (CuBatchScoreMatrix_ssss_cvs2s.cu:252-270). That
                // kernel computes chunk columns c and c+32 of each 64-column
                // block in one thread, and its build fuses the addition for
                // the first (one rounding) but not for the second.
                ss = ((gpos >> 5) & 1) ? ss + cvs * a.cvswgt : __fmaf_rn(cvs, a.cvswgt, ss);
                s = s + ss;
                mod = ss - 0.5f * a.cvswgt;
            } else {
                s = s + ss;
                mod = ss;
            }
        } else if (a.cvswgt > 0.0f && cvs != 0.0f) {
            // CVS alone (CuBatchScoreMatrix_cvs2s.cu:286-299); the modular
            // score starts at zero
            s = s + cvs * a.cvswgt;
            mod = mod + (cvs - 0.5f) * a.cvswgt;
        }
        }

        // DDMS term (CuBatchScoreMatrix_ddms2s_h2.cu:158-186)
        if constexpr (kDdms) {
            const int qlen = s_qlen[r];
            const bool on = dlen >= a.dstsegm;
            if (qlen >= a.dstsegm && __any_sync(kFull, on)) {
                const char* T = reinterpret_cast<const char*>(s_dms);
                const uint32_t* qe = s_qe + r * kQWords;
                const int len2 = on ? dlen : 0;
                const float sum = a.dstsegm == 6 ? ddms_cell<6>(qe, qlen, de, len2, T, a.dstsegm, ks)
                                  : a.dstsegm >= 5 ? ddms_cell<5>(qe, qlen, de, len2, T, a.dstsegm, ks)
                                                   : ddms_cell<1>(qe, qlen, de, len2, T, a.dstsegm, ks);
                const float dm = __fmaf_rn(0.053f * 16.0f, sum, -1.235f) * a.ddmswgt;
                if (on && dm != 0.0f) {
                    // the modular score drops 0.2*DDMSWGT, in the contracted
                    // form of CuBatchScoreMatrix_ddms2s_h2.cu:171
                    s = s + dm;
                    mod = mod + __fmaf_rn(-0.2f, a.ddmswgt, dm);
                }
            }
        }
        if (cvalid) {
            const long long o = (long long)row * a.ld + col;
            a.scores[o] = s;
            a.modscores[o] = mod;
        }
    }
}

// ---------------------------------------------------------------------------
// The profile-profile and SS terms alone (DDMSWGT = CVSWGT = 0, one query):
// one thread owns a column and walks kPlainRows query rows, the column's
// frequencies and denominators in registers.
//
// What bounds these cells are the 20 quotients, whose divisors depend on the
// column alone. With y = 1/d correctly rounded, computed once a column,
// q0 = n y, then twice r = n - d q, q' = q + r y gives the correctly rounded
// quotient by fused multiply-adds (Markstein, IBM J. Res. Dev. 34, 1990: a
// correction of a quotient within one unit in the last place by a correctly
// rounded reciprocal is correctly rounded; the first correction brings it
// there), five operations for a division's reciprocal, its steps and its range
// check. The residuals are exact while nothing underflows, so a block whose
// values leave the ranges below divides. 400 x 2,000 profiles (202 M cells):
// 2.2 ms, bound by instruction issue (about 250 a cell and lane, 160 of them
// the quotients; 2.0 ms with two rows in packed instructions, of half the
// rate), against 3.6 ms with divisions in the general kernel.
constexpr int kPlainCols = 128;
constexpr int kPlainRows = 32;
__device__ __forceinline__ bool plain_range(float v) { return v == 0.0f || (0x1p-40f <= v && v <= 0x1p20f); }
__device__ __forceinline__ bool plain_divisor(float d) { return 0x1p-13f <= d && d <= 2.0f; }

template <bool kDots>
__global__ void __launch_bounds__(kPlainCols)
score_plain_kernel(const ScoreArgs a)
{
    __shared__ float s_sst[kSSCard * kSSCard];
    __shared__ __align__(16) float s_q[kPlainRows][kNAA];
    __shared__ float s_qss[kPlainRows][kNSS];
    __shared__ int s_qri[kPlainRows][kNSS];       // first table entry of the probability's row
    const int tid = threadIdx.x;
    const int col = blockIdx.x * kPlainCols + tid;
    const int rowb = blockIdx.y * kPlainRows;
    const int nrows = min(kPlainRows, a.Lq - rowb);
    const bool cvalid = col < a.ncols;
    const long long gpos = a.col0 + col, N = a.db.N;
    const bool ssw = a.ssswgt > 0.0f;
    bool fast = true;
    for (int i = tid; ssw && i < kSSCard * kSSCard; i += kPlainCols) s_sst[i] = a.sstab[i];
    for (int i = tid; !kDots && i < nrows * kNAA; i += kPlainCols) {
        const int k = i / nrows, r = i - k * nrows;
        const float v = a.q.tf[(long long)k * a.q.N + rowb + r];
        s_q[r][k] = v;
        fast &= plain_range(v);
    }
    for (int i = tid; ssw && i < nrows * kNSS; i += kPlainCols) {
        const int k = i / nrows, r = i - k * nrows;
        const float f = a.q.ss[(long long)k * a.q.N + rowb + r];
        s_qss[r][k] = f;
        s_qri[r][k] = (k * 10 + (int)(f * 9.999f)) * kSSCard;
    }
    float dtf[kNAA], den[kNAA], y[kNAA];
    float dss[kNSS];
    int cj[kNSS];
#pragma unroll
    for (int k = 0; k < kNAA; k++) { dtf[k] = 0.0f; den[k] = 1.0f; }
#pragma unroll
    for (int k = 0; k < kNSS; k++) { dss[k] = 0.0f; cj[k] = k * 10; }
    if (cvalid) {
        if (!kDots) {
            const int p = a.db.pro[gpos];
#pragma unroll
            for (int k = 0; k < kNAA; k++) {
                dtf[k] = a.db.tf[(long long)k * N + gpos];
                den[k] = 0.5f * (__ldg(a.q.bkg + k) + a.db.bkg[(long long)k * a.db.P + p]);
                fast &= plain_range(dtf[k]) & plain_divisor(den[k]);
            }
        }
        if (ssw)
#pragma unroll
            for (int k = 0; k < kNSS; k++) {
                dss[k] = a.db.ss[(long long)k * N + gpos];
                cj[k] = k * 10 + (int)(dss[k] * 9.999f);
            }
    }
    if (!kDots)
#pragma unroll
        for (int k = 0; k < kNAA; k++) y[k] = __fdiv_rn(1.0f, den[k]);
    fast = __syncthreads_and(fast);
    if (!cvalid) return;

    for (int r = 0; r < nrows; r++) {
        const long long o = (long long)(rowb + r) * a.ld + col;
        // profile-profile term (CuBatchScoreMatrix_Init.cu:159-186)
        float acc = 0.0f;
        if (kDots) {
            acc = a.scores[o];
        } else if (fast) {
#pragma unroll
            for (int k = 0; k < kNAA; k++) {
                const float n = s_q[r][k] * dtf[k];
                float q = n * y[k];
                q = __fmaf_rn(__fmaf_rn(-den[k], q, n), y[k], q);
                q = __fmaf_rn(__fmaf_rn(-den[k], q, n), y[k], q);
                acc = acc + q;
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < kNAA; k++) {
                const float b = 0.5f * (__ldg(a.q.bkg + k) + a.db.bkg[(long long)k * a.db.P + a.db.pro[gpos]]);
                acc = acc + __fdiv_rn(s_q[r][k] * a.db.tf[(long long)k * N + gpos], b);
            }
        }
        float s = cb_logf(acc) - a.initshift, mod = 0.0f;
        // SS term (CuBatchScoreMatrix_ssss.cu:209-279)
        if (ssw) {
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < kNSS; i++) {
                const float f1 = s_qss[r][i];
                const int ri = s_qri[r][i];
#pragma unroll
                for (int j = 0; j < kNSS; j++) ss = __fmaf_rn(f1 * dss[j], s_sst[ri + cj[j]], ss);
            }
            if (-99.0f < ss) {
                ss = __fmaf_rn((s_qss[r][2] + 0.1f) * (dss[2] + 0.1f), 0.1111111f, ss);
                ss = ss - 0.05f;
                ss = ss * a.ssswgt;
            }
            s = s + ss;
            mod = ss;
        }
        a.scores[o] = s;
        a.modscores[o] = mod;
    }
}

}  // namespace

// One block per window: a counting sort of the window's columns by
// descending list length (0..kMaxDst). The order within one length is
// arbitrary: it decides only which lane computes a cell, never its value.
__global__ void __launch_bounds__(256)
column_order_kernel(const uint8_t* __restrict__ dstlen, long long col0, int ncols, long long ld, int window,
                    int* __restrict__ order)
{
    __shared__ int s_cnt[kMaxDst + 1];
    const int w0 = blockIdx.x * window;
    const int n = min(window, ncols - w0);
    for (int i = threadIdx.x; i <= kMaxDst; i += blockDim.x) s_cnt[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        atomicAdd(&s_cnt[kMaxDst - min((int)dstlen[col0 + w0 + i], kMaxDst)], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int b = 0; b <= kMaxDst; b++) {
            const int c = s_cnt[b];
            s_cnt[b] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int b = kMaxDst - min((int)dstlen[col0 + w0 + i], kMaxDst);
        order[w0 + atomicAdd(&s_cnt[b], 1)] = w0 + i;
    }
    // slots past the last column (the final window only)
    for (long long i = (long long)w0 + n + threadIdx.x; i < min(ld, (long long)w0 + window);
         i += blockDim.x)
        order[i] = -1;
}

void launch_column_order(const uint8_t* dstlen, long long col0, int ncols, long long ld, int window, int* order,
                         cudaStream_t stream)
{
    if (ncols <= 0) return;
    if (window < 32 || window > kMaxOrderWindow || window % 32)
        throw Error(CBP_ERR_ARG, "column order window must be a multiple of 32 in [32, 4096]");
    column_order_kernel<<<(unsigned)ceil_div(ncols, window), 256, 0, stream>>>(dstlen, col0, ncols, ld, window,
                                                                               order);
    CBP_CHECK_LAUNCH();
}

bool score_plain(const ScoreArgs& a)
{
    return a.q.P == 1 && !(a.ddmswgt > 0.0f) && !(a.cvswgt > 0.0f) && !a.colorder;
}

template <int kRows, bool kStacked>
void launch_score_rows(const ScoreArgs& a, cudaStream_t stream)
{
    dim3 grid((unsigned)ceil_div(a.ncols, kCols), (unsigned)ceil_div(a.Lq, kRows));
    const size_t cvs_smem =
        a.cvswgt > 0.0f ? sizeof(float) * ((kNCV + 2) * kCols + kRows * (kNCV + 1) + 2 * kRows) : 0;
    if (a.ddmswgt > 0.0f) {
        score_matrix_kernel<kRows, kStacked, true><<<grid, kThreads, cvs_smem, stream>>>(a);
    } else if (score_plain(a)) {
        const dim3 pgrid((unsigned)ceil_div(a.ncols, kPlainCols), (unsigned)ceil_div(a.Lq, kPlainRows));
        if (a.dots_in_scores) score_plain_kernel<true><<<pgrid, kPlainCols, 0, stream>>>(a);
        else score_plain_kernel<false><<<pgrid, kPlainCols, 0, stream>>>(a);
    } else score_matrix_kernel<kRows, kStacked, false><<<grid, kThreads, cvs_smem, stream>>>(a);
    CBP_CHECK_LAUNCH();
}

template <int kRows>
void launch_score_rows(const ScoreArgs& a, cudaStream_t stream)
{
    // stacked queries (cbp_process_batch) have a background per row
    if (a.q.P > 1) launch_score_rows<kRows, true>(a, stream);
    else launch_score_rows<kRows, false>(a, stream);
}

void launch_score_matrix(const ScoreArgs& a, cudaStream_t stream)
{
    if (a.ncols <= 0 || a.Lq <= 0) return;
    switch (a.rows) {
    case 8: launch_score_rows<8>(a, stream); break;
    case 16: launch_score_rows<16>(a, stream); break;
    case 32: launch_score_rows<32>(a, stream); break;
    default: throw Error(CBP_ERR_ARG, "score kernel rows per block must be 8, 16 or 32");
    }
}

// Pair-score table over packed distance codes (0..20 saturated, 21 = no
// data), computed on the host (constants
// src/libmycu/cupro/SerializedDstMatchScoresAttr.h:29-31, formula
// src/libmycu/cupro/SerializedDstMatchScores.cuh:347-396). With d1 >= d2 the
// reference's CUDA build evaluates intercept = 0.35 - (d2*-0.4)*0.05 and
// score = d1*slope + intercept as two fused multiply-adds (nvcc contracts
// them by default), so the table does the same with fmaf.
void build_dms_table(float* T)
{
    volatile float s00 = 0.35f, s200 = -0.4f, inv = 0.05f;
    for (int a1 = 0; a1 < kDstCard; a1++)
        for (int a2 = 0; a2 < kDstCard; a2++) {
            if (a1 == kDstNoData || a2 == kDstNoData) { T[a1 * kDstCard + a2] = -1.0f; continue; }
            int d1 = a1 > a2 ? a1 : a2, d2 = a1 > a2 ? a2 : a1;
            volatile float t = (float)d2 * s200;
            volatile float intpt = std::fmaf(-t, inv, s00);
            volatile float sl0 = s200 - s00;
            volatile float slope = sl0 * inv;
            T[a1 * kDstCard + a2] = std::fmaf((float)d1, slope, intpt);
        }
    // what ddms_diagonal() counts on: multiples of 2^-40 (times 2^-7 there), and
    // no sum of a list's values above 1 after that scaling
    for (int i = 0; i < kDstCard * kDstCard; i++) {
        const float v = std::ldexp(T[i], 40);
        if (v != std::rint(v) || !(T[i] <= 1.0f))
            throw Error(CBP_ERR_ARG, "distance pair scores: a value outside the kernel's range");
    }
}

}  // namespace cbp
