// The distance join's count pass over cell tasks.
//
// One CTA of 128 threads takes a task: up to 128*R query points of one cell in
// groups of 32 (warp w holds groups w, w + 4, .., lane = query, in registers)
// against a stretch of that cell's candidate stream (home cell + owned
// neighbour cells, kernel.cu:1403-1538 in the reference).  Candidates are
// staged in shared memory in steps of SJ_STAGE and read as broadcasts; each
// staged candidate is loaded once per thread and evaluated against all R of
// its queries.  Per block of 32 candidates each thread builds a 32-bit hit mask
// per slot; a 5-step butterfly transposes a warp's 32x32 mask so that lane L
// holds candidate L's hits for the mirrored direction (symmetric traversals
// emit (p,q) and (q,p) from one evaluation).
//
// The pass produces per-key pair counts (the row lengths of a batch) and
// records every hit mask, each run's offset inside its key's run (the value an
// atomicAdd on the key's count returns) and the candidates' point ids; the
// emission pass (sj_emit.cu) writes the pairs from those records at the
// exclusive offsets of the counts, so each key's values land contiguously and
// keys come out ascending -- the order thrust::sort_by_key gives the reference
// (GPU.cu:2336) -- without sorting and without evaluating any distance twice.
//
// Predicate (kernel.cu:344-349): the squared distance in the reference build's
// rounding order (ref_dist2), hit iff sqrt(acc) <= eps, evaluated as acc <= T
// with T the largest double whose rounded sqrt is <= eps (identical by
// monotonicity of the correctly rounded square root).
// FP32 filter: |b|^2 - 2 a.b against T - |a|^2 in local coordinates around the
// home cell's centre; pairs inside a proven error band of the threshold are
// re-evaluated with the exact FP64 arithmetic, so the pair set is the FP64 set.
#include "sj_internal.h"
#include "sj_device.cuh"

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <type_traits>

#ifndef SJ_EVAL_UNROLL
#define SJ_EVAL_UNROLL 2    // unrolling of the per-block candidate loop
#endif

namespace {
using namespace sjdev;
constexpr int kEvalUnroll = SJ_EVAL_UNROLL;

constexpr int NW = SJ_CTA / 32;


// Squared distance in the reference build's exact rounding order (pinned by
// its own outputs): the first addition fuses the FIRST product,
//     acc = fma(d0, d0, d1*d1),  then  acc = fma(dl, dl, acc) for l >= 2,
// with d = cand - query (kernel.cu:344-347).  Padded dimensions hold 0 in both
// points and fma(0, 0, acc) == acc, so padding never changes the result.
template <int DP>
__device__ __forceinline__ double ref_dist2(const double *c, const double *q)
{
    const double d0 = __dsub_rn(c[0], q[0]);
    if (DP == 1) return __dmul_rn(d0, d0);
    const double d1 = __dsub_rn(c[1], q[1]);
    double acc = __fma_rn(d0, d0, __dmul_rn(d1, d1));
#pragma unroll
    for (int l = 2; l < DP; l++) {
        const double d = __dsub_rn(c[l], q[l]);
        acc = __fma_rn(d, d, acc);
    }
    return acc;
}

// N coordinates from dimension l0 on of the point at position pos of the join's
// order, in the widest loads that rows of DP doubles allow (32 bytes, 16 bytes;
// rows start on a multiple of that, the array on 256 bytes): a lane loads its own
// point, so every load instruction touches 32 lines whatever its width.
template <int DP, int L0 = 0, int N = DP>
__device__ __forceinline__ void load_point(const double *__restrict__ xs, uint64_t pos, double *x)
{
    static_assert(L0 % 4 == 0 && L0 + N <= DP, "part of a point");
    const double *const src = xs + pos * DP + L0;
    if constexpr (DP % 4 == 0 && N % 4 == 0) {
#pragma unroll
        for (int l = 0; l < N; l += 4)
            asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                : "=d"(x[l]), "=d"(x[l + 1]), "=d"(x[l + 2]), "=d"(x[l + 3])
                : "l"(src + l));
    } else if constexpr (DP % 2 == 0 && N % 2 == 0) {
#pragma unroll
        for (int l = 0; l < N; l += 2) {
            const double2 v = __ldg(reinterpret_cast<const double2 *>(src + l));
            x[l] = v.x;
            x[l + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int l = 0; l < N; l++) x[l] = __ldg(src + l);
    }
}

// Coordinates and point id of a task's query qi.  The sampling estimate's
// queries are the first of their cell in the index's order: its points in id
// order, so the sample covers the cell whatever the join's order of its points.
template <int DP>
__device__ __forceinline__ uint32_t load_query(const sj_join_args &a, const sj_task &t, uint32_t qi, int D,
                                               double (&x)[DP])
{
    if (t.flags & SJ_TASK_SAMPLE) {
        const uint32_t id = a.indexIds[t.qBegin + qi];
#pragma unroll
        for (int l = 0; l < DP; l++) x[l] = l < D ? a.pts[(uint64_t)id * D + l] : 0.0;
        return id;
    }
    const uint64_t pos = t.qBegin + qi;
    load_point<DP>(a.xs, pos, x);
    return a.ids[pos];
}

template <int DP>
__device__ __forceinline__ bool exact_hit(const sj_join_args &a, uint32_t cpos, const sj_task &t, uint32_t qi, int D,
                                          double T)
{
    double q[DP];
    load_query<DP>(a, t, qi, D, q);
    return ref_dist2<DP>(a.xs + (uint64_t)cpos * DP, q) <= T;
}

template <int DP>
struct __align__(16) Stage64 {
    static constexpr int S = (DP <= 8) ? SJ_STAGE : SJ_STAGE / 2;   // divides 1024: 32 blocks of live bits
    double c[S][DP];
};

// FP32 stage: candidates in pairs (2p, 2p+1) so that one packed f32x2
// instruction evaluates a query against both; per pair, float2 0 holds the
// two |b|^2 and float2 1+l the two local coordinates l.
template <int DP>
struct __align__(16) Stage32 {
    static constexpr int CW2 = ((DP + 1) + 1) / 2 * 2;   // float2 per pair, even (16-byte rows)
    static constexpr int S = SJ_STAGE;
    float2 c[S / 2][CW2];
};

template <int DP, bool F32>
struct StageOf { using T = Stage64<DP>; };
template <int DP>
struct StageOf<DP, true> { using T = Stage32<DP>; };

// mask << 1 | sign bit of v: one funnel shift (the value's bits are not
// inspected as a float, so no comparison is generated)
__device__ __forceinline__ uint32_t push_sign(uint32_t mask, float v)
{
    uint32_t r;
    asm("shf.l.wrap.b32 %0, %1, %2, 1;" : "=r"(r) : "r"(__float_as_uint(v)), "r"(mask));
    return r;
}

// FP32 filter over one block of 32 staged candidates for slots R0..R0+RR-1.
//   y = (|b|^2 - tLo) + sum_l (-2 a_l) b_l      (packed f32x2: two candidates per op)
// hit bit <- sign(y): y < 0 proves the FP64 predicate true; y >= delta proves
// it false; 0 <= y < delta is the borderline band.  Bits are shifted in from
// candidate 31 down to 0, so bit i is candidate i.  Instead of a second
// comparison per candidate, lo[r] keeps the smallest bit pattern of y over the
// block: a y in [0, delta) has a smaller pattern than delta's (non-negative
// floats order like their bits; negative ones have the sign bit and never win
// the unsigned minimum), so ymin < bits(delta) tells that the block has a
// borderline candidate, which near_bits() then finds.
template <int DP, int R0, int RR, int R>
__device__ __forceinline__ void eval_block_f32(const Stage32<DP> &st, uint32_t pb, const float2 (&qa)[R][DP],
                                               const float2 (&nt)[R], uint32_t (&hit)[R], uint32_t (&ymin)[R])
{
    constexpr int CW2 = Stage32<DP>::CW2;
#pragma unroll kEvalUnroll
    for (int p = 15; p >= 0; p--) {
        const float4 *row = reinterpret_cast<const float4 *>(&st.c[pb + p][0]);
        float2 y[RR];
        {
            const float4 v = row[0];
            const float2 nb = make_float2(v.x, v.y);
#pragma unroll
            for (int r = 0; r < RR; r++) y[r] = __fadd2_rn(nb, nt[R0 + r]);
            if (DP >= 1) {
                const float2 b = make_float2(v.z, v.w);
#pragma unroll
                for (int r = 0; r < RR; r++) y[r] = __ffma2_rn(qa[R0 + r][0], b, y[r]);
            }
        }
#pragma unroll
        for (int h = 1; h < CW2 / 2; h++) {
            const float4 v = row[h];
            if (2 * h - 1 < DP) {
                const float2 b = make_float2(v.x, v.y);
#pragma unroll
                for (int r = 0; r < RR; r++) y[r] = __ffma2_rn(qa[R0 + r][2 * h - 1], b, y[r]);
            }
            if (2 * h < DP) {
                const float2 b = make_float2(v.z, v.w);
#pragma unroll
                for (int r = 0; r < RR; r++) y[r] = __ffma2_rn(qa[R0 + r][2 * h], b, y[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < RR; r++) {
            hit[R0 + r] = push_sign(hit[R0 + r], y[r].y);
            hit[R0 + r] = push_sign(hit[R0 + r], y[r].x);
            ymin[R0 + r] = min(ymin[R0 + r], min(__float_as_uint(y[r].x), __float_as_uint(y[r].y)));
        }
    }
}

// Borderline candidates of one block for the query of slot qa/nt: the same
// FP32 operations as eval_block_f32 in the same order (so y is bitwise the
// same), one candidate at a time; bit i set when 0 <= y_i < delta.  Runs only
// for blocks whose minimum says that such a candidate exists.
template <int DP>
__device__ __forceinline__ uint32_t near_bits(const Stage32<DP> &st, uint32_t pb, const float2 (&qa)[DP], float2 nt,
                                           float delta)
{
    constexpr int CW2 = Stage32<DP>::CW2;
    uint32_t m = 0;
    for (int p = 0; p < 16; p++) {
        const float *row = reinterpret_cast<const float *>(&st.c[pb + p][0]);
        for (int h = 0; h < 2; h++) {
            float y = __fadd_rn(row[h], nt.x);
#pragma unroll
            for (int l = 0; l < DP; l++) y = __fmaf_rn(qa[l].x, row[2 * (1 + l) + h], y);
            if (__float_as_uint(y) < __float_as_uint(delta)) m |= 1u << (2 * p + h);
        }
    }
    (void)CW2;
    return m;
}

// FP64 predicate over one block of 32 staged candidates for slots R0..R0+RR-1, in
// the reference's rounding order (ref_dist2).  acc >= 0, so acc <= T is the
// sign of bits(acc) - (bits(T) + 1) as 64-bit integers.
template <int DP, int R0, int RR, int R>
__device__ __forceinline__ void eval_block_f64(const Stage64<DP> &st, uint32_t jb, const double (&q)[R][DP],
                                               long long T1, uint32_t (&hit)[R])
{
#pragma unroll kEvalUnroll
    for (int jj = 31; jj >= 0; jj--) {
        const double *cb = &st.c[jb + jj][0];
        double acc[RR];
        {
            const double c0 = cb[0];
            if (DP == 1) {
#pragma unroll
                for (int r = 0; r < RR; r++) {
                    const double d0 = __dsub_rn(c0, q[R0 + r][0]);
                    acc[r] = __dmul_rn(d0, d0);
                }
            } else {
                const double c1 = cb[DP > 1 ? 1 : 0];
#pragma unroll
                for (int r = 0; r < RR; r++) {
                    const double d0 = __dsub_rn(c0, q[R0 + r][0]);
                    const double d1 = __dsub_rn(c1, q[R0 + r][DP > 1 ? 1 : 0]);
                    acc[r] = __fma_rn(d0, d0, __dmul_rn(d1, d1));
                }
            }
        }
#pragma unroll
        for (int l = 2; l < DP; l++) {
            const double cl = cb[l];
#pragma unroll
            for (int r = 0; r < RR; r++) {
                const double d = __dsub_rn(cl, q[R0 + r][l]);
                acc[r] = __fma_rn(d, d, acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < RR; r++) {
            const long long diff = __double_as_longlong(acc[r]) - T1;
            hit[R0 + r] = push_sign(hit[R0 + r], __int_as_float((int)((unsigned long long)diff >> 32)));
        }
    }
}

// Minimum and maximum of v over the warp (every lane takes part).  volatile: its
// callers use the result in one lane only, and a plain asm may be moved there.
__device__ __forceinline__ float2 warp_min_max(float lo, float hi)
{
    float2 r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r.x) : "f"(lo));
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r.y) : "f"(hi));
    return r;
}

// Evaluates block jb of the stage for the slots of act (a subset of the warp's
// nAct slots; other slots' results are undefined).  All slots, or three of four,
// go through the code that loads each candidate once for all of them.
template <int DP, bool F32, int R, class Eval>
__device__ __forceinline__ void eval_slots(uint32_t act, uint32_t nAct, Eval eval)
{
    if (R == 1 || nAct == 1) {
        eval(std::integral_constant<int, 0>{}, std::integral_constant<int, 1>{});
        return;
    }
    if constexpr (R == 2) {
        if (act == 3u) eval(std::integral_constant<int, 0>{}, std::integral_constant<int, 2>{});
        else if (act == 1u) eval(std::integral_constant<int, 0>{}, std::integral_constant<int, 1>{});
        else eval(std::integral_constant<int, 1>{}, std::integral_constant<int, 1>{});
    }
    if constexpr (R == 4) {
        if (__popc(act) >= 3) {
            eval(std::integral_constant<int, 0>{}, std::integral_constant<int, 4>{});
            return;
        }
        if (act == 3u) {
            eval(std::integral_constant<int, 0>{}, std::integral_constant<int, 2>{});
            return;
        }
        if (act == 12u) {
            eval(std::integral_constant<int, 2>{}, std::integral_constant<int, 2>{});
            return;
        }
        if (act & 1u) eval(std::integral_constant<int, 0>{}, std::integral_constant<int, 1>{});
        if (act & 2u) eval(std::integral_constant<int, 1>{}, std::integral_constant<int, 1>{});
        if (act & 4u) eval(std::integral_constant<int, 2>{}, std::integral_constant<int, 1>{});
        if (act & 8u) eval(std::integral_constant<int, 3>{}, std::integral_constant<int, 1>{});
    }
    static_assert(R == 1 || R == 2 || R == 4, "slot sets of eval_slots");
}

// Shared memory of one count-pass CTA.
template <int DP, bool F32, int R>
struct __align__(16) JoinSmem {
    using Stage = typename StageOf<DP, F32>::T;
    static constexpr int S = Stage::S;
    Stage st;
    uint32_t candId[S];
    uint32_t segStart[SJ_MAX_SEG];
    uint32_t segPre[SJ_MAX_SEG + 1];
    uint32_t colCnt[NW][S];
    float2 boxC[S / 32][DP];            // per staged block: (min, max) of each local coordinate
    float2 boxQ[NW * R][DP];            // per group of 32 queries
    double originS[DP];
    uint32_t scanTmp[NW];
    uint32_t curTask;
    unsigned long long taskPairs;
    unsigned long long taskEvals;
    unsigned long long taskRefined;
};

// Count pass over tasks [taskBegin, taskEnd): per-key pair counts (keyCount,
// both directions of symmetric tasks), the batch total, and -- when a.masks is
// set -- every query's hit mask per block of 32 stream positions plus its row
// count, which the emission pass turns into pairs without a second distance
// evaluation.
// Resident CTAs per SM the register allocation must allow.  Count passes in ms on
// exponential sets of 60k to 1M points, batches of 2e8 pairs (1-D: 0.06 to 0.08, a
// launch's latency):
//                               2-D   3-D   4-D   6-D   8-D   12-D  16-D
//   FP32  three                 3.48  2.92  5.28  10.8  2.83  4.57  5.78
//         four (not 6-D)        3.13  2.60  4.55        2.76  4.18  5.54
//         five (6-D)            2.94  2.45  4.35  9.12  2.78  4.12  5.59
//   FP64  one fewer             3.29  3.05  6.06  15.6  4.18  9.04  12.4
//         6, 6, 6, 5, 4, 3, 3   3.17  2.91  6.01  15.3  3.94  8.22  11.7
//         one more              3.12  2.84  6.06  16.2  4.10  8.29  11.4
// (Five have become the better choice for FP32 at two to four dimensions: the kernel
// was another when the line was drawn.)  FP64's chain of dependent operations needs the
// warps more than it minds a few spilled registers (4-D 52 / 60 bytes of stores / loads,
// 6-D 52 / 64, 8-D 8 / 8).
constexpr int sj_join_min_blocks(int DP, bool F32)
{
    if (F32) return DP == 6 ? 5 : 4;
    return DP <= 4 ? 6 : DP <= 6 ? 5 : DP <= 8 ? 4 : 3;
}

template <int DP, bool F32, int R>
__global__ void __launch_bounds__(SJ_CTA, sj_join_min_blocks(DP, F32)) k_join(sj_join_args a, sj_grid_dev g, int queue)
{
    using Smem = JoinSmem<DP, F32, R>;
    constexpr int S = Smem::S;
    __shared__ Smem sm;
    auto &st = sm.st;
    auto &candId = sm.candId;
    auto &segStart = sm.segStart;
    auto &segPre = sm.segPre;
    auto &colCnt = sm.colCnt;
    auto &originS = sm.originS;

    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const int D = g.D;
    const double T = g.thresh;

    const Transpose transpose(lane);
    for (int j = tid; j < NW * S; j += SJ_CTA) (&colCnt[0][0])[j] = 0;

    // this kernel's tasks of the range: entries [first, first + count) of bigList
    const uint32_t first = a.taskBegin - a.smallPre[a.taskBegin];
    const uint32_t count = (a.taskEnd - a.smallPre[a.taskEnd]) - first;
    uint32_t iter = 0;
    for (;;) {
        // ---- fetch the next task
        __syncthreads();
        if (tid == 0) {
            const uint32_t i = queue ? atomicAdd(a.queueHead, 1u) : blockIdx.x + iter;
            sm.curTask = i < count ? a.bigList[first + i] : 0xffffffffu;
            sm.taskPairs = 0ULL;
            sm.taskEvals = 0ULL;
            sm.taskRefined = 0ULL;
        }
        __syncthreads();
        const uint32_t t = sm.curTask;
        if (t == 0xffffffffu || (!queue && iter > 0)) break;
        iter++;
        const sj_task task = a.tasks[t];
        const bool sym = (task.flags & SJ_TASK_SYM) != 0;
        const uint32_t cellA = task.cell;
        const uint32_t aStart = a.cellStart[cellA], aEnd = a.cellStart[cellA + 1];
        const uint32_t nbrBase = a.nbrStart[cellA];
        const uint32_t nSeg = task.segCount;

        // ---- segment table (exclusive prefix of lengths over the task's segments)
        uint32_t locLen[(SJ_MAX_SEG + SJ_CTA - 1) / SJ_CTA];
        uint32_t mySum = 0;
#pragma unroll
        for (int r = 0; r < (SJ_MAX_SEG + SJ_CTA - 1) / SJ_CTA; r++) {
            uint32_t s = tid * ((SJ_MAX_SEG + SJ_CTA - 1) / SJ_CTA) + r;
            uint32_t len = 0;
            if (s < nSeg) {
                uint32_t gs = task.segBase + s;
                uint32_t st0, en;
                if (gs == 0) {
                    st0 = sym ? task.qBegin : aStart;
                    en = aEnd;
                } else {
                    uint32_t b = a.nbrCell[nbrBase + gs - 1];
                    st0 = a.cellStart[b];
                    en = a.cellStart[b + 1];
                }
                segStart[s] = st0;
                len = en - st0;
            }
            locLen[r] = len;
            mySum += len;
        }
        if ((int)tid < DP) {
            // local-coordinate origin: home cell centre (indexed dims), data centre (others)
            double o;
            if ((int)tid < g.k) o = g.minArr[tid] + ((double)a.cellCoord[(uint64_t)cellA * g.k + tid] + 0.5) * g.eps;
            else if ((int)tid < D) o = g.center[tid];
            else o = 0.0;
            originS[tid] = o;
        }
        {
            // block exclusive scan of mySum
            uint32_t x = mySum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            if (lane == 31) sm.scanTmp[warp] = x;
            __syncthreads();
            uint32_t wpre = 0;
            for (uint32_t w = 0; w < warp; w++) wpre += sm.scanTmp[w];
            uint32_t run = wpre + x - mySum;
#pragma unroll
            for (int r = 0; r < (SJ_MAX_SEG + SJ_CTA - 1) / SJ_CTA; r++) {
                uint32_t s = tid * ((SJ_MAX_SEG + SJ_CTA - 1) / SJ_CTA) + r;
                if (s <= nSeg) segPre[s] = run;
                run += locLen[r];
            }
            if (tid == SJ_CTA - 1) segPre[nSeg] = run;   // grand total (also covers nSeg == SJ_MAX_SEG)
        }
        __syncthreads();
        const uint32_t homeEnd = (task.segBase == 0 && (task.flags & SJ_TASK_HOME)) ? segPre[1] : 0u;

        // ---- query points of this warp: slot r holds group r * NW + warp, lane =
        // query; nAct: the warp's groups (warp-uniform).  Neighbouring groups lie
        // close together and go to different warps, so that the warps have about
        // as many tiles left of a stage as each other.
        const uint32_t nG = (task.qCount + 31) / 32;
        const uint32_t nAct = nG > warp ? (nG - warp + NW - 1) / NW : 0u;
        uint32_t qid[R];
        double q64[F32 ? 1 : R][F32 ? 1 : DP];
        float2 qa[F32 ? R : 1][F32 ? DP : 1];   // (-2 a_l, -2 a_l)
        float2 nt[R];                           // (-tLo, -tLo)
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint32_t qi = (uint32_t)r * SJ_CTA + tid;
            const bool v = (uint32_t)r < nAct && qi < task.qCount;
            double src[DP];
            qid[r] = load_query<DP>(a, task, v ? qi : 0u, D, src);
            double na = 0.0;
#pragma unroll
            for (int l = 0; l < DP; l++) {
                const double x = src[l];
                const float ql = (l < D) ? __double2float_rn(x - originS[l]) : 0.0f;
                if (F32) {
                    qa[F32 ? r : 0][F32 ? l : 0] = make_float2(-2.0f * ql, -2.0f * ql);
                    na += (double)ql * (double)ql;
                } else {
                    q64[F32 ? 0 : r][F32 ? 0 : l] = x;
                }
                if ((uint32_t)r < nAct) {
                    const float2 mm = warp_min_max(v ? ql : INFINITY, v ? ql : -INFINITY);
                    if (lane == 0) sm.boxQ[r * NW + warp][l] = mm;
                }
            }
            if (F32) {
                const float tLo = __double2float_rd(T - na - a.margin);
                nt[r] = make_float2(-tLo, -tLo);
            } else {
                nt[r] = make_float2(0.f, 0.f);
            }
        }
        const long long T1 = __double_as_longlong(T) + 1;
        uint32_t *const liveBase = a.masks ? a.masks + (a.maskOff[t] - a.maskOff[a.taskBegin]) : nullptr;
        uint32_t *const colBase = (a.colMasks && sym) ? a.colMasks + (a.colOff[t] - a.colOff[a.taskBegin]) : nullptr;
        const uint64_t candRecOff = a.candOff ? a.candOff[t] - a.candOff[a.taskBegin] : 0;
        uint32_t *const candIdRec = a.candId ? a.candId + candRecOff : nullptr;
        uint32_t *const candRelRec = (a.candRel && sym) ? a.candRel + candRecOff : nullptr;

        uint32_t rowCount[R];   // pairs keyed by each query
        uint32_t live[R];       // blocks of the current 32 in which the group has a hit
        uint32_t colPairs = 0;  // pairs keyed by the candidates this thread adds up
        uint32_t evals = 0;     // candidate evaluations
        uint32_t refined = 0;   // FP32 borderline re-evaluations
#pragma unroll
        for (int r = 0; r < R; r++) rowCount[r] = live[r] = 0;

        // the stream can never extend past the segments actually present
        const uint32_t sEnd = min(task.sEnd, segPre[nSeg]);
        const uint32_t nBlk = (sEnd - task.sBegin + 31) / 32;
        uint32_t *const rowBase = liveBase ? liveBase + sj_live_words(nBlk, nG) : nullptr;
        for (uint32_t sBase = task.sBegin; sBase < sEnd; sBase += S) {
            const uint32_t nIn = min((uint32_t)S, sEnd - sBase);
            __syncthreads();
            // ---- stage candidates
            for (uint32_t j0 = warp * 32; j0 < nIn; j0 += SJ_CTA) {   // a warp stages whole blocks
                const uint32_t j = j0 + lane;
                const bool in = j < nIn;
                float bl[DP];
                if (in) {
                    uint32_t s = sBase + j;
                    uint32_t lo = 0, hi = nSeg;   // largest seg with segPre[seg] <= s
                    while (hi - lo > 1) {
                        uint32_t mid = (lo + hi) >> 1;
                        if (segPre[mid] <= s) lo = mid; else hi = mid;
                    }
                    uint32_t pos = segStart[lo] + (s - segPre[lo]);
                    const uint32_t cid = a.ids[pos];
                    candId[j] = cid;
                    if (candIdRec) candIdRec[s - task.sBegin] = cid;   // the emission's candidate record
                    double src[DP];
                    load_point<DP>(a.xs, pos, src);
                    double nb = 0.0;
#pragma unroll
                    for (int l = 0; l < DP; l++) {
                        const double x = src[l];
                        bl[l] = (l < D) ? __double2float_rn(x - originS[l]) : 0.0f;
                        if constexpr (F32) {
                            float *dst = reinterpret_cast<float *>(&st.c[j >> 1][0]) + (j & 1);
                            dst[2 * (1 + l)] = bl[l];
                            nb += (double)bl[l] * (double)bl[l];
                        } else {
                            st.c[j][l] = x;
                        }
                    }
                    if constexpr (F32) reinterpret_cast<float *>(&st.c[j >> 1][0])[j & 1] = __double2float_rn(nb);
                }
#pragma unroll
                for (int l = 0; l < DP; l++) {
                    const float2 mm = warp_min_max(in ? bl[l] : INFINITY, in ? bl[l] : -INFINITY);
                    if (lane == 0) sm.boxC[j0 >> 5][l] = mm;
                }
            }
            __syncthreads();
            // ---- which (group, block) tiles can hold a hit: lane = slot x 8 +
            // block.  Ruled out: boxes further apart than the radius (pruneT
            // covers the rounding of the local coordinates), and home blocks
            // whose positions all come before the group's queries.
            uint32_t tiles;
            {
                const uint32_t r = lane >> 3, bi = lane & 7;
                const uint32_t blk = sBase + bi * 32;
                bool alive = r < nAct && bi * 32 < nIn;
                if (alive) {
                    float d2 = 0.0f;
#pragma unroll
                    for (int l = 0; l < DP; l++) {
                        const float2 q = sm.boxQ[r * NW + warp][l], cb = sm.boxC[bi][l];
                        const float gap = fmaxf(0.0f, fmaxf(cb.x - q.y, q.x - cb.y));
                        d2 = fmaf(gap, gap, d2);
                    }
                    alive = !(d2 > a.pruneT) && !(sym && blk + 32 <= min(homeEnd, (r * NW + warp) * 32));
                }
                tiles = __ballot_sync(0xffffffffu, alive);
            }
            // ---- hit masks of the blocks that have a tile left.  Only these are
            // visited, and everything a tile needs beyond its distances waits for a
            // hit (record addresses, counts) or for the end of the stage (live
            // bits): with 32 blocks of distances at ~130 instructions a slot, the
            // rest of a tile counts as much.  Count pass at 2-D 21.3 to 15.4 ms,
            // 4-D 39.3 to 30.7, 6-D 74.6 to 62.2 (1M points), 8-D 6.56 to 6.34
            // against visiting every block with all of it.
            uint32_t blocks = (tiles | (tiles >> 8) | (tiles >> 16) | (tiles >> 24)) & 0xffu;
#pragma unroll 1
            while (blocks) {
                const uint32_t bi = __ffs(blocks) - 1;
                blocks &= blocks - 1;
                const uint32_t jb = bi * 32, blk = sBase + jb;
                const uint32_t nb = min(32u, nIn - jb);
                const uint32_t inRange = 0xffffffffu >> (32u - nb);
                const uint32_t col = (tiles >> bi) & 0x01010101u;   // bit 8 r: slot r
                const uint32_t act = (col | (col >> 7) | (col >> 14) | (col >> 21)) & 15u;
                uint32_t hits[R], ymin[R];
#pragma unroll
                for (int r = 0; r < R; r++) { hits[r] = 0; ymin[r] = 0xffffffffu; }
                eval_slots<DP, F32, R>(act, nAct, [&](auto r0, auto rr) {
                    if constexpr (F32)
                        eval_block_f32<DP, decltype(r0)::value, decltype(rr)::value, R>(st, jb >> 1, qa, nt, hits, ymin);
                    else
                        eval_block_f64<DP, decltype(r0)::value, decltype(rr)::value, R>(st, jb, q64, T1, hits);
                });
                const uint32_t hb = home_bits(blk, homeEnd, sym);
                const uint32_t bInTask = (blk - task.sBegin) >> 5;
                uint32_t colHits = 0;   // this lane's candidate: hits over the warp's slots
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (!((act >> r) & 1u)) continue;   // warp-uniform
                    const uint32_t qi = (uint32_t)r * SJ_CTA + tid;
                    const bool qValid = qi < task.qCount;
                    uint32_t rowValid = qValid ? inRange : 0u;
                    if (hb) rowValid &= row_keep(qi, blk, hb);
                    uint32_t h = hits[r];
                    if constexpr (F32) {
                        if (ymin[r] < __float_as_uint(a.delta)) {
                            uint32_t bm = near_bits<DP>(st, jb >> 1, qa[r], nt[r], a.delta) & ~h & rowValid;
                            while (bm) {
                                const int jj = __ffs(bm) - 1;
                                bm &= bm - 1;
                                const uint32_t s = blk + jj;
                                uint32_t lo = 0, hi = nSeg;
                                while (hi - lo > 1) {
                                    const uint32_t mid = (lo + hi) >> 1;
                                    if (segPre[mid] <= s) lo = mid; else hi = mid;
                                }
                                const uint32_t cpos = segStart[lo] + (s - segPre[lo]);
                                refined++;
                                if (exact_hit<DP>(a, cpos, task, qi, D, T)) h |= 1u << jj;
                            }
                        }
                    }
                    const uint32_t rowMask = h & rowValid;   // lane = query, bit = candidate
                    if (!__any_sync(0xffffffffu, rowMask)) continue;   // no hit in the tile
                    live[r] |= 1u << (bInTask & 31);
                    // row words [block][query], column words [block][query group][candidate]
                    if (rowBase && qValid) rowBase[bInTask * task.qCount + qi] = rowMask;
                    rowCount[r] += __popc(rowMask);
                    if (sym) {
                        // the mirrored direction: lane L gets candidate L's hits
                        uint32_t mir = rowMask;
                        if (hb) mir &= mir_keep(qi, blk, hb);
                        const uint32_t colW = transpose(mir);
                        colHits += __popc(colW);
                        if (colBase) colBase[bInTask * nG * 32 + qi] = colW;
                    }
                }
                if (sym) colCnt[warp][jb + lane] = colHits;
            }
            // the live bits of 32 blocks are complete (a stage never crosses them)
            const uint32_t bEnd = (sBase + nIn - task.sBegin + 31) >> 5;   // blocks so far
            if ((bEnd & 31) == 0 || bEnd == nBlk) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (liveBase && (uint32_t)r < nAct && lane == 0)
                        liveBase[((bEnd - 1) >> 5) * nG + r * NW + warp] = live[r];
                    live[r] = 0;
                }
            }
            if (sym) {
                __syncthreads();
                for (uint32_t j = tid; j < nIn; j += SJ_CTA) {
                    uint32_t tot = 0;
#pragma unroll
                    for (int w = 0; w < NW; w++) { tot += colCnt[w][j]; colCnt[w][j] = 0; }
                    // the count before this stage's addition is the offset of
                    // these column pairs inside the candidate's key run
                    const uint32_t rel = tot ? atomicAdd(&a.keyCount[candId[j]], tot) : 0u;
                    if (candRelRec) candRelRec[sBase + j - task.sBegin] = rel;
                    colPairs += tot;
                }
            }
        }
        {
            unsigned long long mine = colPairs;
            uint32_t *const relBase = a.rowRel ? a.rowRel + (a.rowOff[t] - a.rowOff[a.taskBegin]) : nullptr;
#pragma unroll
            for (int r = 0; r < R; r++) {
                if ((uint32_t)r >= nAct) continue;
                const uint32_t qi = (uint32_t)r * SJ_CTA + tid;
                // evaluations of this query: stream positions [sBegin, sEnd), in the
                // symmetric home segment only those at or after the query itself
                if (qi < task.qCount) {
                    const uint32_t from = max(task.sBegin, min(qi, sym ? homeEnd : 0u));
                    evals += sEnd > from ? sEnd - from : 0u;
                }
                // the key's count before this addition: where this task's row
                // run starts inside the query's key run
                const uint32_t rel = rowCount[r] ? atomicAdd(&a.keyCount[qid[r]], rowCount[r]) : 0u;
                if (relBase && qi < task.qCount) relBase[qi] = rel;
                mine += rowCount[r];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
            if (lane == 0 && mine) atomicAdd(&sm.taskPairs, mine);
        }
        // ---- statistics (per task: a re-run of the task overwrites them)
        unsigned long long e = evals, rf = refined;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            e += __shfl_xor_sync(0xffffffffu, e, o);
            rf += __shfl_xor_sync(0xffffffffu, rf, o);
        }
        if (lane == 0) {
            if (e) atomicAdd(&sm.taskEvals, e);
            if (rf) atomicAdd(&sm.taskRefined, rf);
        }
        __syncthreads();
        if (tid == 0) {
            const unsigned long long tp = sm.taskPairs;
            if (tp) {
                atomicAdd(&a.stat[2], tp);
                if (a.batchPairs) atomicAdd(a.batchPairs, tp);
            }
            if (a.taskHits) a.taskHits[t] = (uint32_t)min(tp, 0xffffffffULL);
            if (a.taskEvals) a.taskEvals[t] = (uint32_t)min(sm.taskEvals, 0xffffffffULL);
            if (a.taskRefined) a.taskRefined[t] = (uint32_t)min(sm.taskRefined, 0xffffffffULL);
        }
    }
}

// ------------------------------------------------- tasks of few queries --
// Count pass over the tasks of at most SJ_SMALL_QUERIES query points: one warp a
// task, lane = candidate.  k_join's CTA would leave most of its lanes without a
// query on sparse grids (two points a cell: 2 of 128); here every lane evaluates
// its candidate against the task's queries in turn (packed two per FP32
// instruction), a ballot is the query's row word, the lane's own bits are the
// candidate's column word, and no barrier or segment table is needed: the
// segments go by 32 at a time in registers.  Same operations in the same order
// as k_join, same records.
// Bound: instruction issue (per block of 32 candidates ~60 instructions and
// ~12 + D per query), and for wide points the conversions of the candidates'
// coordinates to FP32 and back for |b|^2, four lanes a cycle each: what the test
// of the first-loaded dimensions saves.  The tasks of 1M clustered points in 16-D
// took k_join 20.4 ms more than its other tasks, this kernel 4.7 ms.
// Dimensions that are loaded and tested first, the last of the padded width: a
// point whose distance in these alone exceeds the radius is out.  The last
// dimensions, because the grid has already put the first (indexed) ones close
// together.  Points of 12 or 16 only: 1M clustered points in 16-D, 9.63 to 4.68 ms
// (5.23 with four dimensions); 500k in 12-D 1.86 to 1.67 (1.87 with four); in 8-D
// the test of the last four gives nothing (1.49 ms either way).
template <int DP>
constexpr int PRE_DIMS = DP >= 12 ? 8 : 0;

template <int DP, bool F32>
struct __align__(16) SmallSmem {
    static constexpr int CW2 = Stage32<DP>::CW2;
    // FP32: per pair of queries the two (-tLo), then the two (-2 a_l) of each dimension
    float2 q2[F32 ? SJ_SMALL_QUERIES / 2 : 1][CW2];
    double q[F32 ? 1 : SJ_SMALL_QUERIES][DP];
    float2 box[DP];             // (min, max) of the queries' local coordinates
    double origin[DP];
    // per pair of queries the (-a_l) of the dimensions that are tested first
    float2 pre[PRE_DIMS<DP> ? SJ_SMALL_QUERIES / 2 : 1][PRE_DIMS<DP> ? PRE_DIMS<DP> : 2];
};

// Squared distance of a point's dimensions [L0, L0 + N) to the box, in FP32.
template <int L0, int N>
__device__ __forceinline__ float box_dist2(const float2 *box, const float *x)
{
    float d2 = 0.0f;
#pragma unroll
    for (int l = L0; l < L0 + N; l++) {
        const float2 q = box[l];
        const float gap = fmaxf(0.0f, fmaxf(x[l] - q.y, q.x - x[l]));
        d2 = fmaf(gap, gap, d2);
    }
    return d2;
}

// Queries from which on testing a block against their box pays: clusters of two points
// a cell, 12-D / 16-D 2.03 / 2.37 ms of count pass with 6, 2.12 / 2.44 with 3, 1.99 /
// 2.32 with 12; below 12 dimensions no difference.
constexpr uint32_t SMALL_BOX = 6;

// Resident CTAs per SM: 3-D / 2-D / 6-D / 8-D / 12-D / 16-D, FP32, 0.173 / 0.364 / 1.60 /
// 1.95 / 2.03 / 2.37 ms with these, 0.191 / 0.420 / 1.80 / 2.04 / 2.42 / 2.72 with one
// fewer, 0.168 / 0.329 / 1.70 / 2.31 / 2.26 / 2.90 with one more (spills; 8-D FP32 spills
// 92 / 68 bytes of stores / loads as it is).
template <int DP, bool F32>
__global__ void __launch_bounds__(SJ_CTA, DP <= 4 ? 6 : DP <= 8 ? 5 : 4) k_join_small(sj_join_args a, sj_grid_dev g, int queue)
{
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int PD = PRE_DIMS<DP>;
    constexpr int ND = PD ? PD : DP;   // dimensions loaded ahead
    __shared__ SmallSmem<DP, F32> smem[NW];
    const uint32_t lane = threadIdx.x & 31u;
    SmallSmem<DP, F32> &sm = smem[threadIdx.x >> 5];
    const int D = g.D;
    const double T = g.thresh;
    const uint32_t deltaBits = __float_as_uint(a.delta);
    const uint32_t first = a.smallPre[a.taskBegin];
    const uint32_t count = a.smallPre[a.taskEnd] - first;
    const uint32_t warps = gridDim.x * NW;
    unsigned long long pairsAll = 0;
    uint32_t i = blockIdx.x * NW + (threadIdx.x >> 5);
    for (;;) {
        if (queue) {
            if (lane == 0) i = atomicAdd(a.queueHead + 1, 1u);
            i = __shfl_sync(FULL, i, 0);
        }
        if (i >= count) break;
        const uint32_t t = a.smallList[first + i];
        i += warps;
        const sj_task task = a.tasks[t];
        const bool sym = (task.flags & SJ_TASK_SYM) != 0;
        const uint32_t qc = task.qCount;
        const uint32_t aStart = a.cellStart[task.cell], aEnd = a.cellStart[task.cell + 1];
        const uint32_t nbrBase = a.nbrStart[task.cell];
        const uint32_t homeEnd = (task.segBase == 0 && (task.flags & SJ_TASK_HOME)) ? aEnd - (sym ? task.qBegin : aStart)
                                                                                   : 0u;
        __syncwarp();   // the previous task is done with the warp's shared memory
        if ((int)lane < DP) {
            // local-coordinate origin, as k_join's
            double o;
            if ((int)lane < g.k) o = g.minArr[lane] + ((double)a.cellCoord[(uint64_t)task.cell * g.k + lane] + 0.5) * g.eps;
            else if ((int)lane < D) o = g.center[lane];
            else o = 0.0;
            sm.origin[lane] = o;
        }
        __syncwarp();
        uint32_t qid;
        {
            double src[DP];
            qid = load_query<DP>(a, task, lane < qc ? lane : 0u, D, src);
            double na = 0.0;
#pragma unroll
            for (int l = 0; l < DP; l++) {
                const double x = src[l];
                const float ql = (l < D && lane < qc) ? __double2float_rn(x - sm.origin[l]) : 0.0f;
                if (qc >= SMALL_BOX) {
                    const float2 mm = warp_min_max(lane < qc ? ql : INFINITY, lane < qc ? ql : -INFINITY);
                    if (lane == 0) sm.box[l] = mm;
                }
                if constexpr (PD > 0) {   // no query: infinitely far
                    if (l >= DP - PD)
                        reinterpret_cast<float *>(&sm.pre[lane >> 1][l - (DP - PD)])[lane & 1] = lane < qc ? -ql : INFINITY;
                }
                if constexpr (F32) {
                    reinterpret_cast<float *>(&sm.q2[lane >> 1][1 + l])[lane & 1] = -2.0f * ql;
                    na += (double)ql * (double)ql;
                } else {
                    sm.q[lane][l] = x;
                }
            }
            if constexpr (F32) {
                const float tLo = __double2float_rd(T - na - a.margin);
                reinterpret_cast<float *>(&sm.q2[lane >> 1][0])[lane & 1] = lane < qc ? -tLo : INFINITY;
            }
        }
        __syncwarp();
        uint32_t *const liveBase = a.masks ? a.masks + (a.maskOff[t] - a.maskOff[a.taskBegin]) : nullptr;
        uint32_t *const colBase = (a.colMasks && sym) ? a.colMasks + (a.colOff[t] - a.colOff[a.taskBegin]) : nullptr;
        const uint64_t candRecOff = a.candOff ? a.candOff[t] - a.candOff[a.taskBegin] : 0;
        uint32_t *const candIdRec = a.candId ? a.candId + candRecOff : nullptr;
        uint32_t *const candRelRec = (a.candRel && sym) ? a.candRel + candRecOff : nullptr;
        const uint32_t nBlk = (task.sEnd - task.sBegin + 31) / 32;
        uint32_t *const rowBase = liveBase ? liveBase + sj_live_words(nBlk, 1) : nullptr;

        uint32_t rowCount = 0, colCount = 0, live = 0, refined = 0;
        // the current 32 segments: lane's start, and prefix of their lengths (stream positions)
        uint32_t seg = 0, segStart = 0, segLen = 0, segIncl = 0, segEnd = 0;   // segEnd: stream position after them
        // candidate of stream position blk + lane, for ascending blocks
        auto locate = [&](uint32_t blk) -> uint32_t {
            const uint32_t s = blk + lane;
            uint32_t cpos = 0;
            for (;;) {
                {
                    // positions inside the current segments: the first with prefix > s
                    const uint32_t base = segEnd - __shfl_sync(FULL, segIncl, 31);   // position of the first one
                    uint32_t lo = 0;
#pragma unroll
                    for (int w = 16; w > 0; w >>= 1) {
                        const uint32_t v = __shfl_sync(FULL, segIncl, lo + w - 1);
                        if (base + v <= s) lo += w;
                    }
                    lo = min(lo, 31u);
                    const uint32_t st = __shfl_sync(FULL, segStart, lo);
                    const uint32_t ex = __shfl_sync(FULL, segIncl - segLen, lo);
                    if (s >= base && s < segEnd) cpos = st + (s - base - ex);
                }
                if (segEnd > blk + 31 || segEnd >= task.sEnd || seg >= task.segCount) return cpos;   // warp-uniform
                // ---- the next 32 segments
                const uint32_t mySeg = seg + lane;
                segStart = segLen = 0;
                if (mySeg < task.segCount) {
                    const uint32_t gs = task.segBase + mySeg;
                    if (gs == 0) {
                        segStart = sym ? task.qBegin : aStart;
                        segLen = aEnd - segStart;
                    } else {
                        const uint32_t nb = a.nbrCell[nbrBase + gs - 1];
                        segStart = a.cellStart[nb];
                        segLen = a.cellStart[nb + 1] - segStart;
                    }
                }
                segIncl = segLen;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, segIncl, o);
                    if (lane >= (uint32_t)o) segIncl += y;
                }
                segEnd += __shfl_sync(FULL, segIncl, 31);
                seg += 32;
            }
        };
        // the next block's candidates are loaded while this one is evaluated
        uint32_t nPos = locate(task.sBegin), nId = a.ids[nPos];
        double nx[ND];
        load_point<DP, DP - ND, ND>(a.xs, nPos, nx);
#pragma unroll 1
        for (uint32_t b = 0; b < nBlk; b++) {
            const uint32_t blk = task.sBegin + 32 * b;
            const uint32_t s = blk + lane;
            const bool in = s < task.sEnd;
            const uint32_t cpos = nPos, cid = nId;
            double c[DP];
#pragma unroll
            for (int l = 0; l < ND; l++) c[DP - ND + l] = nx[l];
            if (b + 1 < nBlk) {
                nPos = locate(blk + 32);
                nId = a.ids[nPos];
                load_point<DP, DP - ND, ND>(a.xs, nPos, nx);
            }
            if (candIdRec && in) candIdRec[s - task.sBegin] = cid;
            const bool home = sym && s < homeEnd;
            const bool anyHome = sym && blk < homeEnd;   // warp-uniform
            uint32_t rowWord = 0, colW = 0;
            float bl[DP];
#pragma unroll
            for (int l = DP - ND; l < DP; l++) bl[l] = (l < D) ? __double2float_rn(c[l] - sm.origin[l]) : 0.0f;
            // the block is ruled out when every candidate lies further from the
            // queries (few) or their box than the radius (as k_join's tiles: pruneT
            // holds for single points, and for a part of the dimensions)
            bool alive = true;
            if constexpr (PD > 0) {
                float m = INFINITY;
                if (qc >= SMALL_BOX) {
                    m = box_dist2<DP - PD, PD>(sm.box, bl);
                } else {
                    for (uint32_t p = 0; 2 * p < qc; p++) {
                        float2 d2 = make_float2(0.0f, 0.0f);
                        const float4 *const row4 = reinterpret_cast<const float4 *>(&sm.pre[p][0]);
#pragma unroll
                        for (int l = 0; l < PD; l += 2) {
                            const float4 v = row4[l / 2];
                            const float b0 = bl[DP - PD + l], b1 = bl[DP - PD + l + 1];
                            const float2 t0 = __fadd2_rn(make_float2(b0, b0), make_float2(v.x, v.y));
                            const float2 t1 = __fadd2_rn(make_float2(b1, b1), make_float2(v.z, v.w));
                            d2 = __ffma2_rn(t0, t0, d2);
                            d2 = __ffma2_rn(t1, t1, d2);
                        }
                        m = fminf(m, fminf(d2.x, d2.y));
                    }
                }
                alive = __any_sync(FULL, in && !(m > a.pruneT));
                if (alive) {
                    load_point<DP, 0, DP - PD>(a.xs, cpos, c);
#pragma unroll
                    for (int l = 0; l < DP - PD; l++) bl[l] = (l < D) ? __double2float_rn(c[l] - sm.origin[l]) : 0.0f;
                }
            }
            if (alive && qc >= SMALL_BOX) alive = __any_sync(FULL, in && !(box_dist2<0, DP>(sm.box, bl) > a.pruneT));
            if (!alive) {
                // no hit: nothing to record but the candidates' ids
            } else if constexpr (F32) {
                float2 b2[DP];
                double nbd = 0.0;
#pragma unroll
                for (int l = 0; l < DP; l++) {
                    b2[l] = make_float2(bl[l], bl[l]);
                    nbd += (double)bl[l] * (double)bl[l];
                }
                const float nbf = __double2float_rn(nbd);
                for (uint32_t p = 0; 2 * p < qc; p++) {
                    const float4 *const row4 = reinterpret_cast<const float4 *>(&sm.q2[p][0]);
                    float4 v = row4[0];
                    float2 y = __fadd2_rn(make_float2(nbf, nbf), make_float2(v.x, v.y));
                    y = __ffma2_rn(make_float2(v.z, v.w), b2[0], y);
#pragma unroll
                    for (int h = 1; h < SmallSmem<DP, F32>::CW2 / 2; h++) {
                        v = row4[h];
                        if (2 * h - 1 < DP) y = __ffma2_rn(make_float2(v.x, v.y), b2[2 * h - 1 < DP ? 2 * h - 1 : 0], y);
                        if (2 * h < DP) y = __ffma2_rn(make_float2(v.z, v.w), b2[2 * h < DP ? 2 * h : 0], y);
                    }
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const uint32_t q = 2 * p + e;
                        const float ye = e ? y.y : y.x;
                        bool keep = in && q < qc;
                        if (anyHome) keep = keep && (!home || s >= q);
                        bool h = __float_as_int(ye) < 0;
                        if (__any_sync(FULL, keep && __float_as_uint(ye) < deltaBits)) {
                            if (keep && __float_as_uint(ye) < deltaBits) {
                                refined++;
                                h = exact_hit<DP>(a, cpos, task, q, D, T);
                            }
                        }
                        h = h && keep;
                        const uint32_t word = __ballot_sync(FULL, h);
                        if (lane == q) rowWord = word;
                        colW |= (h ? 1u : 0u) << (q & 31u);
                    }
                }
            } else {
                for (uint32_t q = 0; q < qc; q++) {
                    const double acc = ref_dist2<DP>(c, sm.q[q]);
                    bool h = in && acc <= T;
                    if (anyHome) h = h && (!home || s >= q);
                    const uint32_t word = __ballot_sync(FULL, h);
                    if (lane == q) rowWord = word;
                    colW |= (h ? 1u : 0u) << q;
                }
            }
            if (home) colW &= s < 32u ? ~(1u << s) : FULL;   // the mirrored direction drops the query itself
            rowCount += __popc(rowWord);
            const bool hit = __any_sync(FULL, rowWord);
            if (hit) {
                live |= 1u << (b & 31);
                if (rowBase && lane < qc) rowBase[(uint64_t)b * qc + lane] = rowWord;
            }
            if (sym) {
                const uint32_t n = __popc(colW);
                const uint32_t rel = n ? atomicAdd(&a.keyCount[cid], n) : 0u;
                if (candRelRec && in) candRelRec[s - task.sBegin] = rel;
                if (hit && colBase) colBase[(uint64_t)b * 32 + lane] = colW;
                colCount += n;
            }
            if (liveBase && ((b & 31) == 31 || b + 1 == nBlk)) {
                if (lane == 0) liveBase[b >> 5] = live;
                live = 0;
            }
        }
        uint32_t evals = 0;
        if (lane < qc) {
            const uint32_t from = max(task.sBegin, min(lane, sym ? homeEnd : 0u));
            evals = task.sEnd > from ? task.sEnd - from : 0u;
            const uint32_t rel = rowCount ? atomicAdd(&a.keyCount[qid], rowCount) : 0u;
            if (a.rowRel) a.rowRel[a.rowOff[t] - a.rowOff[a.taskBegin] + lane] = rel;
        }
        // a task's worst case is below 2^32 pairs and evaluations
        const uint32_t hits = __reduce_add_sync(FULL, (sym ? colCount : 0u) + (lane < qc ? rowCount : 0u));
        evals = __reduce_add_sync(FULL, evals);
        if (F32) refined = __reduce_add_sync(FULL, refined);
        if (lane == 0) {
            pairsAll += hits;
            if (a.taskHits) a.taskHits[t] = hits;
            if (a.taskEvals) a.taskEvals[t] = evals;
            if (a.taskRefined) a.taskRefined[t] = refined;
        }
    }
    if (lane == 0 && pairsAll) {
        atomicAdd(&a.stat[2], pairsAll);
        if (a.batchPairs) atomicAdd(a.batchPairs, pairsAll);
    }
}

// ------------------------------------------------------- task sampling --
// Hits of the tasks of cells that have several query tiles, as a sample of each
// task's own queries and candidates says.  In the spatial order inside the cells a
// tile (four runs of 128 neighbouring points) and a stretch of a stream are unlike
// the cell, and a batch of a dense join holds a few tiles of one cell: the cell's
// mean rate for every task does not predict its batches (figures at k_task_pool).
// One warp a task: up to 64 of its queries, two a lane, against up to 64 of its
// stream positions, both evenly spread, in FP32.
// Bound: the FP32 pipe and the candidates' loads: 0.46 ms for 156k tasks in 6-D, whose
// count pass takes 24 ms.  32 x 32 pairs: 3.6 ms less for 2.2M tasks (count pass 471
// ms), task error 9.3 % in place of 5.4.
constexpr int TASK_SAMPLE_WARPS = 8;

// Place of sample i of m over len: `phase` of the way (in 2^-16) through its part.
__device__ __forceinline__ uint32_t sample_at(uint32_t i, uint32_t m, uint32_t len, uint32_t phase)
{
    return (uint32_t)(((((uint64_t)i << 16) + phase) * len) / ((uint64_t)m << 16));
}

// sample: per task (evaluations, -), evaluations 0: not sampled; the second is set
// to the hits of sj_probe_pairs' pairs.
template <int DP>
__global__ void __launch_bounds__(32 * TASK_SAMPLE_WARPS) k_task_sample(sj_taskgen g, const double *__restrict__ xs,
                                                                        float T, const sj_task *__restrict__ tasks,
                                                                        uint32_t nt, float2 *__restrict__ sample)
{
    constexpr int ROW = (DP + 3) / 4 * 4;
    constexpr int QS = SJ_PROBE_QUERIES / 32;   // queries a lane
    __shared__ __align__(16) float cand[TASK_SAMPLE_WARPS][SJ_PROBE_POS][ROW];
    __shared__ uint32_t candPos[TASK_SAMPLE_WARPS][SJ_PROBE_POS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t t = blockIdx.x * TASK_SAMPLE_WARPS + warp;
    if (t >= nt) return;
    if (!(sample[t].x > 0.0f)) return;
    const sj_task task = tasks[t];
    const bool sym = (task.flags & SJ_TASK_SYM) != 0;
    const uint32_t aStart = g.cellStart[task.cell], aEnd = g.cellStart[task.cell + 1];
    const uint32_t homePos = sym ? task.qBegin : aStart;
    const uint32_t homeLen = (task.segBase == 0 && (task.flags & SJ_TASK_HOME)) ? aEnd - homePos : 0u;
    const uint32_t len = task.sEnd - task.sBegin;
    const uint32_t m = min((uint32_t)SJ_PROBE_POS, len), mq = min((uint32_t)SJ_PROBE_QUERIES, task.qCount);
    // the tasks of a tile take other queries each (golden-ratio phases), so that together they cover it
    const uint32_t phase = (t * 40503u) & 0xffffu;
    // local coordinates around the task's first query
    double o[DP];
    load_point<DP>(xs, task.qBegin, o);
    float q[QS][DP];
    uint32_t qPos[QS];
#pragma unroll
    for (int r = 0; r < QS; r++) {
        const uint32_t i = 32 * r + lane;
        qPos[r] = task.qBegin + (i < mq ? sample_at(i, mq, task.qCount, phase) : 0u);
        double x[DP];
        load_point<DP>(xs, qPos[r], x);
#pragma unroll
        for (int l = 0; l < DP; l++) q[r][l] = i < mq ? (float)(x[l] - o[l]) : INFINITY;   // no query: no hit
    }
    for (uint32_t i = lane; i < m; i += 32) {
        const uint32_t s = task.sBegin + sample_at(i, m, len, 0x8000u);
        uint32_t pos;
        if (s < homeLen) {
            pos = homePos + s;
        } else {
            // the owned neighbour that holds the position: the last entry that starts at or before it
            uint32_t lo = g.nbrStart[task.cell], hi = g.nbrStart[task.cell + 1];
            const uint32_t at = g.nbrPre[lo + (task.segBase ? task.segBase - 1u : 0u)] + (s - homeLen);
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (g.nbrPre[mid] <= at) lo = mid; else hi = mid;
            }
            pos = g.cellStart[g.nbrCell[lo]] + (at - g.nbrPre[lo]);
        }
        candPos[warp][i] = pos;
        double x[DP];
        load_point<DP>(xs, pos, x);
#pragma unroll
        for (int l = 0; l < DP; l++) cand[warp][i][l] = (float)(x[l] - o[l]);
    }
    __syncwarp();
    // a point and itself are counted apart: only where the stretch holds queries
    const uint32_t at = task.qBegin - homePos;
    const bool own = homeLen && task.sBegin < at + task.qCount && task.sEnd > at;
    uint32_t hits = 0;
    const auto count = [&](auto skipSelf) {
#pragma unroll 2
        for (uint32_t j = 0; j < m; j++) {
            float b[ROW];
#pragma unroll
            for (int l = 0; l < ROW; l += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(&cand[warp][j][l]);
                b[l] = v.x;
                b[l + 1] = v.y;
                b[l + 2] = v.z;
                b[l + 3] = v.w;
            }
#pragma unroll
            for (int r = 0; r < QS; r++) {
                float d2 = 0.0f;
#pragma unroll
                for (int l = 0; l < DP; l++) {
                    const float d = b[l] - q[r][l];
                    d2 = fmaf(d, d, d2);
                }
                bool hit = d2 <= T;
                if constexpr (decltype(skipSelf)::value) hit = hit && candPos[warp][j] != qPos[r];
                hits += hit ? 1u : 0u;
            }
        }
    };
    if (own) count(std::true_type{});
    else count(std::false_type{});
    hits = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0) sample[t].y = (float)hits;
}

template <class Kernel>
int occupancy_of(Kernel k, std::atomic<int> (&occ)[64])
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    int o = occ[dev].load();   // per device ordinal, 0 = not measured yet
    if (o == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, SJ_CTA, 0);
        o = b > 0 ? b : 1;
        occ[dev].store(o);
    }
    return o;
}

template <int DP, bool F32>
cudaError_t launch_one(const sj_join_args &a, const sj_grid_dev &g, int queue, uint32_t nBig, uint32_t nSmall,
                       int numSM, int maxCtasPerSM, cudaStream_t s)
{
    static std::atomic<int> occBig[64], occSmall[64];
    // persistent queue: one full wave of resident CTAs (or fewer per SM, to
    // leave room for a kernel of the other stream)
    if (nBig) {
        int perSM = occupancy_of(k_join<DP, F32, sj_query_slots(DP, F32)>, occBig);
        if (maxCtasPerSM > 0 && maxCtasPerSM < perSM) perSM = maxCtasPerSM;
        unsigned grid = queue ? (unsigned)(numSM * perSM) : nBig;
        if (queue && grid > nBig) grid = nBig;
        k_join<DP, F32, sj_query_slots(DP, F32)><<<grid, SJ_CTA, 0, s>>>(a, g, queue);
        sj_note_launch();
    }
    if (nSmall) {
        const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)numSM * occupancy_of(k_join_small<DP, F32>, occSmall),
                                                           ((uint64_t)nSmall + NW - 1) / NW);
        k_join_small<DP, F32><<<grid, SJ_CTA, 0, s>>>(a, g, queue);
        sj_note_launch();
    }
    return cudaGetLastError();
}

template <int DP>
cudaError_t launch_dp(const sj_join_args &a, const sj_grid_dev &g, int fp32, int queue, uint32_t nBig, uint32_t nSmall,
                      int numSM, int maxCtas, cudaStream_t s)
{
    return fp32 ? launch_one<DP, true>(a, g, queue, nBig, nSmall, numSM, maxCtas, s)
                : launch_one<DP, false>(a, g, queue, nBig, nSmall, numSM, maxCtas, s);
}

}  // namespace

cudaError_t sj_launch_join(const sj_join_args &a, const sj_grid_dev &g, int fp32, int queue, uint32_t nBig,
                           uint32_t nSmall, int numSM, int maxCtasPerSM, cudaStream_t s)
{
    switch (g.Dp) {
    case 1: return launch_dp<1>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 2: return launch_dp<2>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 3: return launch_dp<3>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 4: return launch_dp<4>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 6: return launch_dp<6>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 8: return launch_dp<8>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 12: return launch_dp<12>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    case 16: return launch_dp<16>(a, g, fp32, queue, nBig, nSmall, numSM, maxCtasPerSM, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t sj_launch_task_sample(const sj_taskgen &g, const sj_grid_dev &gd, const double *xs, const sj_task *tasks,
                                  uint32_t nt, float2 *sample, cudaStream_t s)
{
    if (nt == 0) return cudaSuccess;
    const unsigned grid = (nt + TASK_SAMPLE_WARPS - 1) / TASK_SAMPLE_WARPS;
    constexpr unsigned B = 32 * TASK_SAMPLE_WARPS;
    const float T = std::min((float)gd.thresh, FLT_MAX);   // (a lane without a query is infinitely far)
    switch (gd.Dp) {
    case 1: k_task_sample<1><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 2: k_task_sample<2><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 3: k_task_sample<3><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 4: k_task_sample<4><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 6: k_task_sample<6><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 8: k_task_sample<8><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 12: k_task_sample<12><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    case 16: k_task_sample<16><<<grid, B, 0, s>>>(g, xs, T, tasks, nt, sample); break;
    default: return cudaErrorInvalidValue;
    }
    sj_note_launch();
    return cudaGetLastError();
}
