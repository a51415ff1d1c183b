// The emission pass: the (key, value) pairs of a batch from the count pass's
// hit masks, with the pairs' set hash.
//
// The count pass (sj_join.cu) leaves, per task of the batch:
//   * live bits per (block of 32 stream positions, group of 32 queries): whether
//     the tile has any hit; only live tiles have hit words;
//   * row words [block][query] (bit = stream position of the block) and, for a
//     symmetric task, column words [block][group][position] (bit = query of the
//     group);
//   * per query the offset of the task's row run inside the query's key run,
//     and per stream position the candidate's point id and the offset of its
//     column run inside the candidate's key run.  Both offsets are the key's
//     count just before the count pass added that run, so the runs of one key
//     tile the key's range exactly.
// With keyStart (the exclusive scan of the per-key counts) every pair's slot
// is keyStart[key] + run offset + rank inside the run: no atomics, and keys
// come out ascending with each key's values contiguous -- the order
// thrust::sort_by_key gives the reference (GPU.cu:2336) -- without a sort.
//
// Work is cut into warp units that warps take from a counter, UN at a time:
//   row unit    (task, group of 32 queries): per 32 blocks, the words of the
//               live blocks; the lines are the queries (key), the values the
//               candidates' ids;
//   column unit (symmetric task, block of 32 positions): the words of the live
//               groups; the lines are the candidates, the values the queries'.
// Both stage up to TW words of every line, and the values they select from, in
// shared memory (asynchronous copies, all in flight together) and go out in one
// of two ways, value, key and hash of every pair in the same pass:
//   windows (many hits): the words of two lines across the lanes; popcounts
//               scanned, the set bits decoded into one list a line in slot order,
//               each list copied out with a uniform key: consecutive entries go
//               to consecutive slots, so the stores are coalesced;
//   lists (few hits, or few words): lane = line; each lane walks its own line's
//               bits into its part of one packed list, which the warp copies out.
//
// Bound: latency and instruction issue together.  In the 6-D capture 69 % of the issue
// slots are used; the largest stall is the wait for a unit's staged words and values
// (long_scoreboard, 3.5 of 10 cycles an issue: a unit stages, waits for all of it, then
// emits), then the fixed-latency chains (2.1).  With the points of a cell in spatial
// order the hits are bunched: on the exponential sets three quarters of the pairs lie
// in tiles more than half full, and 60 % of the live tiles hold a tenth of them.  In a
// full window the copy-out -- two shared loads, two stores and the ~19 integer
// operations of splitmix64 with the key's part taken out -- is most of the
// instructions; in sparse tiles a window's fixed ~100 would be, so those go by lists,
// whose decode is as long as the fullest line.
// Measured (one stream): 6-D, 1e7 points, 3.18e12 pairs 10.2 s, 2.5 TB/s of keys
// and values, where the emission of values (11.4 s) and a second pass that read
// them back, wrote the keys and hashed (6.9 s) took 18.2 s; 2-D, 2M points 34.2 ms.
// Every mask word is checked against its task's sizes before it is decoded (bits
// past the stream end or for queries past the tile, which a consistent count
// pass never sets, are dropped and raise an error flag that the host reports),
// so the decoded entries need no checks.  No distance is evaluated, so the pass
// is the same for both precisions.
#include "sj_internal.h"

#include <atomic>

namespace {

constexpr int EW = 128;             // threads per emission CTA (independent warps)
constexpr int ENW = EW / 32;
constexpr int EMIT_MINB = 7;        // resident CTAs per SM (26 KB of shared memory, 72 registers a thread)
constexpr uint32_t UN = 4;          // consecutive units a warp takes at a time (1 near the end of the batch)
constexpr uint32_t UN_MANY = 8;     // and while more than 32 * UN_MANY units a warp are left: they are tiny
                                    // (16-D clusters, 5M units for 1M pairs: 1.11 ms with 8, 1.28 with 32)
constexpr uint32_t FULL = 0xffffffffu;
constexpr uint32_t TW = 16;         // words per line staged together: windows of two lines
constexpr uint32_t LIM = 31;        // entries a line adds to a list per round: lane l of 32 full lines writes
                                    // entry 31 l + k, (almost) all in different banks
constexpr uint32_t SPARSE = 80;      // hits per staged word (of its 1024 over the lines) below which lists are used
                                    // (20, 40, 80 and 160 within 1 % of each other but 160 on 6-D data: +4 %)
constexpr uint32_t DENSE = 14;      // fullest word of a window above which every bit is tested in turn
static_assert(SJ_CTA * sj_query_slots(1, true) / 32 <= TW, "a task's query groups fit the staged words");

struct __align__(16) LineInfo {
    uint32_t base;          // windows: the line's next slot; lists: slot of list entry 0 if it were this line's
    uint32_t key, hi2, add; // the line's key and its part of the pair hash
};

struct WarpSmem {
    uint32_t tile[TW][33];  // [staged word][line]
    uint32_t val[TW * 32];  // value of bit i of staged word j: val[32 j + i]
    uint16_t ent[1024];     // windows: two lists of up to 512 byte offsets into val; lists: (line << 9) | index
    LineInfo line[32];
};

// asynchronous copy of one word (or a zero when !have; src is not read then)
__device__ __forceinline__ void copy_word(uint32_t *dst, const uint32_t *src, bool have)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(have ? 4 : 0)
                 : "memory");
}

// inclusive scan over groups of W lanes
template <int W>
__device__ __forceinline__ uint32_t incl_scan(uint32_t x, uint32_t lane)
{
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o, W);
        if ((lane & (W - 1)) >= (uint32_t)o) x += y;
    }
    return x;
}

// Index of the highest set bit of m (m != 0).
__device__ __forceinline__ uint32_t top_bit(uint32_t m)
{
    uint32_t b;
    asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(m));
    return b;
}

// The pair hash, splitmix64(key << 32 | value), with the key's part separated:
// both are point ids below 2^31, so adding the increment's low half to the
// value never carries and the high half depends on the key alone.  Written in
// 32-bit halves (18 integer instructions).
struct KeyHash {
    uint32_t hi2, add;   // high word << 2 (xored into the low word); high word's contribution to the first product
};

__device__ __forceinline__ KeyHash key_hash(uint32_t key)
{
    const uint32_t hi = key + 0x9e3779b9u;
    return {hi << 2, (hi ^ (hi >> 30)) * 0x1ce4e5b9u};
}

__device__ __forceinline__ uint64_t pair_hash(KeyHash kh, uint32_t val)
{
    const uint32_t y = val + 0x7f4a7c15u;
    const uint32_t lo = y ^ (y >> 30) ^ kh.hi2;
    const uint64_t z = (uint64_t)lo * 0x1ce4e5b9u;
    uint32_t zl = (uint32_t)z, zh = lo * 0xbf58476du + kh.add + (uint32_t)(z >> 32);
    zl ^= __funnelshift_r(zl, zh, 27);
    zh ^= zh >> 27;
    const uint64_t p = (uint64_t)zl * 0x133111ebu;
    const uint32_t ql = (uint32_t)p;
    const uint32_t qh = zh * 0x133111ebu + (zl * 0x94d049bbu + (uint32_t)(p >> 32));
    return ((uint64_t)(qh ^ (qh >> 31)) << 32) | (ql ^ __funnelshift_r(ql, qh, 31));
}

// Output of one warp: the arrays, and the hash of the pairs written so far.
struct Out {
    int32_t *__restrict__ key;
    int32_t *__restrict__ val;
    uint64_t cap;
    unsigned long long hash;
};

// Writes tag + 4 * (index of each set bit of m) to the list from entry k on,
// lowest bit first; n = popc(m).  sparse: the bits highest first, two a step,
// filling from the end.  dense: all 32 bits tested, no bit scans and no loop.
__device__ __forceinline__ void decode_sparse(uint32_t m, uint32_t n, uint32_t tag, uint16_t *buf, uint32_t k)
{
    uint16_t *p = buf + k + n;
    for (; n >= 2; n -= 2) {
        const uint32_t b0 = top_bit(m);
        m ^= 1u << b0;
        const uint32_t b1 = top_bit(m);
        m ^= 1u << b1;
        p[-1] = (uint16_t)(tag + 4 * b0);
        p[-2] = (uint16_t)(tag + 4 * b1);
        p -= 2;
    }
    if (n) p[-1] = (uint16_t)(tag + 4 * top_bit(m));
}

__device__ __forceinline__ void decode_dense(uint32_t m, uint32_t n, uint32_t tag, uint32_t j, uint16_t *buf, uint32_t k)
{
    // The lanes start at different bits (2 j for word j of the line) and wrap
    // around: full words begin 64 bytes apart in the list, and lanes walking them
    // in step would all hit two banks.
    const uint32_t r = 2 * j;
    uint32_t p = (uint32_t)__cvta_generic_to_shared(buf + k) + 2 * __popc(m & ((1u << r) - 1u));
    uint32_t t = tag + 4 * r;
    m = __funnelshift_r(m, m, r);
    const uint32_t back = 2 * n;
#pragma unroll
    for (int b = 0; b < 32; b++) {
        if (b > 0 && b % 2 == 0)
            asm volatile("{ .reg .pred q; setp.eq.u32 q, %2, %4;\n\t"
                         "@q sub.u32 %0, %0, %3;\n\t"
                         "@q sub.u32 %1, %1, 128; }"
                         : "+r"(p), "+r"(t)
                         : "r"(r), "r"(back), "r"(32 - b));
        asm volatile("{ .reg .pred q; .reg .b32 t;\n\t"
                     "and.b32 t, %1, %3; setp.ne.u32 q, t, 0;\n\t"
                     "@q st.shared.u16 [%0], %2;\n\t"
                     "@q add.u32 %0, %0, 2; }"
                     : "+r"(p)
                     : "r"(m), "r"(t), "r"(1u << b)
                     : "memory");
        t += 4;
    }
}

// Copies the list's entries [e0, e0 + n) of one line (byte offsets into w.val) to
// slots B, B + 1 ..
template <bool KEYS>
__device__ __forceinline__ void copy_line(Out &o, const WarpSmem &w, uint32_t lane, uint32_t e0, uint32_t n,
                                          const LineInfo &li)
{
    const uint32_t B = li.base, key = li.key;
    const KeyHash kh{li.hi2, li.add};
    uint32_t ent = (uint32_t)__cvta_generic_to_shared(w.ent + e0 + lane);
    const uint32_t val = (uint32_t)__cvta_generic_to_shared(w.val);
    int32_t *pv = o.val + (uint64_t)B + lane;
    int32_t *pk = KEYS ? o.key + (uint64_t)B + lane : nullptr;
#pragma unroll 1
    for (; n >= 128; n -= 128) {
        uint32_t at[4], v[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(at[i]) : "r"(ent + 64 * i));
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[i]) : "r"(val + at[i]));
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            pv[32 * i] = (int32_t)v[i];
            if (KEYS) pk[32 * i] = (int32_t)key;
            o.hash += pair_hash(kh, v[i]);
        }
        ent += 256;
        pv += 128;
        if (KEYS) pk += 128;
    }
#pragma unroll 1
    for (uint32_t e = lane; e < n; e += 32) {
        uint32_t at, v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(at) : "r"(ent));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(val + at));
        *pv = (int32_t)v;
        if (KEYS) *pk = (int32_t)key;
        o.hash += pair_hash(kh, v);
        ent += 64;
        pv += 32;
        if (KEYS) pk += 32;
    }
}

// Emits the hits of 32 lines over the nl staged words: a window holds 2 lines of
// up to 16 words, 4 of up to 8, 8 of up to 4 or 16 of up to 2; lines: mask of the
// lines with hits.  w.line holds the lines.
template <bool KEYS>
__device__ __forceinline__ void emit_windows(Out &o, WarpSmem &w, uint32_t lane, uint32_t nl, uint32_t lines)
{
    const uint32_t sh = nl > 2 ? 32 - __clz(nl - 1) : 1u;   // words per line: 2^sh
    const uint32_t W = 1u << sh, j = lane & (W - 1), lw = lane >> sh, lpw = 32u >> sh;
    const uint32_t inWindow = (1u << lpw) - 1u;             // at most 16 lines
#pragma unroll 1
    for (uint32_t l0 = 0; l0 < 32; l0 += lpw) {
        if (!((lines >> l0) & inWindow)) continue;
        const uint32_t word = j < nl ? w.tile[j][l0 + lw] : 0u;
        const uint32_t cnt = __popc(word);
        uint32_t incl = cnt;   // over the line's words
#pragma unroll 1
        for (uint32_t d = 1; d < W; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, d, W);
            if (j >= d) incl += y;
        }
        const bool dense = __any_sync(FULL, cnt > DENSE);
        const uint32_t at = lw * (W * 32) + incl - cnt;   // a list of W * 32 entries per line
        __syncwarp();   // the previous window's copy-out is done with the lists
        if (dense) decode_dense(word, cnt, j * 128, j, w.ent, at);
        else decode_sparse(word, cnt, j * 128, w.ent, at);
        __syncwarp();
#pragma unroll 1
        for (uint32_t i = 0; i < lpw; i++) {
            const uint32_t n = __shfl_sync(FULL, incl, W * i + W - 1);
            if (n) copy_line<KEYS>(o, w, lane, i * (W * 32), n, w.line[l0 + i]);
        }
    }
}

// Emits the hits of 32 lines, lane = line: cnt of them in the nonzero words nz,
// slots up to `end`.
template <bool KEYS>
__device__ __forceinline__ void emit_lists(Out &o, WarpSmem &w, uint32_t lane, uint32_t cnt, uint32_t nz,
                                           uint32_t end)
{
    uint32_t rem = cnt, word = 0, tag = 0;   // lines go from their last hit to the first
#pragma unroll 1
    while (__any_sync(FULL, rem)) {
        const uint32_t c = min(rem, LIM);
        const uint32_t incl = incl_scan<32>(c, lane);
        const uint32_t T = __shfl_sync(FULL, incl, 31);
        end -= c;
        rem -= c;
        w.line[lane].base = end - (incl - c);
        uint16_t *p = w.ent + incl;
#pragma unroll 1
        for (uint32_t k = c; k; k--) {
            if (!word) {
                const uint32_t j = top_bit(nz);
                nz ^= 1u << j;
                word = w.tile[j][lane];
                tag = (lane << 9) | (j << 5);
            }
            const uint32_t b = top_bit(word);
            word ^= 1u << b;
            *--p = (uint16_t)(tag + b);
        }
        __syncwarp();
#pragma unroll 2
        for (uint32_t e = lane; e < T; e += 32) {
            const uint32_t en = w.ent[e];
            const LineInfo l = w.line[en >> 9];
            const uint32_t v = w.val[en & 0x1ffu];
            o.val[l.base + e] = (int32_t)v;
            if (KEYS) o.key[l.base + e] = (int32_t)l.key;
            o.hash += pair_hash(KeyHash{l.hi2, l.add}, v);
        }
        __syncwarp();   // the list is read before the next round overwrites it
    }
}

// Unit k of task t: query group k (rows), or for k >= nG block k - nG of 32
// positions of a symmetric task (columns).  Both are the same loop over live
// words: word x of the unit is words[x * stride + lane] for line = lane and its
// bit i selects value vals[32 x + i] of nv values.  (One code path, so that the
// kernel stays inside the instruction caches with every warp at another place:
// with rows and columns inlined apart the warps waited for instructions for 11 of
// 19 cycles an issue.)
template <bool KEYS>
__device__ __forceinline__ void emit_unit(const sj_join_args &a, Out &o, uint32_t t, uint32_t k, WarpSmem &w,
                                          uint32_t lane)
{
    const sj_task *const tp = a.tasks + t;
    const uint32_t qBegin = tp->qBegin, qc = tp->qCount, L = tp->sEnd - tp->sBegin;
    const uint32_t nBlk = (L + 31) / 32, nG = (qc + 31) / 32;
    const uint32_t *const live = a.masks + (a.maskOff[t] - a.maskOff[a.taskBegin]);
    const uint64_t rec = a.candOff[t] - a.candOff[a.taskBegin];
    const bool row = k < nG;
    const uint32_t *words, *vals;
    uint32_t stride, nv, nLine, nLive;   // nLive: words of live bits
    uint32_t key = 0, next = 0, colLive = 0;
    if (row) {
        nLine = min(32u, qc - 32 * k);
        words = live + sj_live_words(nBlk, nG) + 32 * k;
        stride = qc;
        vals = a.candId + rec;
        nv = L;
        nLive = (nBlk + 31) / 32;
        if (lane < nLine) {
            key = a.ids[qBegin + 32 * k + lane];
            next = a.keyStart[key] + a.rowRel[a.rowOff[t] - a.rowOff[a.taskBegin] + 32 * k + lane];
        }
    } else {
        const uint32_t b = k - nG;
        // the live bits of a block lie in one word per group (at most TW groups)
        const bool lv = lane < nG && ((__ldg(live + (b >> 5) * nG + lane) >> (b & 31)) & 1u);
        colLive = __ballot_sync(FULL, lv);
        if (!colLive) return;
        nLine = min(32u, L - 32 * b);
        words = a.colMasks + (a.colOff[t] - a.colOff[a.taskBegin]) + (uint64_t)b * nG * 32;
        stride = 32;
        vals = a.ids + qBegin;
        nv = qc;
        nLive = 1;
        if (lane < nLine) {
            key = a.candId[rec + 32 * b + lane];
            next = a.keyStart[key] + a.candRel[rec + 32 * b + lane];
        }
    }
    __syncwarp();   // the previous unit is done with the lines
    {
        const KeyHash kh = key_hash(key);
        w.line[lane] = LineInfo{next, key, kh.hi2, kh.add};
    }
    uint32_t c0 = 0, myLive = 0, chunks = 0, x0 = 0, m = 0;
    bool more = true;
#pragma unroll 1
    do {
        // ---- stage the next live words, up to TW of them
        uint32_t nl = 0, cut = 32;   // cut: values of the last word (32: all)
#pragma unroll 1
        while (nl < TW) {
            if (!m) {
                if (!chunks) {
                    if (c0 >= nLive) {
                        more = false;
                        break;
                    }
                    myLive = row ? (c0 + lane < nLive ? __ldg(live + (uint64_t)(c0 + lane) * nG + k) : 0u)
                                 : (lane == 0 ? colLive : 0u);
                    chunks = __ballot_sync(FULL, myLive);
                    c0 += 32;
                    continue;
                }
                const uint32_t ci = __ffs(chunks) - 1;
                chunks &= chunks - 1;
                m = __shfl_sync(FULL, myLive, ci);
                x0 = (c0 - 32 + ci) * 32;
            }
            const uint32_t x = x0 + __ffs(m) - 1;
            m &= m - 1;
            const uint32_t rem = 32 * x < nv ? nv - 32 * x : 0u;   // values from the word's first on
            copy_word(&w.tile[nl][lane], words + (uint64_t)x * stride + lane, lane < nLine && rem);
            copy_word(&w.val[nl * 32 + lane], vals + 32 * x + lane, lane < rem);
            if (rem < 32u) cut = rem;   // the stream's or the tile's last word
            nl++;
        }
        if (!nl) break;
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (cut < 32u) {   // this lane's own copy: the last word staged
            const uint32_t v = w.tile[nl - 1][lane];
            if (v >> cut) {   // bits past the stream end or the tile
                atomicMax(&a.stat[6], 1ULL);
                w.tile[nl - 1][lane] = v & ((1u << cut) - 1u);
            }
        }
        uint32_t cnt = 0, nz = 0;   // lane = line
#pragma unroll 4
        for (uint32_t j = 0; j < nl; j++) {
            const uint32_t v = w.tile[j][lane];
            cnt += __popc(v);
            if (v) nz |= 1u << j;
        }
        if (__any_sync(FULL, cnt && (uint64_t)next + cnt > o.cap)) {   // a consistent count pass never gets here
            atomicMax(&a.stat[3], 1ULL);
        } else if (nl > 2 && __reduce_add_sync(FULL, cnt) >= SPARSE * nl) {
            w.line[lane].base = next;
            __syncwarp();
            emit_windows<KEYS>(o, w, lane, nl, __ballot_sync(FULL, cnt));
        } else {
            __syncwarp();
            emit_lists<KEYS>(o, w, lane, cnt, nz, next + cnt);
        }
        next += cnt;
        __syncwarp();   // the words and lists are free again
    } while (more);
}

template <bool KEYS>
__global__ void __launch_bounds__(EW, EMIT_MINB) k_emit(sj_join_args a)
{
    __shared__ WarpSmem smem[ENW];
    const uint32_t lane = threadIdx.x & 31u;
    WarpSmem &w = smem[threadIdx.x >> 5];
    // a batch whose count exceeded the output buffer is re-planned by the host
    if (a.batchPairs && *a.batchPairs > a.capacity) {
        if (threadIdx.x == 0 && blockIdx.x == 0) atomicMax(&a.stat[5], 1ULL);
        return;
    }
    const uint64_t u0 = a.unitOff[a.taskBegin];
    const uint32_t nUnits = (uint32_t)(a.unitOff[a.taskEnd] - u0);
    Out o{a.outKey, a.outVal, a.capacity, 0ULL};
    const uint32_t manyUnits = 32 * UN_MANY * gridDim.x * ENW;
    const uint32_t endGame = 8 * UN * gridDim.x * ENW;   // units left below which warps take them one by one
    uint32_t take = nUnits > manyUnits ? UN_MANY : nUnits > endGame ? UN : 1u;
    for (;;) {
        // (units are not taken ahead of their turn: a warp that holds one while it
        // is busy with another costs more at the end than the counter's latency)
        uint32_t un = 0;
        if (lane == 0) un = atomicAdd(a.queueHead, take);
        un = __shfl_sync(FULL, un, 0);
        if (un >= nUnits) break;
        const uint32_t unEnd = nUnits - un < take ? nUnits : un + take;
        if (nUnits - un < manyUnits) take = nUnits - un < endGame ? 1u : UN;
        // the first unit's task: the last t with unitOff[t] - u0 <= un, 32 probes a step
        uint32_t lo = a.taskBegin, hi = a.taskEnd;
        while (hi - lo > 1) {
            const uint32_t step = (hi - lo + 31) / 32;
            const uint32_t probe = lo + (lane + 1) * step;
            const bool below = probe < hi && a.unitOff[probe] - u0 <= un;   // a prefix of the lanes
            lo += __popc(__ballot_sync(FULL, below)) * step;
            hi = min(hi, lo + step);
        }
        uint32_t tBeg = (uint32_t)(a.unitOff[lo] - u0), tEnd = (uint32_t)(a.unitOff[lo + 1] - u0);
        for (; un < unEnd; un++) {
            while (un >= tEnd) {   // the next task (every task has a unit)
                lo++;
                tBeg = tEnd;
                tEnd = (uint32_t)(a.unitOff[lo + 1] - u0);
            }
            if (a.taskHits && a.taskHits[lo] == 0) {   // the count pass found no pair in this task
                un = tEnd - 1;
                continue;
            }
            const uint32_t k = un - tBeg;
            if (k && a.tasks[lo].qCount <= 32) {
                // column units of one query group: on to the next live block (sparse
                // tasks, most of whose units are dead: 16-D clusters 1.49 to 1.11 ms)
                const uint32_t b = k - 1;
                const uint32_t w32 = a.masks[a.maskOff[lo] - a.maskOff[a.taskBegin] + (b >> 5)] >> (b & 31);
                if (!(w32 & 1u)) {
                    un = min(un + (w32 ? __ffs(w32) - 1 : 32 - (b & 31)), tEnd) - 1;
                    continue;
                }
            }
            emit_unit<KEYS>(a, o, lo, un - tBeg, w, lane);
        }
    }
    unsigned long long h = o.hash;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) h += __shfl_xor_sync(FULL, h, d);
    if (lane == 0 && h) atomicAdd(&a.stat[4], h);
}

template <bool KEYS>
int emit_occupancy()
{
    constexpr int MAXDEV = 64;
    static std::atomic<int> occ[MAXDEV];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= MAXDEV) dev = 0;
    int o = occ[dev].load();
    if (o == 0) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_emit<KEYS>, EW, 0);
        o = b > 0 ? b : 1;
        occ[dev].store(o);
    }
    return o;
}

template <bool KEYS>
cudaError_t launch(const sj_join_args &a, int numSM, int maxCtasPerSM, cudaStream_t s)
{
    int perSM = emit_occupancy<KEYS>();
    if (maxCtasPerSM > 0 && maxCtasPerSM < perSM) perSM = maxCtasPerSM;
    k_emit<KEYS><<<(unsigned)(numSM * perSM), EW, 0, s>>>(a);
    sj_note_launch();
    return cudaGetLastError();
}

}  // namespace

cudaError_t sj_launch_emit(const sj_join_args &a, int keys, int numSM, int maxCtasPerSM, cudaStream_t s)
{
    if (a.taskEnd == a.taskBegin) return cudaSuccess;
    return keys ? launch<true>(a, numSM, maxCtasPerSM, s) : launch<false>(a, numSM, maxCtasPerSM, s);
}
