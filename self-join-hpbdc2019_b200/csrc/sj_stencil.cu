// Owned neighbour-cell lists and per-cell estimator features.
//
// The reference enumerates the clamped 3^k stencil per query POINT with a
// binary search per neighbour (kernel.cu:1455-1534, 387-396).  Here the
// stencil is enumerated once per non-empty CELL, by one warp, over the
// linear-id ordering (dim k-1 most significant): each level narrows the range
// of the sorted id array to the cells sharing a coordinate prefix, so empty
// sub-stencils drop out early (sparse high-dimensional grids).  The levels are
// walked breadth first: eight prefixes at a time, four lanes each, the four
// lanes searching the four bounds of the prefix's three children; the children
// that hold cells are compacted, in id order, into the next level's list.  The
// last dimension takes a lane a prefix: its up to three cells follow one another
// in the id array, so one search finds them.  A walk whose lowest TREE_DIMS dimensions are reached depth first (k > TREE_DIMS)
// keeps the lists at 3^(TREE_DIMS-1) entries.
// Bound: latency of the dependent searches (about 60 steps a cell at k = 6, which
// the lanes of a warp take side by side).  One thread a cell, depth first with
// six searches a prefix and its stack in local memory, took 10.3 ms a pass on
// 466,982 cells at k = 6 (1M points, 16-D); this form's figures stand at
// k_neighbours.
//
// Ownership rules decide which cell of an adjacent pair evaluates it:
//   FULL      every neighbour (mode 3/7/9 semantics; one direction emitted)
//   LID       neighbours with a larger linear id (kernel.cu:1529-1534)
//   UNICOMP   the highest differing dimension's coordinate of the owner is odd
//             (stamploops.h)
//   BUNICOMP  checkerboard colour rules for k = 2, 3 (kernel.cu:1346-1392)
// Each rule assigns every adjacent pair to exactly one owner.
#include "sj_internal.h"

namespace {

__device__ __forceinline__ uint32_t lower_bound_u64(const uint64_t *__restrict__ a, uint32_t lo, uint32_t hi,
                                                    unsigned long long key)
{
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Offsets of a neighbour, two bits per dimension: 0, 1, 2 for -1, 0, +1.
constexpr uint32_t CODE_HOME = 0x55555555u;   // every dimension 1

// a: lane j holds the cell's coordinate of dimension j; odd: bit j set when it is odd
__device__ __forceinline__ bool owns(int pattern, int k, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t odd,
                                     uint32_t code, uint32_t c, uint32_t b)
{
    switch (pattern) {
    case SJ_PAT_FULL:
        return true;
    case SJ_PAT_LID:
        return b > c;   // cells are sorted by linear id
    case SJ_PAT_UNICOMP: {
        const uint32_t diff = code ^ CODE_HOME;   // not home: some dimension differs
        const int d = diff ? (31 - __clz(diff)) >> 1 : 0;
        return (odd >> d) & 1u;
    }
    case SJ_PAT_BUNICOMP: {
        const uint32_t v0 = a0 + (code & 3u) - 1u, v1 = a1 + ((code >> 2) & 3u) - 1u;
        if (k == 2) {
            if (((a0 + a1) & 1u) != 0) return (a1 <= v1) && (a0 != v0);
            return (a1 < v1) || (v1 < a1 && v0 == a0);
        } else {
            const uint32_t v2 = a2 + ((code >> 4) & 3u) - 1u;
            if (((a0 + a1 + a2) & 1u) != 0)
                return (a0 != v0 && a1 <= v1 && a2 <= v2) || (a0 == v0 && a1 <= v1 && a2 < v2) ||
                       (a1 < v1 && v2 < a2);
            return (a1 < v1 && a2 <= v2) || (a0 == v0 && v1 < a1 && a2 <= v2) ||
                   (a0 != v0 && a1 < v1 && v2 < a2) || (a1 == v1 && a2 < v2);
        }
    }
    }
    return false;
}

constexpr int TREE_DIMS = 6;                 // dimensions walked breadth first at most
constexpr int NBR_THREADS = 128;

constexpr int pow3(int e) { return e <= 0 ? 1 : 3 * pow3(e - 1); }

// Prefixes of one level: their cells [lo, hi), the linear id of the first place,
// the offsets.
template <int N>
struct TreeList {
    uint32_t lo[N], hi[N], code[N];
    unsigned long long base[N];
};

struct TreeRef {
    uint32_t *lo, *hi, *code;
    unsigned long long *base;
};

template <int N>
__device__ __forceinline__ TreeRef ref(TreeList<N> &l)
{
    return {l.lo, l.hi, l.code, l.base};
}

// Two lists in turn: the last level's prefixes (3^(DIMS-1)) and the one's before.
template <int DIMS>
struct NbrSmem {
    TreeList<pow3(DIMS - 1)> last;
    TreeList<pow3(DIMS - 2)> before;
    uint32_t hist[8];
};

// pass 0: count owned neighbours (out = counts), full-stencil candidates and
//         features; pass 1: write owned neighbour cell indices (out = list).
// Measured (both passes, one B200): 466,982 cells at k = 6 20.3 ms depth first,
// 6.93 breadth first with four lanes a prefix at the leaves too, 5.88 with one;
// 5,583 and 6,980 cells at k = 6 3.7 to 0.1 ms; 125k cells at k = 3 0.27 to 0.17 ms
// with one lane a prefix at the leaves.
// GROUP lanes a cell: 32, or 8 where the tree has at most 27 leaves (two prefixes
// at a time; a warp then has four cells).
template <int DIMS, int GROUP>
__global__ void __launch_bounds__(NBR_THREADS) k_neighbours(
    const uint64_t *__restrict__ cellLid, const uint32_t *__restrict__ cellCoord,
    const uint32_t *__restrict__ cellStart, uint32_t nCells, sj_grid_dev g, int pattern,
    const uint32_t *__restrict__ nbrStart, uint32_t *__restrict__ out, uint64_t *__restrict__ candFull,
    unsigned long long *__restrict__ candTotal, float *__restrict__ feat, int pass)
{
    constexpr int CELLS = NBR_THREADS / GROUP;
    __shared__ NbrSmem<DIMS> smem[CELLS];
    const uint32_t lane = threadIdx.x & (GROUP - 1);   // of the group
    const uint32_t shift = threadIdx.x & 31u & ~(uint32_t)(GROUP - 1);
    const uint32_t FULL = (GROUP == 32 ? 0xffffffffu : (1u << (GROUP & 31)) - 1u) << shift;   // the group's lanes
    NbrSmem<DIMS> &sm = smem[threadIdx.x / GROUP];
    const uint32_t c = blockIdx.x * CELLS + threadIdx.x / GROUP;
    if (c >= nCells) return;
    const auto ballot = [&](bool v) { return __ballot_sync(FULL, v) >> shift; };
    const auto shfl = [&](uint32_t v, int src) { return __shfl_sync(FULL, v, src, GROUP); };
    const int k = g.k;
    const uint32_t aj = (int)lane < k ? cellCoord[(uint64_t)c * k + lane] : 0u;   // lane j: coordinate j
    const uint32_t odd = ballot(aj & 1u);
    const uint32_t a0 = shfl(aj, 0), a1 = shfl(aj, 1), a2 = shfl(aj, 2);
    const uint32_t myOcc = cellStart[c + 1] - cellStart[c];
    const uint32_t ltmask = (1u << lane) - 1u;
    const uint32_t highHome = k < 16 ? CODE_HOME << (2 * k) : 0u;   // dimensions at or above k are unchanged
    // bound q of the children of a prefix in dimension j: the first of its cells
    // [lo, hi) at or after coordinate a_j - 1 + q (q = lane & 3)
    const uint32_t q = lane & 3u;
    auto bound = [&](int j, uint32_t a, unsigned long long base, uint32_t lo, uint32_t hi) -> uint32_t {
        if (q == 0 && a == 0) return lo;   // no coordinate below 0
        return lower_bound_u64(cellLid, lo, hi, base + ((unsigned long long)a + q - 1ULL) * g.mult[j]);
    };

    uint32_t owned = 0, writePos = pass == 1 ? nbrStart[c] : 0u;
    unsigned long long stencilOcc = 0;            // this lane's part
    float ownW = 0.0f, ownW1 = 0.0f, ownW2 = 0.0f;   // (as feat's f9, f13, f14; this lane's part)
    if (feat && lane < 8) sm.hist[lane] = 0;

    // prefixes of the dimensions above the tree, depth first (k > TREE_DIMS)
    uint32_t dLo[SJ_MAX_K - TREE_DIMS + 1], dHi[SJ_MAX_K - TREE_DIMS + 1], dCode = 0;
    unsigned long long dBase[SJ_MAX_K - TREE_DIMS + 1];
    int t[SJ_MAX_K - TREE_DIMS + 1];
    const int top = k > TREE_DIMS ? k - TREE_DIMS : 0;   // depth of the depth-first part
    // the owned neighbours of the linear-id pattern come after the cell itself
    dLo[0] = (pass == 1 && pattern == SJ_PAT_LID) ? c + 1 : 0u;
    dHi[0] = nCells;
    dBase[0] = 0;
    t[0] = 0;
    int depth = 0;
    for (;;) {
        if (depth < top) {
            // the next child of the prefix at this depth
            const int j = k - 1 - depth;
            if (t[depth] == 3) {
                if (depth == 0) break;
                depth--;
                t[depth]++;
                continue;
            }
            const uint32_t a = shfl(aj, j);
            const long long v = (long long)a + t[depth] - 1;
            uint32_t l = 0, h = 0;
            unsigned long long id = 0;
            if (v >= 0 && v < (long long)g.nCells[j]) {
                id = dBase[depth] + (unsigned long long)v * g.mult[j];
                l = lower_bound_u64(cellLid, dLo[depth], dHi[depth], id);
                h = lower_bound_u64(cellLid, l, dHi[depth], id + g.mult[j]);
            }
            if (l >= h) {
                t[depth]++;
                continue;
            }
            dCode = (dCode & ~(3u << (2 * j))) | ((uint32_t)t[depth] << (2 * j));
            dLo[depth + 1] = l;
            dHi[depth + 1] = h;
            dBase[depth + 1] = id;
            depth++;
            t[depth] = 0;
            continue;
        }
        // ---- the tree below the prefix, breadth first
        uint32_t n = 1;
        // dimension j reads `last` when j is even: dimension 0 has the longest list
        const bool topEven = ((k - 1 - depth) & 1) == 0;
        TreeRef L = topEven ? ref(sm.last) : ref(sm.before), N = topEven ? ref(sm.before) : ref(sm.last);
        __syncwarp(FULL);
        if (lane == 0) {
            L.lo[0] = dLo[depth];
            L.hi[0] = dHi[depth];
            L.base[0] = dBase[depth];
            L.code[0] = dCode;
        }
        __syncwarp(FULL);
        for (int j = k - 1 - depth; j > 0 && n; j--) {
            const uint32_t a = shfl(aj, j);
            uint32_t made = 0;
            for (uint32_t i0 = 0; i0 < n; i0 += GROUP / 4) {
                const uint32_t i = i0 + (lane >> 2);
                uint32_t r = 0, code = 0;
                unsigned long long base = 0;
                if (i < n) {
                    base = L.base[i];
                    code = L.code[i];
                    r = bound(j, a, base, L.lo[i], L.hi[i]);
                }
                const uint32_t end = __shfl_down_sync(FULL, r, 1, GROUP);
                const bool have = i < n && q < 3 && r < end && !(q == 0 && a == 0) && a + q - 1u < g.nCells[j];
                const uint32_t m = ballot(have);
                code |= q << (2 * j);
                if (have) {
                    const uint32_t at = made + __popc(m & ltmask);
                    N.lo[at] = r;
                    N.hi[at] = end;
                    N.base[at] = base + ((unsigned long long)a + q - 1ULL) * g.mult[j];
                    N.code[at] = code;
                }
                made += __popc(m);
            }
            __syncwarp(FULL);
            n = made;
            const TreeRef x = L;
            L = N;
            N = x;
        }
        // ---- leaves, a lane a prefix: its cells with coordinate a0 - 1 to a0 + 1 in
        // dimension 0 follow one another in the id array (mult[0] == 1), so one
        // search finds them all
        for (uint32_t i0 = 0; i0 < n; i0 += GROUP) {
            const uint32_t i = i0 + lane;
            uint32_t r0 = 0, ownBits = 0;
            if (i < n) {
                const unsigned long long base = L.base[i];
                const uint32_t hi = L.hi[i], prefix = L.code[i] | highHome;
                r0 = lower_bound_u64(cellLid, L.lo[i], hi, base + (a0 ? a0 - 1u : 0u));
#pragma unroll
                for (uint32_t e = 0; e < 3; e++) {
                    const uint32_t r = r0 + e;
                    if (r >= hi) break;
                    const unsigned long long off = cellLid[r] - base;   // the cell's coordinate
                    if (off > (unsigned long long)a0 + 1ULL) break;
                    const uint32_t full = prefix | ((uint32_t)off + 1u - a0);
                    const bool home = r == c;
                    const bool own = !home && owns(pattern, k, a0, a1, a2, odd, full, c, r);
                    if (own) ownBits |= 1u << e;
                    if (pass == 0) {
                        const uint32_t occ = cellStart[r + 1] - cellStart[r];
                        stencilOcc += occ;
                        if (feat && !home) {
                            const int bin = 31 - __clz(occ);
                            atomicAdd(&sm.hist[bin > 7 ? 7 : bin], 1u);
                            if (own) {
                                const uint32_t diff = full ^ CODE_HOME;
                                const int w = __popc((diff | (diff >> 1)) & CODE_HOME);   // dimensions that differ
                                const float wo = (float)occ * g.offW[w];
                                ownW += wo;
                                if (w == 1) ownW1 += wo;
                                else if (w == 2) ownW2 += wo;
                            }
                        }
                    }
                }
            }
            const uint32_t cnt = __popc(ownBits);
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < GROUP; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, incl, o, GROUP);
                if (lane >= (uint32_t)o) incl += y;
            }
            if (pass == 1) {
                uint32_t at = writePos + owned + incl - cnt;
#pragma unroll
                for (uint32_t e = 0; e < 3; e++)
                    if ((ownBits >> e) & 1u) out[at++] = r0 + e;
            }
            owned += shfl(incl, GROUP - 1);
        }
        __syncwarp(FULL);
        if (depth == 0) break;
        depth--;
        t[depth]++;
    }
    if (pass != 0) return;
#pragma unroll
    for (int o = GROUP / 2; o > 0; o >>= 1) {
        stencilOcc += __shfl_xor_sync(FULL, stencilOcc, o);
        ownW += __shfl_xor_sync(FULL, ownW, o);
        ownW1 += __shfl_xor_sync(FULL, ownW1, o);
        ownW2 += __shfl_xor_sync(FULL, ownW2, o);
    }
    __syncwarp(FULL);
    if (lane == 0) {
        out[c] = owned;
        candFull[c] = stencilOcc * (unsigned long long)myOcc;
        if (candTotal) atomicAdd(candTotal, stencilOcc * (unsigned long long)myOcc);
    }
    for (uint32_t e = lane; feat && e < SJ_NFEAT; e += GROUP) {
        float nst = 1.0f;
        for (int d = 0; d < k; d++) nst *= 3.0f;
        nst -= 1.0f;
        // occupancy, neighbour-occupancy histogram, eps / cell width,
        // dimension; f9, f13, f14: the expected hits with the owned
        // neighbours (all offset classes, face neighbours, edge neighbours)
        // under a locally uniform density, log2(1 + occupancy x weighted sum)
        const float o = (float)myOcc;
        float f;
        if (e == 0) f = log2f(1.0f + o);
        else if (e < 9) f = (float)sm.hist[e - 1] / nst;
        else if (e == 9) f = log2f(1.0f + o * ownW);
        else if (e == 10) f = log2f(1.0f + (float)stencilOcc);
        else if (e == 11) f = 1.0f;                          // eps / cell width (cells are eps wide)
        else if (e == 12) f = (float)g.D / 16.0f;
        else if (e == 13) f = log2f(1.0f + o * ownW1);
        else if (e == 14) f = log2f(1.0f + o * ownW2);
        else f = log2f((float)g.eps) / 8.0f;
        feat[(uint64_t)c * SJ_NFEAT + e] = f;
    }
}

}  // namespace

cudaError_t sj_launch_neighbours(const uint64_t *cellLid, const uint32_t *cellCoord, const uint32_t *cellStart,
                                 uint32_t nCells, sj_grid_dev g, int pattern, const uint32_t *nbrStart,
                                 uint32_t *nbrCountOrCell, uint64_t *candFull, unsigned long long *candTotal,
                                 float *feat, int pass, cudaStream_t s)
{
    if (nCells == 0) return cudaSuccess;
    const auto go = [&](auto kernel, unsigned group) {
        const unsigned cells = NBR_THREADS / group;
        kernel<<<(nCells + cells - 1) / cells, NBR_THREADS, 0, s>>>(cellLid, cellCoord, cellStart, nCells, g, pattern,
                                                                   nbrStart, nbrCountOrCell, candFull, candTotal,
                                                                   feat, pass);
    };
    // the lists hold 3^(dimensions - 1) prefixes: small ones leave room for more warps
    switch (g.k < TREE_DIMS ? g.k : TREE_DIMS) {
    case 1:
    case 2: go(k_neighbours<2, 8>, 8); break;
    case 3: go(k_neighbours<3, 8>, 8); break;
    case 4: go(k_neighbours<4, 32>, 32); break;
    case 5: go(k_neighbours<5, 32>, 32); break;
    default: go(k_neighbours<TREE_DIMS, 32>, 32); break;
    }
    sj_note_launch();
    return cudaGetLastError();
}
