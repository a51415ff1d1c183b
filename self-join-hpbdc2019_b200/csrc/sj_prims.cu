// Device primitives: exclusive scan (u32), stable LSD radix sort, CSR append.
#include <atomic>

#include "sj_internal.h"

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;   // 2048 elements per block

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t warpSums[SCAN_THREADS / 32];
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane_id() >= (uint32_t)o) x += y;
    }
    const int w = threadIdx.x >> 5;
    if (lane_id() == 31) warpSums[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t s = (lane_id() < SCAN_THREADS / 32) ? warpSums[lane_id()] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane_id() >= (uint32_t)o) s += y;
        }
        if (lane_id() < SCAN_THREADS / 32) warpSums[lane_id()] = s;   // inclusive warp prefixes
    }
    __syncthreads();
    uint32_t warpPrefix = (w > 0) ? warpSums[w - 1] : 0u;
    *total = warpSums[SCAN_THREADS / 32 - 1];
    __syncthreads();
    return warpPrefix + x - v;
}

// A thread's SCAN_ITEMS consecutive elements as two 16-byte accesses where the
// array allows them (base is a multiple of SCAN_ITEMS): a batch's key counts are
// read twice and written twice per scan, and in 4-byte steps a warp's access
// touches every 32-byte sector eight times (2M keys: 45 us a scan, 27 this way).
static_assert(SCAN_ITEMS == 8, "two 16-byte accesses a thread");

__device__ __forceinline__ bool scan_wide(const uint32_t *p, uint64_t base, uint64_t n)
{
    return base + SCAN_ITEMS <= n && (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

__device__ __forceinline__ void scan_load(const uint32_t *in, uint64_t base, uint64_t n, uint32_t (&v)[SCAN_ITEMS])
{
    if (scan_wide(in, base, n)) {
        const uint4 x = *reinterpret_cast<const uint4 *>(in + base), y = *reinterpret_cast<const uint4 *>(in + base + 4);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; i++) v[i] = (base + i < n) ? in[base + i] : 0u;
    }
}

__device__ __forceinline__ void scan_store(uint32_t *out, uint64_t base, uint64_t n, const uint32_t (&v)[SCAN_ITEMS])
{
    if (scan_wide(out, base, n)) {
        *reinterpret_cast<uint4 *>(out + base) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4 *>(out + base + 4) = make_uint4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; i++)
            if (base + i < n) out[base + i] = v[i];
    }
}

// Scans the block's tile with `off` as its offset; returns the tile's total.
__device__ __forceinline__ uint32_t scan_tile(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *zeroIn,
                                              uint32_t blockOff)
{
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS], s = 0;
    scan_load(in, base, n, v);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) s += v[i];
    if (zeroIn) {
        const uint32_t zero[SCAN_ITEMS] = {};
        scan_store(zeroIn, base, n, zero);
    }
    uint32_t tot;
    uint32_t off = blockOff + block_exclusive_scan(s, &tot);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        const uint32_t x = v[i];
        v[i] = off;
        off += x;
    }
    scan_store(out, base, n, v);
    return tot;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t *__restrict__ in, uint64_t n,
                                                              uint32_t *__restrict__ sums)
{
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS], s = 0;
    scan_load(in, base, n, v);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) s += v[i];
    uint32_t tot;
    block_exclusive_scan(s, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Scans one tile per block; adds the block's offset from `blockOffsets`
// (nullptr for a single-block scan, which also writes the grand total).
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tile(const uint32_t *in, uint32_t *out, uint64_t n,
                                                            const uint32_t *__restrict__ blockOffsets,
                                                            uint32_t *total_dev, uint32_t *zeroIn)
{
    const uint32_t tot = scan_tile(in, out, n, zeroIn, blockOffsets ? blockOffsets[blockIdx.x] : 0u);
    if (!blockOffsets && total_dev && threadIdx.x == 0) *total_dev = tot;
}

// Second pass of the two-launch scan: each block finds its offset by summing
// the tile sums of all blocks before it (read from L2; used while the tile
// count is small), then scans its tile; the last block writes the total.
constexpr uint64_t SCAN_LOOKUP_MAX_TILES = 4096;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tile_lookup(const uint32_t *in, uint32_t *out, uint64_t n,
                                                                   const uint32_t *__restrict__ sums,
                                                                   uint32_t *total_dev, uint32_t *zeroIn)
{
    uint32_t part = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += SCAN_THREADS) part += sums[b];
    uint32_t blockOff;   // sum of all earlier tiles (the block total of the parts)
    block_exclusive_scan(part, &blockOff);
    const uint32_t tot = scan_tile(in, out, n, zeroIn, blockOff);
    if (total_dev && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_dev = blockOff + tot;
}

__global__ void k_scan_total(const uint32_t *scannedSums, const uint32_t *sums, uint64_t nb, uint32_t *total_dev)
{
    if (threadIdx.x == 0 && blockIdx.x == 0 && total_dev) *total_dev = scannedSums[nb - 1] + sums[nb - 1];
}

// A scan of up to SCAN_ONE elements in one launch of one block (in place, or out
// apart): the task builder and the small sorts scan a few thousand counts many
// times a join, and a launch costs more than the block.
constexpr int SCAN_ONE_THREADS = 1024;
constexpr int SCAN_ONE_ITEMS = 16;
constexpr uint64_t SCAN_ONE = (uint64_t)SCAN_ONE_THREADS * SCAN_ONE_ITEMS;

__global__ void __launch_bounds__(SCAN_ONE_THREADS) k_scan_one(const uint32_t *in, uint32_t *out, uint32_t n,
                                                               uint32_t *total_dev, uint32_t *zeroIn)
{
    __shared__ uint32_t ws[32];
    const uint32_t per = (n + SCAN_ONE_THREADS - 1) / SCAN_ONE_THREADS;   // consecutive elements of a thread
    const uint32_t base = threadIdx.x * per;
    uint32_t v[SCAN_ONE_ITEMS], sum = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ONE_ITEMS; i++) {
        v[i] = ((uint32_t)i < per && base + i < n) ? in[base + i] : 0u;
        sum += v[i];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane_id() >= (uint32_t)o) x += y;
    }
    if (lane_id() == 31) ws[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t s = ws[threadIdx.x];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane_id() >= (uint32_t)o) s += y;
        }
        ws[threadIdx.x] = s;
    }
    __syncthreads();
    uint32_t run = x - sum + (threadIdx.x >= 32 ? ws[(threadIdx.x >> 5) - 1] : 0u);
#pragma unroll
    for (int i = 0; i < SCAN_ONE_ITEMS; i++) {
        if ((uint32_t)i < per && base + i < n) {
            if (zeroIn) zeroIn[base + i] = 0u;
            out[base + i] = run;
            run += v[i];
        }
    }
    if (total_dev && threadIdx.x == 0) *total_dev = ws[31];
}

uint64_t ceil_div(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

size_t scan_temp_elems(uint64_t n)
{
    size_t e = 0;
    while (n > (uint64_t)SCAN_TILE) {
        uint64_t nb = ceil_div(n, SCAN_TILE);
        e += 2 * nb;
        n = nb;
    }
    return e + 1;
}

cudaError_t scan_rec(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *temp, uint32_t *total_dev,
                     cudaStream_t s, uint32_t *zeroIn = nullptr)
{
    if (n == 0) {
        if (total_dev) return cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s);
        return cudaSuccess;
    }
    if (n <= (uint64_t)SCAN_TILE) {
        k_scan_tile<<<1, SCAN_THREADS, 0, s>>>(in, out, n, nullptr, total_dev, zeroIn); sj_note_launch();
        return cudaGetLastError();
    }
    if (n <= SCAN_ONE) {
        k_scan_one<<<1, SCAN_ONE_THREADS, 0, s>>>(in, out, (uint32_t)n, total_dev, zeroIn); sj_note_launch();
        return cudaGetLastError();
    }
    uint64_t nb = ceil_div(n, SCAN_TILE);
    uint32_t *sums = temp, *scanned = temp + nb;
    k_scan_reduce<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, sums); sj_note_launch();
    if (nb <= SCAN_LOOKUP_MAX_TILES) {
        k_scan_tile_lookup<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, out, n, sums, total_dev, zeroIn);
        sj_note_launch();
        return cudaGetLastError();
    }
    cudaError_t e = scan_rec(sums, scanned, nb, temp + 2 * nb, nullptr, s);
    if (e != cudaSuccess) return e;
    if (total_dev) {
        k_scan_total<<<1, 32, 0, s>>>(scanned, sums, nb, total_dev);
        sj_note_launch();
    }
    k_scan_tile<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, out, n, scanned, nullptr, zeroIn); sj_note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------- radix sort --

constexpr int RS_THREADS = 256;
constexpr int RS_CHUNKS = 8;                       // chunks of RS_THREADS keys per tile
constexpr int RS_TILE = RS_THREADS * RS_CHUNKS;    // 2048 keys per block
constexpr int RS_WARPS = RS_THREADS / 32;

template <typename K>
__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(const K *__restrict__ keys, uint64_t n, int shift,
                                                           uint32_t *__restrict__ blockHist, uint32_t nb)
{
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    uint64_t base = (uint64_t)blockIdx.x * RS_TILE;
#pragma unroll
    for (int c = 0; c < RS_CHUNKS; c++) {
        uint64_t idx = base + (uint64_t)c * RS_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&h[(uint32_t)(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
    blockHist[(uint64_t)threadIdx.x * nb + blockIdx.x] = h[threadIdx.x];   // digit-major
}

// Stable scatter: keys keep their input order within a digit.
template <typename K>
__global__ void __launch_bounds__(RS_THREADS) k_radix_scatter(const K *__restrict__ keysIn,
                                                              const uint32_t *__restrict__ valsIn,
                                                              K *__restrict__ keysOut, uint32_t *__restrict__ valsOut,
                                                              uint64_t n, int shift,
                                                              const uint32_t *__restrict__ digitOffsets, uint32_t nb)
{
    __shared__ uint32_t base[256];
    __shared__ uint32_t warpCnt[RS_WARPS][256];
    base[threadIdx.x] = digitOffsets[(uint64_t)threadIdx.x * nb + blockIdx.x];
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) warpCnt[w][threadIdx.x] = 0;
    __syncthreads();
    const int w = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t ltmask = (1u << lane) - 1u;
    uint64_t tileBase = (uint64_t)blockIdx.x * RS_TILE;
    for (int c = 0; c < RS_CHUNKS; c++) {
        uint64_t idx = tileBase + (uint64_t)c * RS_THREADS + threadIdx.x;
        bool valid = idx < n;
        K key = valid ? keysIn[idx] : (K)0;
        uint32_t val = valid ? valsIn[idx] : 0u;
        uint32_t d = valid ? ((uint32_t)(key >> shift) & 255u) : 256u;
        uint32_t peers = __match_any_sync(0xffffffffu, d);
        uint32_t rank = __popc(peers & ltmask);
        if (valid && rank == 0) warpCnt[w][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t pre = 0;
            for (int v = 0; v < w; v++) pre += warpCnt[v][d];
            uint32_t pos = base[d] + pre + rank;
            keysOut[pos] = key;
            valsOut[pos] = val;
        }
        __syncthreads();
        uint32_t add = 0;
#pragma unroll
        for (int v = 0; v < RS_WARPS; v++) { add += warpCnt[v][threadIdx.x]; warpCnt[v][threadIdx.x] = 0; }
        base[threadIdx.x] += add;
        __syncthreads();
    }
}

template <typename K>
cudaError_t radix_sort(K *keys, uint32_t *vals, K *keysAlt, uint32_t *valsAlt, uint64_t n, int bits, void *temp,
                       int *resultInAlt, cudaStream_t s)
{
    *resultInAlt = 0;
    if (n <= 1 || bits <= 0) return cudaSuccess;
    uint32_t nb = (uint32_t)ceil_div(n, RS_TILE);
    uint32_t *hist = (uint32_t *)temp;
    uint32_t *scanTemp = hist + (size_t)256 * nb;
    K *kin = keys, *kout = keysAlt;
    uint32_t *vin = vals, *vout = valsAlt;
    int alt = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        k_radix_hist<K><<<nb, RS_THREADS, 0, s>>>(kin, n, shift, hist, nb); sj_note_launch();
        cudaError_t e = scan_rec(hist, hist, (uint64_t)256 * nb, scanTemp, nullptr, s);
        if (e != cudaSuccess) return e;
        k_radix_scatter<K><<<nb, RS_THREADS, 0, s>>>(kin, vin, kout, vout, n, shift, hist, nb); sj_note_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        K *tk = kin; kin = kout; kout = tk;
        uint32_t *tv = vin; vin = vout; vout = tv;
        alt ^= 1;
    }
    *resultInAlt = alt;
    return cudaSuccess;
}

// Appends a batch to a device CSR neighbour table: key k's run
// [start[k], start[k+1]) of vals (start[n] = *total) goes to
// cols[rowPtr[k] + fill[k] ...] and fill[k] grows by its length.  A warp takes
// 32 consecutive keys and copies each run with all lanes.  A run that would
// pass its row's end or the caller's capacity is not written and sets *err.
__global__ void __launch_bounds__(256) k_csr_append(const uint32_t *__restrict__ start,
                                                    const uint32_t *__restrict__ total, uint64_t n,
                                                    const int32_t *__restrict__ vals,
                                                    const uint64_t *__restrict__ rowPtr, uint32_t *__restrict__ fill,
                                                    int32_t *__restrict__ cols, uint64_t colsCap,
                                                    unsigned long long *__restrict__ err)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t k0 = ((uint64_t)blockIdx.x * 256 + (threadIdx.x & ~31u));
    if (k0 >= n) return;
    const uint64_t k = k0 + lane;
    const uint32_t tot = *total;
    const uint32_t st = k < n ? start[k] : tot;
    const uint32_t en = k + 1 < n ? start[k + 1] : tot;
    unsigned long long dst = 0;
    bool ok = true;
    if (en > st) {
        const uint64_t rowEnd = rowPtr[k + 1];
        dst = rowPtr[k] + fill[k];
        ok = dst + (en - st) <= rowEnd && rowEnd <= colsCap;
        if (ok) fill[k] += en - st;
        else atomicMax(err, 1ULL);
    }
    uint32_t live = __ballot_sync(0xffffffffu, en > st && ok);
    while (live) {
        const int i = __ffs(live) - 1;
        live &= live - 1;
        const uint32_t s0 = __shfl_sync(0xffffffffu, st, i);
        const uint32_t e0 = __shfl_sync(0xffffffffu, en, i);
        const unsigned long long d0 = __shfl_sync(0xffffffffu, dst, i);
        for (uint32_t p = lane; p < e0 - s0; p += 32) cols[d0 + p] = vals[s0 + p];
    }
}

// Rows of a table that is one batch: rowPtr[k] = start[k] (rowPtr[n] = *total) and
// the rows' lengths.
__global__ void __launch_bounds__(256) k_csr_rows(const uint32_t *__restrict__ start,
                                                  const uint32_t *__restrict__ total, uint64_t n,
                                                  uint64_t *__restrict__ rowPtr, uint32_t *__restrict__ len)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t s = start[k], e = k + 1 < n ? start[k + 1] : *total;
    rowPtr[k] = s;
    len[k] = e - s;
    if (k + 1 == n) rowPtr[n] = e;
}

// *bad = 1 + a row whose fill is not its length (0: none)
__global__ void __launch_bounds__(256) k_csr_check(const uint64_t *__restrict__ rowPtr,
                                                   const uint32_t *__restrict__ fill, uint64_t n,
                                                   unsigned long long *__restrict__ bad)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n && rowPtr[k + 1] - rowPtr[k] != fill[k]) atomicMax(bad, (unsigned long long)k + 1ULL);
}

__global__ void __launch_bounds__(256) k_u32_to_u64(const uint32_t *__restrict__ in, uint64_t n,
                                                    unsigned long long *__restrict__ out)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

__global__ void __launch_bounds__(256) k_u32_to_f32(const uint32_t *__restrict__ in, uint64_t n,
                                                    float *__restrict__ out)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}

}  // namespace

cudaError_t sj_csr_rows(const uint32_t *start, const uint32_t *total, uint64_t n, uint64_t *rowPtr, uint32_t *len,
                        cudaStream_t s)
{
    if (n == 0) return cudaMemsetAsync(rowPtr, 0, sizeof(uint64_t), s);
    k_csr_rows<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(start, total, n, rowPtr, len);
    sj_note_launch();
    return cudaGetLastError();
}

cudaError_t sj_csr_check(const uint64_t *rowPtr, const uint32_t *fill, uint64_t n, unsigned long long *bad,
                         cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_csr_check<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(rowPtr, fill, n, bad);
    sj_note_launch();
    return cudaGetLastError();
}

cudaError_t sj_u32_to_u64(const uint32_t *in, uint64_t n, unsigned long long *out, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_u32_to_u64<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(in, n, out);
    sj_note_launch();
    return cudaGetLastError();
}

cudaError_t sj_u32_to_f32(const uint32_t *in, uint64_t n, float *out, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_u32_to_f32<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(in, n, out);
    sj_note_launch();
    return cudaGetLastError();
}

cudaError_t sj_csr_append(const uint32_t *start, const uint32_t *total, uint64_t n, const int32_t *vals,
                          const uint64_t *rowPtr, uint32_t *fill, int32_t *cols, uint64_t colsCap,
                          unsigned long long *err, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_csr_append<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(start, total, n, vals, rowPtr, fill, cols, colsCap, err);
    sj_note_launch();
    return cudaGetLastError();
}

static std::atomic<unsigned long long> g_launches{0};
void sj_note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
unsigned long long sj_launch_total() { return g_launches.load(std::memory_order_relaxed); }

size_t sj_scan_temp_bytes(uint64_t n) { return scan_temp_elems(n) * sizeof(uint32_t); }

cudaError_t sj_exclusive_scan_u32(const uint32_t *in, uint32_t *out, uint64_t n, void *temp, uint32_t *total_dev,
                                  cudaStream_t s)
{
    return scan_rec(in, out, n, (uint32_t *)temp, total_dev, s);
}

cudaError_t sj_exclusive_scan_u32_clear(uint32_t *in, uint32_t *out, uint64_t n, void *temp, uint32_t *total_dev,
                                        cudaStream_t s)
{
    return scan_rec(in, out, n, (uint32_t *)temp, total_dev, s, in);
}

size_t sj_radix_temp_bytes(uint64_t n)
{
    uint64_t nb = ceil_div(n ? n : 1, RS_TILE);
    return (size_t)256 * nb * sizeof(uint32_t) + sj_scan_temp_bytes((uint64_t)256 * nb);
}

cudaError_t sj_radix_sort_u64_u32(uint64_t *keys, uint32_t *vals, uint64_t *keysAlt, uint32_t *valsAlt, uint64_t n,
                                  int bits, void *temp, int *resultInAlt, cudaStream_t s)
{
    return radix_sort<uint64_t>(keys, vals, keysAlt, valsAlt, n, bits, temp, resultInAlt, s);
}

cudaError_t sj_radix_sort_u32_u32(uint32_t *keys, uint32_t *vals, uint32_t *keysAlt, uint32_t *valsAlt, uint64_t n,
                                  int bits, void *temp, int *resultInAlt, cudaStream_t s)
{
    return radix_sort<uint32_t>(keys, vals, keysAlt, valsAlt, n, bits, temp, resultInAlt, s);
}
