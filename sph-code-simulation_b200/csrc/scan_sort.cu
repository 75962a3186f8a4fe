// scan_sort.cu — device-wide exclusive scan and stable LSD radix sort.
//
// The octree build sorts particles by their Morton-path keys (BHTree::make
// replacement, src/bhtree.cpp:59-115).  The sort is an LSD radix sort with
// 8-bit digits: one read of the keys counts the digits of all passes, then each
// pass is one kernel that reads and writes every key and value once.  A tile
// (2048 keys) ranks its keys stably (warp match + per-warp counts), learns the
// counts of the tiles before it by decoupled look-back (D. Merrill and M.
// Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016; one
// histogram read and one look-back kernel per digit is the sort of A. Adinets and
// D. Merrill, "Onesweep: a faster least significant digit radix sort for GPUs", 2022),
// stages its keys digit-contiguously in shared memory and writes them so that
// consecutive threads store consecutive addresses.
// Below about 200 K keys a pass is bound by launches and the latency of the
// chain inside a tile; with separate histogram, scan and scatter kernels the
// eight passes of 17 K keys took 24 launches and 170 us, of 131 K keys 40
// launches and 241 us.
#include <cstdint>
#include <cuda_runtime.h>

#include "scan_sort.cuh"

namespace sphgpu {

namespace {

constexpr int SCAN_BLOCK = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, v, o);
        if(lane >= o) v += u;
    }
    return v;
}

// Exclusive scan of one value per thread across the block; returns the
// block total in *total.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* smem /* >= 32 */, T* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const T incl = warp_incl_scan(v);
    if(lane == 31) smem[warp] = incl;
    __syncthreads();
    if(warp == 0) {
        T s = lane < nwarps ? smem[lane] : T(0);
        const T si = warp_incl_scan(s);
        if(lane < nwarps) smem[lane] = si - s;
        if(lane == nwarps - 1) smem[32] = si;
    }
    __syncthreads();
    const T r = incl - v + smem[warp];
    *total = smem[32];
    __syncthreads();
    return r;
}

template <typename T>
__global__ void k_tile_reduce(const T* __restrict__ in, long long n, T* __restrict__ sums)
{
    __shared__ T sm[33];
    const long long base = (long long)blockIdx.x * SCAN_TILE;
    T acc = 0;
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + (long long)k * SCAN_BLOCK + threadIdx.x;
        if(i < n) acc += in[i];
    }
    T tot;
    block_excl_scan(acc, sm, &tot);
    if(threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Exclusive scan of one tile, plus an optional per-tile offset.
template <typename T>
__global__ void k_tile_scan(const T* __restrict__ in, long long n, T* __restrict__ out,
                            const T* __restrict__ offsets, T* __restrict__ total)
{
    __shared__ T sm[33];
    const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
    T v[SCAN_ITEMS];
    T acc = 0;
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + k;
        v[k] = i < n ? in[i] : T(0);
        acc += v[k];
    }
    T tot;
    T run = block_excl_scan(acc, sm, &tot);
    if(offsets) run += offsets[blockIdx.x];
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k) {
        const long long i = base + k;
        if(i < n) out[i] = run;
        run += v[k];
    }
    if(total && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *total = run;
}

// returns the number of kernels launched
template <typename T>
int scan_rec(const T* in, T* out, long long n, T* total, ScanScratch& s, int depth, cudaStream_t st)
{
    const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if(tiles <= 1) {
        k_tile_scan<T><<<1, SCAN_BLOCK, 0, st>>>(in, n, out, (const T*)nullptr, total);
        return 1;
    }
    T* sums = reinterpret_cast<T*>(s.level[depth]);
    T* sums_scanned = sums + tiles;
    k_tile_reduce<T><<<(unsigned)tiles, SCAN_BLOCK, 0, st>>>(in, n, sums);
    const int inner = scan_rec<T>(sums, sums_scanned, tiles, (T*)nullptr, s, depth + 1, st);
    k_tile_scan<T><<<(unsigned)tiles, SCAN_BLOCK, 0, st>>>(in, n, out, sums_scanned, total);
    return inner + 2;
}

// ------------------------------------------------------------------ radix
constexpr int RS_BLOCK = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_BLOCK * RS_ITEMS;
constexpr int RS_WARPS = RS_BLOCK / 32;
constexpr int RS_PASSES = 8;
// status word of a tile's digit: count with its state in the top two bits
constexpr unsigned RS_COUNT = 1u << 30, RS_PREFIX = 2u << 30, RS_VALUE = RS_COUNT - 1u;
constexpr int RS_GAVE_UP = 16;     // PASS_GUARD_SORT (common.cuh)
constexpr int RS_POLLS = 1 << 22;  // far beyond any wait for a tile that runs

// scratch of one sort: everything the passes count in, cleared together
struct RadixScratch {
    unsigned* hist;    // [passes][256]
    unsigned* next;    // [passes] tiles taken
    unsigned* status;  // [passes][tiles][256]
};

__host__ __device__ inline long long rs_tiles(long long n) { return (n + RS_TILE - 1) / RS_TILE; }

// digit counts of all passes in one read of the keys
__global__ void __launch_bounds__(RS_BLOCK) k_rs_hist(const uint64_t* __restrict__ keys, int n, int passes,
                                                      unsigned* __restrict__ hist)
{
    __shared__ unsigned h[RS_PASSES][256];
    for(int p = 0; p < passes; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    for(long long i = (long long)blockIdx.x * RS_BLOCK + threadIdx.x; i < n; i += (long long)gridDim.x * RS_BLOCK) {
        const uint64_t k = keys[i];
        for(int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 0xff], 1u);
    }
    __syncthreads();
    for(int p = 0; p < passes; ++p) {
        const unsigned c = h[p][threadIdx.x];
        if(c) atomicAdd(&hist[p * 256 + threadIdx.x], c);
    }
}

// One pass: the tile's keys ranked stably by digit, the counts of the tiles
// before it taken from their status words (each tile publishes its own counts
// first and their running sums as soon as it knows them; a tile that has only
// counts is added and the look goes one tile further back), then written out
// digit-contiguously.  Tiles are numbered in the order their blocks start, so
// every tile waited for is running or done; the polls are counted all the
// same, and a block that gives up reports it and leaves.
__global__ void __launch_bounds__(RS_BLOCK) k_rs_pass(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                      uint64_t* __restrict__ kout, uint32_t* __restrict__ vout, int n,
                                                      int shift, const unsigned* __restrict__ hist,
                                                      unsigned* __restrict__ next, unsigned* status, int* __restrict__ gave_up)
{
    __shared__ unsigned s_goff[256];       // global offset of digit d for this tile, less its tile-local start
    __shared__ unsigned s_loff[256];       // tile-local start of digit d
    __shared__ unsigned s_wcnt[RS_WARPS][256];
    __shared__ unsigned s_scan[33];
    __shared__ unsigned s_tile;
    __shared__ uint64_t s_key[RS_TILE];
    __shared__ uint32_t s_val[RS_TILE];

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if(t == 0) s_tile = atomicAdd(next, 1u);
    for(int w = 0; w < RS_WARPS; ++w) s_wcnt[w][t] = 0;
    __syncthreads();
    const long long tile = s_tile, base = tile * RS_TILE;
    const unsigned lt_mask = (1u << lane) - 1u;

    // a warp's keys lie one after the other, 32 per round
    uint64_t key[RS_ITEMS];
    uint32_t val[RS_ITEMS];
    unsigned rank[RS_ITEMS];
    const long long mine = base + (long long)warp * (32 * RS_ITEMS) + lane;
#pragma unroll
    for(int r = 0; r < RS_ITEMS; ++r) {
        const long long i = mine + 32 * r;
        key[r] = i < n ? kin[i] : ~0ull;
        val[r] = i < n ? vin[i] : 0u;
    }
#pragma unroll
    for(int r = 0; r < RS_ITEMS; ++r) {
        const bool valid = mine + 32 * r < n;
        const unsigned d = valid ? (unsigned)((key[r] >> shift) & 0xff) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        unsigned before = 0;
        if(valid && lane == leader) {
            before = s_wcnt[warp][d];
            s_wcnt[warp][d] = before + __popc(peers);
        }
        rank[r] = __shfl_sync(0xffffffffu, before, leader) + __popc(peers & lt_mask);
        __syncwarp();
    }
    __syncthreads();
    // digit t: counts of the warps before each, and of the whole tile
    unsigned cnt = 0;
    for(int w = 0; w < RS_WARPS; ++w) {
        const unsigned c = s_wcnt[w][t];
        s_wcnt[w][t] = cnt;
        cnt += c;
    }
    volatile unsigned* st = status;
    st[tile * 256 + t] = (tile == 0 ? RS_PREFIX : RS_COUNT) | cnt;
    unsigned tot;
    const unsigned gbase = block_excl_scan(hist[t], s_scan, &tot);
    const unsigned loff = block_excl_scan(cnt, s_scan, &tot);
    unsigned sum = 0;
    for(long long k = tile - 1; k >= 0; --k) {
        unsigned v = st[k * 256 + t];
        for(int polls = 0; v < RS_COUNT; ++polls) {
            if(polls >= RS_POLLS) {
                atomicOr(gave_up, RS_GAVE_UP);
                v = RS_PREFIX;
                break;
            }
            v = st[k * 256 + t];
        }
        sum += v & RS_VALUE;
        if(v >= RS_PREFIX) break;
    }
    if(tile > 0) st[tile * 256 + t] = RS_PREFIX | (sum + cnt);
    s_loff[t] = loff;
    s_goff[t] = gbase + sum - loff;
    __syncthreads();
#pragma unroll
    for(int r = 0; r < RS_ITEMS; ++r) {
        if(mine + 32 * r < n) {
            const unsigned d = (unsigned)((key[r] >> shift) & 0xff);
            const unsigned lp = s_loff[d] + s_wcnt[warp][d] + rank[r];
            s_key[lp] = key[r];
            s_val[lp] = val[r];
        }
    }
    __syncthreads();
    const int count = (int)min((long long)RS_TILE, (long long)n - base);
    for(int k = t; k < count; k += RS_BLOCK) {
        const uint64_t q = s_key[k];
        const unsigned o = s_goff[(unsigned)((q >> shift) & 0xff)] + (unsigned)k;
        if(o < (unsigned)n) {  // (always, unless a block gave up)
            kout[o] = q;
            vout[o] = s_val[k];
        }
    }
}

}  // namespace

size_t scan_scratch_bytes(long long n)
{
    // geometric series of per-level tile sums (x2 for scanned copies), padded
    size_t total = 0;
    long long m = n;
    while(m > SCAN_TILE) {
        m = (m + SCAN_TILE - 1) / SCAN_TILE;
        total += (size_t)(2 * m + 64) * 8;
    }
    return total + 1024;
}

void scan_scratch_init(ScanScratch& s, void* buf, long long n)
{
    char* p = static_cast<char*>(buf);
    long long m = n;
    int d = 0;
    while(m > SCAN_TILE && d < ScanScratch::MAXLEV) {
        m = (m + SCAN_TILE - 1) / SCAN_TILE;
        s.level[d++] = p;
        p += (size_t)(2 * m + 64) * 8;
    }
}

int exclusive_scan(const int* in, int* out, long long n, int* total, ScanScratch& s, cudaStream_t st)
{
    return scan_rec<int>(in, out, n, total, s, 0, st);
}
int exclusive_scan(const unsigned* in, unsigned* out, long long n, unsigned* total, ScanScratch& s, cudaStream_t st)
{
    return scan_rec<unsigned>(in, out, n, total, s, 0, st);
}
int exclusive_scan(const unsigned long long* in, unsigned long long* out, long long n, unsigned long long* total,
                   ScanScratch& s, cudaStream_t st)
{
    return scan_rec<unsigned long long>(in, out, n, total, s, 0, st);
}

static size_t radix_words(long long n) { return (size_t)RS_PASSES * 256 + 64 + (size_t)RS_PASSES * 256 * rs_tiles(n); }

size_t radix_scratch_bytes(int n) { return radix_words(n) * sizeof(unsigned) + 256; }

// Sorts (keys, vals) by the low `bits` bits of the keys; results end up in
// (keys, vals) again (the alternate buffers are used as ping-pong).  A pass
// whose look-back gave up sets RS_GAVE_UP in *gave_up.
int radix_sort(uint64_t*& keys, uint32_t*& vals, uint64_t*& keys_alt, uint32_t*& vals_alt, int n, int bits,
               void* scratch, int* gave_up, cudaStream_t st)
{
    if(n <= 1) return 0;
    const int ntiles = (int)rs_tiles(n), passes = (bits + 7) / 8;
    RadixScratch s;
    s.hist = static_cast<unsigned*>(scratch);
    s.next = s.hist + RS_PASSES * 256;
    s.status = s.next + 64;
    const size_t words = (size_t)RS_PASSES * 256 + 64 + (size_t)passes * 256 * ntiles;
    cudaMemsetAsync(scratch, 0, words * sizeof(unsigned), st);
    k_rs_hist<<<min(ntiles, 148 * 4), RS_BLOCK, 0, st>>>(keys, n, passes, s.hist);
    for(int p = 0; p < passes; ++p) {
        k_rs_pass<<<ntiles, RS_BLOCK, 0, st>>>(keys, vals, keys_alt, vals_alt, n, 8 * p, s.hist + 256 * p, s.next + p,
                                               s.status + (size_t)256 * ntiles * p, gave_up);
        uint64_t* tk = keys;
        keys = keys_alt;
        keys_alt = tk;
        uint32_t* tv = vals;
        vals = vals_alt;
        vals_alt = tv;
    }
    return 1 + passes;
}

}  // namespace sphgpu
