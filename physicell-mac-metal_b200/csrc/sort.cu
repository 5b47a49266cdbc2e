// sort.cu — stable LSD radix sort of (key, value) pairs and a warp-shuffle
// exclusive scan (sm_100a).  The sort backs pcg_sort_pairs_static (the
// secretion order has its own instance-segmented sort, secorder.cu); the
// scan turns the per-voxel counts of the mechanics binning into the
// cell-start table, and serves the secretion run list's tile counts.
//
// One radix pass over D-bit digits, two launches:
//   k_radix_hist     per-tile digit counts -> hist[tile][digit]
//   k_radix_scatter  each warp ranks its contiguous 256 keys with one
//                    ballot per digit bit (peers with the same digit) and a
//                    per-warp running count, warps are combined in warp
//                    order; the tile is laid out in shared memory in digit
//                    order and written back so that consecutive threads
//                    store consecutive elements of one digit's run, at the
//                    digit's first place + the counts of the tiles before
//                    (every tile adds up the rows of all tiles itself: at
//                    most 128 KB of L2 for the 262144 pairs of the static
//                    sort, less time than a scan of the counts between the
//                    two launches: 200003 pairs of 20 bits 38.7 -> 30.5 us,
//                    and 23.1 with one kernel of the chain waiting at a time).
// Ranks follow input order within a warp, warps follow tile order and
// tiles follow each other in order, so each pass is stable.
#include "pcg_kernels.cuh"

namespace pcg {

namespace {
constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;     // 2048 keys per tile
constexpr int kWarps = kThreads / 32;
constexpr int kDigitBits = 8;
constexpr int kRadix = 1 << kDigitBits;
constexpr uint32_t kMask = kRadix - 1;
}  // namespace

__global__ void __launch_bounds__(kThreads) k_radix_hist(const uint32_t* __restrict__ keys, uint32_t n, int shift,
                                                         uint32_t* __restrict__ hist)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    __shared__ uint32_t h[kRadix];
    for (int i = threadIdx.x; i < kRadix; i += kThreads) h[i] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * kTile;
    uint32_t kk[kItems];   // all loads in flight together
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t i = base + k * kThreads + threadIdx.x;
        kk[k] = i < n ? keys[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        if (base + k * kThreads + threadIdx.x < n) atomicAdd(&h[(kk[k] >> shift) & kMask], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < kRadix; d += kThreads) hist[blockIdx.x * kRadix + d] = h[d];
}

__global__ void __launch_bounds__(kThreads) k_radix_scatter(const uint32_t* __restrict__ kin,
                                                            const uint32_t* __restrict__ vin,
                                                            uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                            uint32_t n, int shift,
                                                            const uint32_t* __restrict__ hist, uint32_t ntiles)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    __shared__ uint32_t wcnt[kWarps][kRadix];
    __shared__ uint32_t gbase[kRadix];
    __shared__ uint32_t tbase[kRadix];      // first place of each digit in the tile
    __shared__ uint32_t wtot[kWarps], rtot[kWarps];
    __shared__ __align__(16) uint32_t sk[kTile], sv[kTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // What bounds a pass is latency, so the loads of the pairs, then of the
    // counts, are in flight together before the ranks (whose warp barriers
    // order memory) need them.
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t base = blockIdx.x * kTile + warp * (32 * kItems);
    uint32_t kk[kItems], vv[kItems], rk[kItems], peers[kItems];
    int dg[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const uint32_t i = base + r * 32 + lane;
        kk[r] = i < n ? kin[i] : 0u;
        vv[r] = i < n ? vin[i] : 0u;
    }
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&wcnt[0][0])[i] = 0;
    {
        // each digit's count in all tiles and in those before this one: a
        // quarter of the rows per thread, four digits at a time, 32 rows in
        // flight (8: a sort takes 42.5 us)
        const uint32_t c = threadIdx.x & 63u, g = threadIdx.x >> 6;
        const uint4* rows = reinterpret_cast<const uint4*>(hist) + c;
        uint4 all = make_uint4(0, 0, 0, 0), pre = all;
        for (uint32_t t0 = g; t0 < ntiles; t0 += 128u) {
            uint4 v[32];
#pragma unroll
            for (int u = 0; u < 32; ++u) {
                const uint32_t t = t0 + 4u * u;
                v[u] = t < ntiles ? rows[t * (kRadix / 4)] : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 32; ++u) {
                const uint32_t m = t0 + 4u * u < blockIdx.x ? 0xffffffffu : 0u;
                all.x += v[u].x;
                all.y += v[u].y;
                all.z += v[u].z;
                all.w += v[u].w;
                pre.x += v[u].x & m;
                pre.y += v[u].y & m;
                pre.z += v[u].z & m;
                pre.w += v[u].w & m;
            }
        }
        reinterpret_cast<uint4*>(sk)[threadIdx.x] = all;   // sk, sv: [quarter][digit] until the tile is laid out
        reinterpret_cast<uint4*>(sv)[threadIdx.x] = pre;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        dg[r] = base + r * 32 + lane < n ? static_cast<int>((kk[r] >> shift) & kMask) : kRadix;   // kRadix marks an empty lane
        peers[r] = same_digit<kDigitBits>(static_cast<uint32_t>(dg[r]));
    }
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const bool ok = dg[r] < kRadix;
        const uint32_t at = ok ? wcnt[warp][dg[r]] : 0u;
        rk[r] = at + __popc(peers[r] & lt);
        __syncwarp();
        if (ok && (peers[r] & lt) == 0u) wcnt[warp][dg[r]] = at + __popc(peers[r]);
        __syncwarp();
    }
    __syncthreads();
    static_assert(kThreads == kRadix, "one thread per digit");
    {
        const int d = threadIdx.x;
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = wcnt[w][d];
            wcnt[w][d] = sum;
            sum += c;
        }
        uint32_t rsum = 0, rpre = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            rsum += sk[q * kRadix + d];
            rpre += sv[q * kRadix + d];
        }
        // exclusive scans of the digit totals across the block: this tile's
        // and all tiles'
        uint32_t incl = sum, rincl = rsum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            const uint32_t z = __shfl_up_sync(0xffffffffu, rincl, o);
            if (lane >= o) {
                incl += y;
                rincl += z;
            }
        }
        if (lane == 31) {
            wtot[warp] = incl;
            rtot[warp] = rincl;
        }
        __syncthreads();
        uint32_t before = 0, rbefore = 0;
        for (int w = 0; w < warp; ++w) {
            before += wtot[w];
            rbefore += rtot[w];
        }
        tbase[d] = before + incl - sum;
        gbase[d] = rbefore + rincl - rsum + rpre;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        if (dg[r] < kRadix) {
            const uint32_t t = tbase[dg[r]] + wcnt[warp][dg[r]] + rk[r];
            sk[t] = kk[r];
            sv[t] = vv[r];
        }
    }
    __syncthreads();
    const uint32_t count = min(static_cast<uint32_t>(kTile), n - blockIdx.x * kTile);
    for (uint32_t t = threadIdx.x; t < count; t += kThreads) {
        const uint32_t k = sk[t];
        const int d = static_cast<int>((k >> shift) & kMask);
        const uint32_t dst = gbase[d] + (t - tbase[d]);
        kout[dst] = k;
        vout[dst] = sv[t];
    }
}

// ------------------------------------------------------------------ scan

// Up to kOneBlock values are scanned by one block in one launch (one tile by
// k_scan_tiles: a 1024-thread block would wait for an SM of its own).  Scans
// over more reduce, then scan: k_tile_sums writes every tile's total, the totals
// are scanned (recursively), and k_scan_tiles scans every tile once more,
// starting from its scanned total -- one read pass and one read / write pass
// over the values.

constexpr int kOneThreads = 1024;
constexpr int kOneItems = 8;   // groups of 4 consecutive values per thread
constexpr uint64_t kOneBlock = 4ull * kOneItems * kOneThreads;   // 32768

// Exclusive scan of n <= kOneBlock values.  Thread t holds values 4t .. 4t + 3
// of each group of 4096: all loads are in flight together, the groups' warp
// scans overlap, and one pass over the 8 x 32 warp totals joins them.  Bound
// by latency: two round trips to L2 and two barriers, where three launches of
// the tile kernels pay theirs each (the forces of 2000 cells, whose cell-start
// table has 4356 voxels, 21.6 -> 18.5 us; of 20000 cells in 17576 voxels 29.8
// -> 27.1, in 29791 27.7 -> 26.3).
__global__ void __launch_bounds__(kOneThreads) k_scan_one(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                          uint32_t n)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    __shared__ uint32_t wtot[kOneItems * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    uint32_t v[kOneItems][4], pre[kOneItems];
#pragma unroll
    for (int h = 0; h < kOneItems; ++h) {
        const uint32_t i = 4096u * h + 4u * threadIdx.x;
        if (aligned && i + 4u <= n) {
            const uint4 q = *reinterpret_cast<const uint4*>(in + i);
            v[h][0] = q.x; v[h][1] = q.y; v[h][2] = q.z; v[h][3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[h][k] = i + k < n ? in[i + k] : 0u;
        }
    }
#pragma unroll
    for (int h = 0; h < kOneItems; ++h) {
        uint32_t tot = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t x = v[h][k];
            v[h][k] = tot;
            tot += x;
        }
        uint32_t incl = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        pre[h] = incl - tot;
        if (lane == 31) wtot[h * 32 + warp] = incl;
    }
    __syncthreads();
    if (warp == 0) {   // the warp totals, in order: 8 consecutive ones per lane
        uint32_t w[kOneItems], tot = 0;
#pragma unroll
        for (int k = 0; k < kOneItems; ++k) {
            w[k] = tot;
            tot += wtot[lane * kOneItems + k];
        }
        uint32_t incl = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
#pragma unroll
        for (int k = 0; k < kOneItems; ++k) wtot[lane * kOneItems + k] = w[k] + incl - tot;
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < kOneItems; ++h) {
        const uint32_t i = 4096u * h + 4u * threadIdx.x, p = pre[h] + wtot[h * 32 + warp];
        if (aligned && i + 4u <= n) {
            *reinterpret_cast<uint4*>(out + i) = make_uint4(v[h][0] + p, v[h][1] + p, v[h][2] + p, v[h][3] + p);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i + k < n) out[i + k] = v[h][k] + p;
        }
    }
}

// Sum of one 2048-value tile per block.
__global__ void __launch_bounds__(kThreads) k_tile_sums(const uint32_t* __restrict__ in, uint64_t n,
                                                        uint32_t* __restrict__ sums)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    __shared__ uint32_t wsum[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kTile + static_cast<uint64_t>(threadIdx.x) * kItems;
    uint32_t tot = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint64_t i = base + k;
        tot += i < n ? in[i] : 0u;
    }
    tot = __reduce_add_sync(0xffffffffu, tot);
    if (lane == 0) wsum[warp] = tot;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) t += wsum[w];
        sums[blockIdx.x] = t;
    }
}

// Exclusive scan of 256 per-thread values across the block: returns the
// sum of the values of the threads before this one; *total gets the sum of
// all (wsum: kWarps + 1 shared words).
__device__ __forceinline__ uint32_t block_exclusive(uint32_t x, uint32_t* wsum, uint32_t* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < kWarps ? wsum[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < kWarps; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < kWarps) wsum[lane] = wi - w;
        if (lane == kWarps - 1) wsum[kWarps] = wi;
    }
    __syncthreads();
    const uint32_t before = wsum[warp] + (incl - x);
    *total = wsum[kWarps];
    __syncthreads();   // wsum is reused by the next call
    return before;
}

// Exclusive scan of one 2048-value tile per block, each tile starting from
// offs[blockIdx.x] when offs != nullptr.  The tile is two halves of 1024
// values; in each, thread t owns values 4t .. 4t + 3, moved as one 16-byte
// access when the tile is whole and the arrays 16-byte aligned, so that a
// warp's loads and stores are contiguous.
__global__ void __launch_bounds__(kThreads) k_scan_tiles(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                         uint64_t n, const uint32_t* __restrict__ offs)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    static_assert(kTile == 2 * 4 * kThreads, "two halves of four values per thread");
    __shared__ uint32_t wsum[kWarps + 1];
    const uint64_t tile = static_cast<uint64_t>(blockIdx.x) * kTile;
    const bool vec = tile + kTile <= n && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    uint32_t run = offs ? offs[blockIdx.x] : 0u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint64_t i0 = tile + static_cast<uint64_t>(h) * (kTile / 2) + 4ull * threadIdx.x;
        uint32_t v[4];
        if (vec) {
            const uint4 q = *reinterpret_cast<const uint4*>(in + i0);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = i0 + k < n ? in[i0 + k] : 0u;
        }
        uint32_t tot = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t x = v[k];
            v[k] = tot;
            tot += x;
        }
        uint32_t half_total = 0;
        const uint32_t pre = run + block_exclusive(tot, wsum, &half_total);
        if (vec) {
            *reinterpret_cast<uint4*>(out + i0) = make_uint4(v[0] + pre, v[1] + pre, v[2] + pre, v[3] + pre);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i0 + k < n) out[i0 + k] = v[k] + pre;
        }
        run += half_total;
    }
}

static uint64_t tiles_of(uint64_t n) { return (n + kTile - 1) / kTile; }

cudaError_t sort_kernels_load()
{
    // querying a kernel's attributes loads its module on the current device
    // (lazy loading defers that to the first launch otherwise)
    cudaFuncAttributes a;
    const void* ks[] = {reinterpret_cast<const void*>(&k_radix_hist), reinterpret_cast<const void*>(&k_radix_scatter)};
    for (const void* k : ks) {
        const cudaError_t e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

size_t scan_scratch_bytes(uint64_t n)
{
    size_t bytes = 0;
    uint64_t m = tiles_of(n);
    while (m > 1) {
        bytes += ((m * sizeof(uint32_t) + 255) / 256) * 256;
        m = tiles_of(m);
    }
    return bytes + 256;
}

int scan_launches(uint64_t n)
{
    return n <= kOneBlock ? 1 : 2 + scan_launches(tiles_of(n));   // (one tile or one block: one launch)
}

static cudaError_t scan_rec(cudaStream_t st, const uint32_t* in, uint32_t* out, uint64_t n, char* scratch)
{
    const uint64_t nt = tiles_of(n);
    if (nt == 0) return cudaSuccess;
    if (nt == 1) return launch_chained(st, k_scan_tiles, 1, kThreads, 0, in, out, n, nullptr);
    if (n <= kOneBlock) return launch_chained(st, k_scan_one, 1, kOneThreads, 0, in, out, static_cast<uint32_t>(n));
    uint32_t* sums = reinterpret_cast<uint32_t*>(scratch);
    char* next = scratch + ((nt * sizeof(uint32_t) + 255) / 256) * 256;
    launch_chained(st, k_tile_sums, static_cast<unsigned>(nt), kThreads, 0, in, n, sums);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = scan_rec(st, sums, sums, nt, next);
    if (e != cudaSuccess) return e;
    launch_chained(st, k_scan_tiles, static_cast<unsigned>(nt), kThreads, 0, in, out, n, sums);
    return cudaGetLastError();
}

cudaError_t scan_exclusive(cudaStream_t st, const uint32_t* in, uint32_t* out, uint64_t n, void* scratch)
{
    return scan_rec(st, in, out, n, static_cast<char*>(scratch));
}

// ------------------------------------------------------------------ sort

static int passes_for(int bits) { return bits <= 0 ? 0 : (bits + kDigitBits - 1) / kDigitBits; }

size_t radix_sort_scratch_bytes(uint32_t n, int bits)
{
    (void)bits;
    return tiles_of(n ? n : 1) * kRadix * sizeof(uint32_t);
}

int radix_sort_launches(uint32_t n, int bits)
{
    (void)n;
    const int p = passes_for(bits);
    return p == 0 ? 2 : 2 * p;
}

cudaError_t radix_sort_pairs(cudaStream_t st, const uint32_t* k_in, const uint32_t* v_in, uint32_t* k_out,
                             uint32_t* v_out, uint32_t* k_tmp, uint32_t* v_tmp, uint32_t n, int bits, void* scratch)
{
    if (n == 0) return cudaSuccess;
    const uint32_t nt = static_cast<uint32_t>(tiles_of(n));
    uint32_t* hist = static_cast<uint32_t*>(scratch);
    const int passes = passes_for(bits);
    if (passes == 0) {
        cudaError_t e = cudaMemcpyAsync(k_out, k_in, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return e;
        return cudaMemcpyAsync(v_out, v_in, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
    }
    // ping-pong so that the last pass writes (k_out, v_out)
    const uint32_t* ks = k_in;
    const uint32_t* vs = v_in;
    for (int p = 0; p < passes; ++p) {
        // pass p writes out when (passes - 1 - p) is even, tmp otherwise
        const bool to_out = ((passes - 1 - p) & 1) == 0;
        uint32_t* kd = to_out ? k_out : k_tmp;
        uint32_t* vd = to_out ? v_out : v_tmp;
        const int shift = p * kDigitBits;
        cudaError_t e = launch_chained(st, k_radix_hist, nt, kThreads, 0, ks, n, shift, hist);
        if (e == cudaSuccess) e = launch_chained(st, k_radix_scatter, nt, kThreads, 0, ks, vs, kd, vd, n, shift, hist, nt);
        if (e != cudaSuccess) return e;
        ks = kd;
        vs = vd;
    }
    return cudaSuccess;
}

}  // namespace pcg
