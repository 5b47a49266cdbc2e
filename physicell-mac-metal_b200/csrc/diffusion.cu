// diffusion.cu — LOD Thomas sweeps, Dirichlet reset and gradients (sm_100a).
//
// Reference semantics: shaders/diffusion_2d.metal:28-157 (x sweep) and
// :165-292 (y sweep), one tridiagonal solve per line over the interior
// nodes 1..n-2 with the decay on the diagonal; src/microenvironment.mm:127-152
// (applyDirichletBC); :282-342 (computeGradients).  The z sweep applies the
// same per-line rule along k.
//
// The solve.  Every line of one (instance, substrate, axis) family has the
// same matrix, so g_i = c / den_i and 1 / den_i are one table (LineRule,
// built in FP64 on the host).  With h_i = (rho_i + fold_i) / den_i the
// reference's two passes are
//     forward   d_i = g_i d_{i-1} + h_i        (d_0 = 0)
//     backward  x_i = g_i x_{i+1} + d_i        (x_{n-1} = 0)
// one FMUL + one FFMA, then one FFMA per value, 2 n dependent steps.  Here a
// line is eliminated from both ends towards its middle (a twisted
// factorisation): the left half as above, the right half by the mirrored
// recurrence (the matrix is symmetric, so its coefficients are the same
// ones counted from the right end), a 2 x 2 system in the middle, and both
// halves substituted outwards.  The same operations per value, but two
// independent chains of n / 2 each way: one thread runs them side by side
// (split_line), or two lanes of a warp take one each (lane_half, in the
// fused 2-D steps).  End nodes keep their value or take the Dirichlet target.
//
// Data movement.  density is [s][k][j][i] FP32 with rows padded to a pitch
// px = nx rounded up to 4 floats, so every row starts on 16 bytes.  Each
// warp of a persistent CTA runs its own pipeline of shared-memory stages:
// lane 0 issues one TMA tensor copy (cp.async.bulk.tensor) of the warp's
// next tile into a free stage, completion is counted on one mbarrier per
// stage, the warp solves the current stage in place and writes it back with
// one tensor store.  Tiles are loaded while the previous one is solved, so
// HBM sees a deep queue with few threads.
//   x tile:   32 lines (one per lane) stored [line][P], P = row_smem_pitch(nx)
//             (2-D map, box P x 32); all lanes walk their lines in step,
//             4 values per 16-byte shared access, coefficients broadcast;
//   y/z tile: 32 adjacent columns x n rows stored [row][32] (3-D map, box
//             32 x n); lane = column.
// Lines too long for a tensor box are solved by one warp each, as scans of
// the two affine recurrences over the warp's lanes (k_sweep_long).
// Every value is read from HBM once and written once per sweep.  Waits are
// bounded: a wait that runs out records PCG_DEV_TIMEOUT in the status word,
// drains what it issued, and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "lines.cuh"

namespace pcg {

// The LineRule a tile descriptor carries.
__device__ __forceinline__ LineRule rule_of(const SweepTile& t)
{
    LineRule r;
    r.tab = t.tab;
    r.n = t.n;
    r.fold = t.fold;
    r.T = t.T;
    r.dir = t.inst >> 31;
    r.inst = t.inst & 0x7fffffffu;
    return r;
}

__device__ __forceinline__ bool tile_on(const LineRule& r, const uint8_t* __restrict__ mask)
{
    return mask == nullptr || (mask[r.inst] & STEP_DIFFUSE);
}

// Column tile lane -> (slab, column).
__device__ __forceinline__ uint32_t lane_slab(const SweepTile& tile, int lane) { return static_cast<uint32_t>(lane) / tile.width; }
__device__ __forceinline__ uint32_t lane_col(const SweepTile& tile, int lane) { return static_cast<uint32_t>(lane) % tile.width; }

// The lane's line lies on a face of the block (3-D: x faces and, for z
// lines, y faces; 2-D y lines: x faces).
__device__ __forceinline__ bool on_face(const SweepTile& tile, int lane)
{
    const uint32_t i = tile.i0 + lane_col(tile, lane);
    if (i == 0u || i + 1u == tile.nx) return true;
    if (tile.face & TILE_AXIS_Z) {
        const uint32_t j = tile.outer + lane_slab(tile, lane);
        return j == 0u || j + 1u == tile.outer_n;
    }
    return false;
}

// ------------------------------------------------------------------ tile geometry

// Tensor coordinates of a column tile's box: (x, slab, line position).
__device__ __forceinline__ void tile_coords(const SweepTile& tile, int* c)
{
    c[0] = static_cast<int>(tile.i0);
    c[1] = static_cast<int>(tile.outer);
    c[2] = 0;
}

// Issue (lane 0) the load of 'tile' into stage 'st' and of its rule's
// coefficient table into 'stab' (the stage's table area), both counted on
// 'bar'.
template <bool kRows>
__device__ __forceinline__ void issue_tile_load(const SweepTile& tile, const float* __restrict__ tab, const void* tmaps,
                                                float* st, float* stab, uint64_t* bar, int lane)
{
    if (lane != 0) return;
    const uint32_t n = tile.n;
    const uint32_t tb = tab_floats(n) * 4u;    // 32-byte multiple, 32-byte aligned source
    const void* map = static_cast<const unsigned char*>(tmaps) + static_cast<size_t>(tile.map) * 128;
    if (kRows) {
        mbar_arrive_expect_tx(bar, 32u * row_smem_pitch(n) * 4u + tb);   // the whole box, fill included
        tensor_load2(st, map, 0, static_cast<int>(tile.outer), bar);
    } else {
        int c[3];
        tile_coords(tile, c);
        mbar_arrive_expect_tx(bar, 32u * n * 4u + tb);
        tensor_load3(st, map, c[0], c[1], c[2], bar);
    }
    bulk_load(stab, tab + tile.tab, tb, bar);
}

template <bool kRows>
__device__ __forceinline__ void issue_tile_store(const SweepTile& tile, const void* tmaps, const float* st, int lane)
{
    if (lane != 0) return;
    const void* map = static_cast<const unsigned char*>(tmaps) + static_cast<size_t>(tile.map) * 128;
    if (kRows) {
        tensor_store2(map, 0, static_cast<int>(tile.outer), st);
    } else {
        int c[3];
        tile_coords(tile, c);
        tensor_store3(map, c[0], c[1], c[2], st);
    }
    bulk_commit();
}

// ------------------------------------------------------------------ tile solves

__device__ __forceinline__ void solve_rows(float* st, const LineRule& r, const float* t, int lane, int count)
{
    if (lane >= count) return;
    row_line(st + lane * static_cast<int>(row_smem_pitch(r.n)), r, t);
}

// y/z tile: lane = column, rows at st + j * 32 (32 lanes, 32 banks).
__device__ __forceinline__ void solve_cols(float* st, const SweepTile& tile, const LineRule& r,
                                           const float* t, int lane, bool apply_faces)
{
    if (lane_col(tile, lane) >= tile.count || lane_slab(tile, lane) >= tile.nslab) return;
    const int n = static_cast<int>(r.n);
    float* c = st + lane;
    if (apply_faces && (tile.face & TILE_FACE) && on_face(tile, lane)) {
        for (int j = 0; j < n; ++j) c[j * 32] = r.T;   // applyDirichletBC fused: the line lies on a face
        return;
    }
    if (n >= 3)
        split_line(
            t, n, r.fold,
            [c](int q) {
                return make_float4(c[(4 * q) * 32], c[(4 * q + 1) * 32], c[(4 * q + 2) * 32], c[(4 * q + 3) * 32]);
            },
            [c](int q, float4 v) {
                c[(4 * q) * 32] = v.x;
                c[(4 * q + 1) * 32] = v.y;
                c[(4 * q + 2) * 32] = v.z;
                c[(4 * q + 3) * 32] = v.w;
            });
    if (r.dir) {
        c[0] = r.T;
        c[(n - 1) * 32] = r.T;
    }
}

// ------------------------------------------------------------------ pipelined kernel

// Shared memory: kBarBytes of mbarriers ([warp][stage]), then the stages
// ([warp][stage][stage_floats], 128-byte aligned).  Between them, one tile
// descriptor per stage ([warp][stage], 64 bytes): the descriptor of the tile
// a stage holds, stashed when its load is issued.  Both regions are sized
// for the launch shape and rounded to 128 bytes.
constexpr int kBarBytes = 512;    // at most 16 warps x 4 stages
__host__ __device__ constexpr int round128(int b) { return (b + 127) & ~127; }
__host__ __device__ constexpr int sweep_bar_bytes(int warps, int nstages) { return round128(warps * nstages * 8); }
__host__ __device__ constexpr int sweep_header_bytes(int warps, int nstages)
{
    return sweep_bar_bytes(warps, nstages) + round128(warps * nstages * 64);
}

template <bool kRows>
__global__ void __launch_bounds__(256, 1) k_sweep_tma(const SweepTile* __restrict__ tiles, uint32_t ntiles,
                                                   const float* __restrict__ tab, const void* __restrict__ tmaps,
                                                   int stage_floats, int nstages, int tab_area, int apply_faces,
                                                   const uint8_t* __restrict__ mask, unsigned* __restrict__ status)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    // stage: [tile data][tab_area floats of coefficient table]
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem) + warp * nstages;
    SweepTile* descs = reinterpret_cast<SweepTile*>(smem + sweep_bar_bytes(nwarps, nstages)) + warp * nstages;
    float* stages = reinterpret_cast<float*>(smem + sweep_header_bytes(nwarps, nstages)) +
                    static_cast<size_t>(warp) * nstages * stage_floats;
    if (lane == 0)
        for (int s = 0; s < nstages; ++s) mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();

    const uint32_t gw = blockIdx.x * nwarps + warp, tw = gridDim.x * nwarps;
    const uint32_t ntw = gw < ntiles ? (ntiles - gw + tw - 1) / tw : 0u;
    const int ahead = nstages - 1;   // loads in flight while one stage is solved
    uint32_t issued = 0;
    bool ok = true;
    // 'nd' is the descriptor of the next tile to issue, loaded one tile
    // ahead so its latency hides behind the current solve
    SweepTile nd{};
    if (ntw) nd = tiles[gw];
    auto issue = [&]() {
        const int s = static_cast<int>(issued % nstages);
        float* st = stages + s * stage_floats;
        issue_tile_load<kRows>(nd, tab, tmaps, st, st + stage_floats - tab_area, &bars[s], lane);
        if (lane == 0) descs[s] = nd;
        ++issued;
        if (issued < ntw) nd = tiles[gw + issued * tw];
    };
    while (issued < ntw && static_cast<int>(issued) < ahead) issue();
    for (uint32_t k = 0; k < ntw; ++k) {
        // refill: tile k + ahead goes to the stage of tile k - 1, whose store
        // (issued last) must have finished reading shared memory
        if (issued < ntw) {
            bulk_wait_read<0>();
            __syncwarp();
            issue();
        }
        const int s = static_cast<int>(k % nstages);
        if (!mbar_wait(&bars[s], (k / nstages) & 1u, status)) {
            ok = false;
            break;
        }
        __syncwarp();
        const SweepTile tile = descs[s];
        const LineRule r = rule_of(tile);
        float* st = stages + s * stage_floats;
        const float* t = st + stage_floats - tab_area;
        if (tile_on(r, mask)) {
            if (kRows) {
                solve_rows(st, r, t, lane, static_cast<int>(tile.count));
            } else {
                solve_cols(st, tile, r, t, lane, apply_faces != 0);
            }
        }
        fence_async_smem();
        __syncwarp();
        issue_tile_store<kRows>(tile, tmaps, st, lane);
    }
    if (!ok) {
        // let every load this warp issued land before the CTA exits (bounded)
        for (uint32_t k = 0; k < issued; ++k) {
            const int s = static_cast<int>(k % nstages);
            if (!mbar_wait(&bars[s], (k / nstages) & 1u, status)) break;
        }
    }
    bulk_wait_all();
}

// ------------------------------------------------------- fused x + y sweeps of a plane

// One CTA per x-y plane (one z slab of one instance-substrate): the plane
// (rows of pitch P = row_smem_pitch(nx), zero-filled past nx) and both
// rules' tables come in with one tensor box and two bulk copies; every row
// is solved (x sweep), then every column (y sweep), and the plane goes back
// with one tensor store.  ZK: x-z planes, columns only.  The steps on each
// line are those of the x and y tile kernels, so the result is the same
// bits, but the plane crosses HBM once for both sweeps.  Several CTAs per
// SM overlap one plane's copies with another's solves, and each CTA
// prefetches into L2 (a tensor-box prefetch, no shared memory) the plane of
// the CTA 'ahead' jobs later, so that CTA's load is served from L2.
// Large x-z planes come in strips of columns (z lines are independent).
//
// What bounds it: the x + y pass by the shared-memory wavefronts of its two
// solves beside HBM, the z pass by HBM.  Per chunk of a warp's lines a solve
// moves 16 wavefronts of values and, until g settles, 3 of table; keeping
// the settled g and 1 / den in registers took the 120^3 x + y pass from
// 75.1 to 65.9 us (332 MB, 5.0 TB/s; z 54.8 us, 6.1 TB/s), with 80 registers
// 80^3 from 68.4 to 60.6 and 48^3 from 56.8 to 50.5; four 150^3 fields 73.3 +
// 55.5 -> 57.6 + 45.9 us (one thread per line, not 128).  Measured and not
// taken: a line's chunks held in registers between the passes (fewer
// wavefronts, but unrolled code starves on instruction fetch: 120^3 79 us),
// half a line per thread with the halves in two warps (66-89 us).
template <bool ZK>
__global__ void __launch_bounds__(256, 3)
    k_sweep_planes(const PlaneJob* __restrict__ jobs, const float* __restrict__ tab, const void* __restrict__ tmaps,
                   int apply_faces, const uint8_t* __restrict__ mask, unsigned* __restrict__ status, uint32_t ahead)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
    float* pl = reinterpret_cast<float*>(smem + 128);
    // the job, the tables and the tensor maps are written once, before any
    // step; the density and the mask may be the predecessor's
    const PlaneJob jb = jobs[blockIdx.x];
    const uint32_t ii = jb.inst & kPlaneInstMask;
    const uint32_t nx = jb.nx, ny = jb.ny, P = ZK ? jb.pitch : plane_pitch(nx, false);
    float* tx = pl + plane_data_floats(ZK ? P : nx, ny, ZK);
    float* ty = ZK ? tx : tx + tab_floats(nx);
    const void* map = static_cast<const unsigned char*>(tmaps) + static_cast<size_t>(jb.map) * 128;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    }
    if (!await_predecessors()) return;
    if (mask && !(mask[ii] & STEP_DIFFUSE)) return;   // the whole CTA leaves together
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t tbx = ZK ? 0u : tab_floats(nx) * 4u, tby = tab_floats(ny) * 4u;
        mbar_arrive_expect_tx(bar, P * ny * 4u + tbx + tby);   // the whole box, fill included
        if (ZK) {
            tensor_load3(pl, map, static_cast<int>(jb.x0), static_cast<int>(jb.row0), 0, bar);
        } else {
            tensor_load2(pl, map, 0, static_cast<int>(jb.row0), bar);
            bulk_load(tx, tab + jb.tab_x, tbx, bar);
        }
        bulk_load(ty, tab + jb.tab_y, tby, bar);
        // the plane of a CTA that starts a little later ('ahead' jobs on,
        // about a quarter of a residency): into L2 now, so its load is an
        // L2 hit rather than a wait on HBM
        if (ahead != 0 && blockIdx.x + ahead < gridDim.x) {
            const PlaneJob nj = jobs[blockIdx.x + ahead];
            if (!mask || (mask[nj.inst & kPlaneInstMask] & STEP_DIFFUSE)) {
                const void* nmap = static_cast<const unsigned char*>(tmaps) + static_cast<size_t>(nj.map) * 128;
                if (ZK) tensor_prefetch3(nmap, static_cast<int>(nj.x0), static_cast<int>(nj.row0), 0);
                else tensor_prefetch2(nmap, 0, static_cast<int>(nj.row0));
            }
        }
    }
    bool got;
    if (status[1] & PCG_DEV_TEST_GIVE_UP) {   // test switch: this wait's bound ran out
        if (threadIdx.x == 0) atomicOr(status, PCG_DEV_TIMEOUT);
        got = false;
    } else {
        got = mbar_wait(bar, 0, status);
    }
    if (!__syncthreads_and(got)) {
        // a wait ran out: one more bounded wait for the copies before the
        // CTA releases its shared memory
        if (threadIdx.x == 0 && !got) mbar_wait(bar, 0, status);
        return;
    }
    LineRule rx{}, ry{};
    rx.n = nx;
    rx.fold = jb.fold_x;
    rx.T = jb.T_x;
    rx.dir = (jb.inst & kPlaneDirX) ? 1u : 0u;
    ry.n = ny;
    ry.fold = jb.fold_y;
    ry.T = jb.T_y;
    ry.dir = (jb.inst & kPlaneDirY) ? 1u : 0u;
    if (!ZK) {
        for (uint32_t r = threadIdx.x; r < ny; r += blockDim.x) row_line(pl + r * P, rx, tx);
        __syncthreads();
    }
    // faces of the block's last sweep (2-D: y, 3-D: z; applyDirichletBC): x
    // faces, and a whole z plane on a y face
    const bool faces = apply_faces && (jb.inst & kPlaneFaces) != 0;
    const bool slab_face = faces && (jb.inst & kPlaneSlabFace) != 0;
    if (!slab_face)
        for (uint32_t c = threadIdx.x; c < nx; c += blockDim.x) plane_col(pl + c, static_cast<int>(P), ry, ty);
    if (faces) {
        __syncthreads();
        // every column, or the block's first and last where the job has them
        const uint32_t x0 = ZK ? jb.x0 : 0u, last = (ZK ? jb.full_nx : nx) - 1u - x0;
        for (uint32_t j = threadIdx.x; j < ny; j += blockDim.x) {
            if (slab_face)
                for (uint32_t c = 0; c < nx; ++c) pl[j * P + c] = ry.T;
            if (x0 == 0) pl[j * P] = ry.T;
            if (last < nx) pl[j * P + last] = ry.T;
        }
    }
    dependents_may_launch();   // late: waiting blocks take slots and issue from this one's solves
    fence_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
        if (ZK) tensor_store3(map, static_cast<int>(jb.x0), static_cast<int>(jb.row0), 0, pl);
        else tensor_store2(map, 0, static_cast<int>(jb.row0), pl);
        bulk_commit();
        bulk_wait_read<0>();   // shared memory may be released once the store has read it
    }
}

// ------------------------------------------------------- any line length

// Lines too long for a tensor box (and any line without a tensor map): one
// warp per line, kLongLines lines per CTA (8 adjacent columns: one 32-byte
// sector per row), 2^log_parts CTAs per tile of up to 32 lines.  Both
// recurrences are affine, d_i = g_i d_{i-1} + h_i and x_i = g_i x_{i+1} +
// d_i, so lane l takes K consecutive positions, runs them from zero, the 32
// (product of g, end value) pairs are scanned with shuffles, and the lane
// runs its positions again from the value the scan gives it: 4 K + 10
// dependent steps where one thread per line has 2 n.
// Values and tables are staged in shared memory with one pad per K
// positions, so that the lanes' runs hit different banks, and a line's g
// and values stay in registers between the passes.  A line longer than one
// segment of 32 K positions keeps d in place in global memory between a
// forward and a backward walk over its segments.
//
// What bounds it: the latency of those steps and of one round trip to
// memory.  A diffusion step (x and y) of 701 x 530 voxels, two substrates,
// takes 14.2 us, where one thread per line in place (n dependent,
// uncoalesced accesses) took 516; the x sweep of 300-voxel lines (2 x 300 x
// 300 x 60) 95 us, where 32-line tiles with bulk row copies took 335.  The
// check for values that are not finite costs 1 to 2 %; within the register
// bound below, since the fourth block of an SM goes at 65 registers and with it
// a fifth of the rate (300^3: 385 -> 465 us).
template <int K>
__host__ __device__ constexpr int long_stride() { return 32 * (K + 1) + 4; }   // 4 mod 32: 8 columns hit 8 bank groups

template <int K>
__device__ __forceinline__ int long_at(int i) { return i + i / K; }

// One direction of a line's segment: v[k] = h (forward) or d (backward) in,
// the recurrence's values out; 'edge' enters at the segment's first
// position in walking order.  Returns the value at the last one.
//   The product G of many g below 1 underflows to 0, and 0 times an infinite
// value would be NaN where a walk position by position carries it on undamped.
// WILD: an infinite a is multiplied by 'one' instead: 1, or 0 where the rule
// has no coupling and every g is 0.  finite: the lane's scanned value is (an
// infinite or NaN value anywhere on a segment leaves some lane's not finite).
template <int K, bool BACK, bool WILD>
__device__ __forceinline__ float long_scan(float (&v)[K], const float (&g)[K], float edge, float one, bool& finite, int lane)
{
    auto term = [one](float m, float a, float d) { return fmaf(WILD && fabsf(a) == INFINITY ? one : m, a, d); };
    float D = 0.f, G = 1.f;
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const int k = BACK ? K - 1 - q : q;
        D = fmaf(g[k], D, v[k]);
        G *= g[k];
    }
    // inclusive scan of the affine maps in walking order
    const int pos = BACK ? 31 - lane : lane;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float Dp = BACK ? __shfl_down_sync(0xffffffffu, D, o) : __shfl_up_sync(0xffffffffu, D, o);
        const float Gp = BACK ? __shfl_down_sync(0xffffffffu, G, o) : __shfl_up_sync(0xffffffffu, G, o);
        if (pos >= o) {
            D = term(G, Dp, D);
            G *= Gp;
        }
    }
    finite = fabsf(D) < INFINITY;
    const float Dx = BACK ? __shfl_down_sync(0xffffffffu, D, 1) : __shfl_up_sync(0xffffffffu, D, 1);
    const float Gx = BACK ? __shfl_down_sync(0xffffffffu, G, 1) : __shfl_up_sync(0xffffffffu, G, 1);
    float x = pos == 0 ? edge : term(Gx, edge, Dx);
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const int k = BACK ? K - 1 - q : q;
        x = fmaf(g[k], x, v[k]);
        v[k] = x;
    }
    return __shfl_sync(0xffffffffu, x, BACK ? 0 : 31);
}

// A line of one segment that holds an infinite or NaN value, from and to the
// lane's place in the stage (out of line: its registers are not the sweep's).
template <int K>
__device__ __noinline__ void long_wild(float* s, const float* sg, const float* si, int n, float fold, float one, int lane)
{
    float v[K], g[K];
    bool finite;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = lane * K + k, at = lane * (K + 1) + k;
        g[k] = sg[at];
        v[k] = (s[k] + (i == 1 || i == n - 2 ? fold : 0.f)) * si[at];
    }
    long_scan<K, false, true>(v, g, 0.f, one, finite, lane);
    // the forward walk leaves NaN (0 times infinity) at the end node and past
    // it, where the way back starts from 0
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (lane * K + k >= n - 1) v[k] = 0.f;
    long_scan<K, true, true>(v, g, 0.f, one, finite, lane);
#pragma unroll
    for (int k = 0; k < K; ++k) s[k] = v[k];
}

template <int K>
__global__ void __launch_bounds__(32 * kLongLines, K <= 16 ? 4 : 2) k_sweep_long(float* __restrict__ dens,
                                                                const SweepTile* __restrict__ tiles, int log_parts,
                                                                const float* __restrict__ tab, int apply_faces,
                                                                const uint8_t* __restrict__ mask)
{
    constexpr int kSeg = 32 * K, kStride = long_stride<K>();
    extern __shared__ float sh[];
    float* sg = sh + kLongLines * kStride;   // g of the segment's positions
    float* si = sg + kStride;                // 1 / den
    const SweepTile tile = tiles[blockIdx.x >> log_parts];   // written once, before any step
    const uint32_t l0 = (blockIdx.x & ((1u << log_parts) - 1u)) * kLongLines;   // the CTA's first line of the tile
    const LineRule r = rule_of(tile);
    if (!await_predecessors()) return;
    dependents_may_launch();
    if (l0 >= tile.count || !tile_on(r, mask)) return;   // the whole CTA leaves together
    const int n = static_cast<int>(r.n), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool rows = (tile.face & TILE_ROWS) != 0;
    const float* t = tab + r.tab + seq_table_offset(r.n);
    // the line and position a thread moves at step i: rows, one line per
    // warp; columns, 8 adjacent lines per row of threads
    const int line = rows ? warp : static_cast<int>(threadIdx.x & 7u);
    const int p0 = rows ? lane : static_cast<int>(threadIdx.x >> 3), dp = 32;
    const bool mine = l0 + line < tile.count;
    const size_t ls = rows ? tile.rs : 1, ps = rows ? 1 : tile.rs;
    float* gl = dens + tile.base + static_cast<size_t>(l0 + line) * ls;
    float* sl = sh + line * kStride;
    const bool face = !rows && apply_faces && (tile.face & TILE_FACE) && mine && on_face(tile, static_cast<int>(l0) + line);
    const float* sv = sh + warp * kStride + lane * (K + 1);
    float* sw = sh + warp * kStride + lane * (K + 1);
    float v[K], g[K];

    auto load = [&](int s0) {   // the segment's values and table; end nodes and places past the line as zeros
        for (int p = static_cast<int>(threadIdx.x); p < kSeg; p += static_cast<int>(blockDim.x)) {
            const int i = s0 + p;
            sg[long_at<K>(p)] = i < n ? __ldg(t + ((i >> 2) << 3) + (i & 3)) : 0.f;
            si[long_at<K>(p)] = i < n ? __ldg(t + ((i >> 2) << 3) + 4 + (i & 3)) : 0.f;
        }
#pragma unroll 8
        for (int p = p0; p < kSeg; p += dp) {
            const int i = s0 + p;
            sl[long_at<K>(p)] = (mine && i > 0 && i < n - 1) ? gl[static_cast<size_t>(i) * ps] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = sv[k];
            g[k] = sg[lane * (K + 1) + k];
        }
    };
    auto to_rhs = [&](int s0) {   // h_i = (rho_i + fold_i) / den_i
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = s0 + lane * K + k;
            const float f = (i == 1 || i == n - 2) ? r.fold : 0.f;
            v[k] = (v[k] + f) * si[lane * (K + 1) + k];
        }
    };
    auto store = [&](int s0, bool last, bool put = true) {   // interior values (and, at the end, the end nodes' targets and the faces)
        if (put) {
#pragma unroll
            for (int k = 0; k < K; ++k) sw[k] = v[k];
        }
        __syncthreads();
        if (mine) {
#pragma unroll 8
            for (int p = p0; p < kSeg; p += dp) {
                const int i = s0 + p;
                if (i >= n) continue;
                const bool end = i == 0 || i == n - 1;
                if (last && (face || (end && r.dir))) gl[static_cast<size_t>(i) * ps] = r.T;
                else if (!end) gl[static_cast<size_t>(i) * ps] = sl[long_at<K>(p)];
            }
        }
        __syncthreads();   // the stage may be loaded again
    };

    bool finite;
    auto coupled = [&]() { return n > 3 && __ldg(t + 1) > 0.f ? 1.f : 0.f; };   // long_scan's 'one': g of the first interior node
    if (n <= kSeg) {
        load(0);
        to_rhs(0);
        long_scan<K, false, false>(v, g, 0.f, 0.f, finite, lane);
        long_scan<K, true, false>(v, g, 0.f, 0.f, finite, lane);
        const bool wild = __any_sync(0xffffffffu, !finite);
        if (wild) long_wild<K>(sw, sg, si, n, r.fold, coupled(), lane);
        store(0, true, !wild);
        return;
    }
    const float one = coupled();
    float edge = 0.f;
    int s0 = 0;
    for (; s0 < n; s0 += kSeg) {
        load(s0);
        to_rhs(s0);
        edge = long_scan<K, false, true>(v, g, edge, one, finite, lane);
        store(s0, false);
    }
    edge = 0.f;
    for (s0 -= kSeg; s0 >= 0; s0 -= kSeg) {
        load(s0);
        edge = long_scan<K, true, true>(v, g, edge, one, finite, lane);
        store(s0, true);
    }
}

// ------------------------------------------------------------- Dirichlet

__global__ void k_dirichlet(float* __restrict__ dens, const FaceJob* __restrict__ jobs)
{
    if (!await_predecessors()) return;
    dependents_may_launch();
    const FaceJob jb = jobs[blockIdx.x];
    float* base = dens + jb.base;
    const uint32_t nx = jb.nx, ny = jb.ny, nz = jb.nz;
    const size_t px = jb.px, slab = px * ny;
    // edges of every slab (microenvironment.mm:140-150)
    const uint32_t per = 2u * nx + 2u * ny;
    const size_t total = static_cast<size_t>(nz) * per;
    for (size_t e = threadIdx.x; e < total; e += blockDim.x) {
        const uint32_t k = static_cast<uint32_t>(e / per), q = static_cast<uint32_t>(e % per);
        uint32_t i, j;
        if (q < nx) { i = q; j = 0; }
        else if (q < 2u * nx) { i = q - nx; j = ny - 1; }
        else if (q < 2u * nx + ny) { i = 0; j = q - 2u * nx; }
        else { i = nx - 1; j = q - 2u * nx - ny; }
        base[k * slab + j * px + i] = jb.T;
    }
    if (nz > 1) {   // z faces (3-D rule)
        const size_t plane = static_cast<size_t>(nx) * ny;
        for (size_t e = threadIdx.x; e < 2 * plane; e += blockDim.x) {
            const size_t k = (e < plane) ? 0 : (nz - 1);
            const size_t v = e % plane;
            base[k * slab + (v / nx) * px + (v % nx)] = jb.T;
        }
    }
}

// ------------------------------------------------------------- gradients

__global__ void k_gradients(const float* __restrict__ dens, float* __restrict__ gx, float* __restrict__ gy,
                            float* __restrict__ gz, const GradJob* __restrict__ jobs)
{
    const GradJob jb = jobs[blockIdx.y];
    const size_t nx = jb.nx, ny = jb.ny, nz = jb.nz, nv = nx * ny * nz, px = jb.px;
    const float* D = dens + jb.base;
    for (size_t n = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; n < nv;
         n += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t i = n % nx, j = (n / nx) % ny, k = n / (nx * ny);
        const size_t a = (k * ny + j) * px + i;       // device offset of voxel n
        const size_t o = jb.out_base + n;             // dense output
        const size_t sy = px, sz = px * ny;
        double v;
        if (nx == 1) v = 0.0;
        else if (i == 0) v = (static_cast<double>(D[a + 1]) - D[a]) * jb.inv_dx;
        else if (i == nx - 1) v = (static_cast<double>(D[a]) - D[a - 1]) * jb.inv_dx;
        else v = (static_cast<double>(D[a + 1]) - D[a - 1]) * 0.5 * jb.inv_dx;
        if (gx) gx[o] = static_cast<float>(v);
        if (ny == 1) v = 0.0;
        else if (j == 0) v = (static_cast<double>(D[a + sy]) - D[a]) * jb.inv_dy;
        else if (j == ny - 1) v = (static_cast<double>(D[a]) - D[a - sy]) * jb.inv_dy;
        else v = (static_cast<double>(D[a + sy]) - D[a - sy]) * 0.5 * jb.inv_dy;
        if (gy) gy[o] = static_cast<float>(v);
        if (nz > 1) {
            if (k == 0) v = (static_cast<double>(D[a + sz]) - D[a]) * jb.inv_dz;
            else if (k == nz - 1) v = (static_cast<double>(D[a]) - D[a - sz]) * jb.inv_dz;
            else v = (static_cast<double>(D[a + sz]) - D[a - sz]) * 0.5 * jb.inv_dz;
        } else {
            v = 0.0;
        }
        if (gz) gz[o] = static_cast<float>(v);
    }
}

// ------------------------------------------------------------- launchers

size_t sweep_tma_smem(int warps, int nstages, int stage_floats)
{
    return static_cast<size_t>(sweep_header_bytes(warps, nstages)) +
           static_cast<size_t>(warps) * nstages * stage_floats * sizeof(float);
}

cudaError_t allow_max_smem(const void* fn)
{
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    return e;
}

int sweep_tma_occupancy(bool rows, int warps, int nstages, int stage_floats)
{
    const void* fn = rows ? reinterpret_cast<const void*>(k_sweep_tma<true>)
                          : reinterpret_cast<const void*>(k_sweep_tma<false>);
    if (warps < 1 || warps * nstages * 8 > kBarBytes || nstages < 2) return 0;
    if (allow_max_smem(fn) != cudaSuccess) return 0;
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, warps * 32, sweep_tma_smem(warps, nstages, stage_floats)) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return b;
}

cudaError_t launch_sweep_tma(cudaStream_t st, bool rows, const SweepTile* tiles, uint32_t ntiles,
                             const float* tab, const void* tmaps, int apply_faces,
                             const uint8_t* mask, unsigned* status, TmaCfg cfg)
{
    if (ntiles == 0) return cudaSuccess;
    // stages start 128-byte aligned (tensor copies), the table area on 32 bytes
    if (cfg.stage_floats % 32 != 0 || cfg.tab_floats % 8 != 0 || cfg.tab_floats >= cfg.stage_floats)
        return cudaErrorInvalidValue;
    const size_t smem = sweep_tma_smem(cfg.warps, cfg.stages, cfg.stage_floats);
    if (rows)
        launch_chained(st, k_sweep_tma<true>, cfg.grid, cfg.warps * 32, smem, tiles, ntiles, tab, tmaps,
                                                                   cfg.stage_floats, cfg.stages, cfg.tab_floats,
                                                                   apply_faces, mask, status);
    else
        launch_chained(st, k_sweep_tma<false>, cfg.grid, cfg.warps * 32, smem, tiles, ntiles, tab, tmaps,
                                                                    cfg.stage_floats, cfg.stages, cfg.tab_floats,
                                                                    apply_faces, mask, status);
    return cudaGetLastError();
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link-time dependency on libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
    }
    return fn;
}

bool encode_column_map(void* map128, float* block, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t px, int axis,
                       uint32_t n, uint32_t width)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    if (!fn || n == 0 || n > kTensorMaxN || (px & 3u) || (reinterpret_cast<uintptr_t>(block) & 15u)) return false;
    if (width != 32u && width != 16u && width != 8u) return false;
    const cuuint64_t row = static_cast<cuuint64_t>(px) * 4u, slab = row * ny;
    // y lines: (x, z, y); z lines: (x, y, z) -- the line runs along the last dimension
    const cuuint64_t dims[3] = {nx, axis == 1 ? nz : ny, axis == 1 ? ny : nz};
    const cuuint64_t strides[2] = {axis == 1 ? slab : row, axis == 1 ? row : slab};
    const cuuint32_t box[3] = {width, 32u / width, n};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    const CUresult r = fn(static_cast<CUtensorMap*>(map128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, block, dims, strides,
                          box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

bool encode_row_map(void* map128, float* block, uint32_t nx, uint64_t rows, uint32_t px)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    const uint32_t P = row_smem_pitch(nx);
    if (!fn || nx == 0 || nx > kRowTensorMaxN || rows == 0 || (px & 3u) || px < nx ||
        (reinterpret_cast<uintptr_t>(block) & 15u))
        return false;
    const cuuint64_t dims[2] = {nx, rows};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(px) * 4u};
    const cuuint32_t box[2] = {P, 32u};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = fn(static_cast<CUtensorMap*>(map128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, block, dims, strides,
                          box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

bool encode_plane_map(void* map128, float* block, uint32_t nx, uint32_t ny, uint64_t rows, uint32_t px)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    const uint32_t P = row_smem_pitch(nx);
    if (!fn || nx == 0 || nx > kRowTensorMaxN || ny == 0 || ny > 256 || rows == 0 || (px & 3u) || px < nx ||
        (reinterpret_cast<uintptr_t>(block) & 15u))
        return false;
    const cuuint64_t dims[2] = {nx, rows};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(px) * 4u};
    const cuuint32_t box[2] = {P, ny};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = fn(static_cast<CUtensorMap*>(map128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, block, dims, strides,
                          box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// x-z planes of one instance-substrate for the z lines: dims (x, y, z), box
// width x 1 x nz (width columns, a multiple of 4, one y, every z).
bool encode_xz_plane_map(void* map128, float* block, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t px, uint32_t width)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    const uint32_t bx = width;
    if (!fn || nx == 0 || bx == 0 || (bx & 3u) || bx > 256 || nz == 0 || nz > 256 || ny == 0 || (px & 3u) || px < nx ||
        (reinterpret_cast<uintptr_t>(block) & 15u))
        return false;
    const cuuint64_t row = static_cast<cuuint64_t>(px) * 4u;
    const cuuint64_t dims[3] = {nx, ny, nz};
    const cuuint64_t strides[2] = {row, row * ny};
    const cuuint32_t box[3] = {bx, 1u, nz};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    const CUresult r = fn(static_cast<CUtensorMap*>(map128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, block, dims, strides,
                          box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

size_t sweep_planes_smem(uint32_t floats) { return 128 + static_cast<size_t>(floats) * sizeof(float); }

static const void* plane_kernel(bool z)
{
    return z ? reinterpret_cast<const void*>(&k_sweep_planes<true>) : reinterpret_cast<const void*>(&k_sweep_planes<false>);
}

cudaError_t sweep_planes_prepare()
{
    for (bool z : {false, true}) {
        cudaError_t e = allow_max_smem(plane_kernel(z));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(plane_kernel(z), cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int sweep_planes_ctas(bool z, int threads, uint32_t floats)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, plane_kernel(z), threads, sweep_planes_smem(floats)) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t launch_sweep_planes(cudaStream_t st, bool z, int threads, const PlaneJob* jobs, uint32_t njobs,
                                const float* tab, const void* tmaps, uint32_t floats, int apply_faces,
                                const uint8_t* mask, unsigned* status, uint32_t ahead)
{
    if (njobs == 0) return cudaSuccess;
    return launch_chained(st, z ? k_sweep_planes<true> : k_sweep_planes<false>, njobs, threads, sweep_planes_smem(floats), jobs,
                          tab, tmaps, apply_faces, mask, status, ahead);
}

template <int K>
static cudaError_t long_variant(cudaStream_t st, float* dens, const SweepTile* tiles, uint32_t ntiles, int log_parts,
                                const float* tab, int apply_faces, const uint8_t* mask)
{
    const size_t smem = static_cast<size_t>(kLongLines + 2) * long_stride<K>() * sizeof(float);   // at most 43 KB
    launch_chained(st, k_sweep_long<K>, ntiles << log_parts, 32 * kLongLines, smem, dens, tiles, log_parts, tab, apply_faces, mask);
    return cudaGetLastError();
}

cudaError_t launch_sweep_long(cudaStream_t st, float* dens, const SweepTile* tiles, uint32_t ntiles, uint32_t lines,
                              const float* tab, int nmax, int apply_faces, const uint8_t* mask)
{
    if (ntiles == 0) return cudaSuccess;
    const int log_parts = lines <= kLongLines ? 0 : lines <= 2 * kLongLines ? 1 : 2;
    // positions per lane: the fewest that hold the longest line in one
    // segment (a lane's steps, registers and shared memory grow with them),
    // at most 32; longer lines take several segments
    if (nmax <= 32 * 12) return long_variant<12>(st, dens, tiles, ntiles, log_parts, tab, apply_faces, mask);
    if (nmax <= 32 * 16) return long_variant<16>(st, dens, tiles, ntiles, log_parts, tab, apply_faces, mask);
    if (nmax <= 32 * 24) return long_variant<24>(st, dens, tiles, ntiles, log_parts, tab, apply_faces, mask);
    return long_variant<32>(st, dens, tiles, ntiles, log_parts, tab, apply_faces, mask);
}

cudaError_t launch_dirichlet(cudaStream_t st, float* dens, const FaceJob* jobs, uint32_t njobs)
{
    if (njobs == 0) return cudaSuccess;
    launch_chained(st, k_dirichlet, njobs, 256, 0, dens, jobs);
    return cudaGetLastError();
}

cudaError_t launch_gradients(cudaStream_t st, const float* dens, float* gx, float* gy, float* gz,
                             const GradJob* jobs, uint32_t njobs, uint64_t max_voxels)
{
    if (njobs == 0) return cudaSuccess;
    uint64_t bx = (max_voxels + 255) / 256;
    if (bx > 4096) bx = 4096;
    if (bx == 0) bx = 1;
    dim3 grid(static_cast<unsigned>(bx), njobs);
    k_gradients<<<grid, 256, 0, st>>>(dens, gx, gy, gz, jobs);
    return cudaGetLastError();
}

}  // namespace pcg
