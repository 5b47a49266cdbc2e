// steps2d.cu — several main-loop sub-steps of a 2-D simulation in one launch
// (sm_100a).
//
// In 2-D a sub-step (src/main.mm:341-366: x and y sweeps, Dirichlet reset,
// secretion) never couples two substrates of one instance or two instances,
// and a plane of up to 227 KB stays in one CTA's shared memory, so a CTA
// takes its plane in, runs any number of sub-steps on it and puts it back:
// the density crosses L2 / HBM once per call instead of three times per
// sub-step, and a sub-step costs block barriers instead of launches.
//
// What bounds it: the latency of the lines' chains and of the cells' FP64
// updates within one SM (a few planes), their shared-memory traffic (many).
// Lines of up to 128 positions are solved by two lanes of a warp, one per
// half, the half's values in registers between the passes; the halves meet
// through a shuffle.  Longer lines, whose halves would not fit the registers,
// are solved by one thread each in shared memory (split_line).  10 sub-steps
// of 50 x 50 voxels: 37.5 -> 16.8 us without cells, 59.2 -> 25.5 with 500,
// against a plane pass and a secretion launch per sub-step; 181 x 117 with
// three substrates, no cells: 86.5 -> 52.2.
#include "lines.cuh"
#include "secrete.cuh"

namespace pcg {

namespace {

__device__ __forceinline__ float4 table4(uint32_t a)
{
    float4 v;
    asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// One half of a line of n >= 13 positions per lane: lanes 0-15 of the warp
// hold the left halves of 16 lines, lanes 16-31 their right halves.  'p' is
// the line's position 0, ROW: stored contiguously, else P floats apart.  R:
// the left half's chunks.  act = false: the lane takes part without
// storing.  The steps on each position are split_line's: the same bits.
template <int R, bool ROW>
__device__ __forceinline__ void lane_half(const float* tab, const LineRule& r, float* p, int P, bool act)
{
    const SplitTable sp(static_cast<int>(r.n));
    const int hl = sp.hl, nq = sp.nq;
    const bool right = (threadIdx.x & 16u) != 0;
    const int cnt = right ? nq - hl : hl;   // chunks of this lane's half: hl or hl - 1
    const int lead = right ? 4 * nq - static_cast<int>(r.n) : 0;
    const float* t = tab + (right ? sp.right() : 0);
    const int s = ROW ? 0 : (right ? -P : P);
    float* base = ROW ? (right ? p + 4 * (nq - 1) : p) : (right ? p + (4 * nq - 1) * P : p);
    auto ld = [&](int k) {
        if (ROW) {
            const float4 v = *reinterpret_cast<const float4*>(base + (right ? -4 * k : 4 * k));
            return right ? reversed(v) : v;
        }
        const float* c = base + 4 * k * s;
        return make_float4(c[0], c[s], c[2 * s], c[3 * s]);
    };
    auto st = [&](int k, float4 v) {
        if (ROW) {
            *reinterpret_cast<float4*>(base + (right ? -4 * k : 4 * k)) = right ? reversed(v) : v;
            return;
        }
        float* c = base + 4 * k * s;
        c[0] = v.x;
        c[s] = v.y;
        c[2 * s] = v.z;
        c[3 * s] = v.w;
    };
    // the table runs two chunks ahead of the recurrence, and stays where it
    // is written: loads gathered at the top would take the line's registers
    constexpr int kAhead = R > 2 ? 2 : 1, kBuf = kAhead + 1;
    const uint32_t ta = smem_u32(t);
    float4 v[R], g[kBuf], iv[kBuf];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = ld(k);   // a right half one chunk shorter reads the left's innermost one, unused
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
        g[k] = table4(ta + 32u * k);
        iv[k] = table4(ta + 32u * k + 16u);
    }
    const float end0 = take_end(v[0], lead, r.fold);
    const float end = r.dir ? r.T : end0;
    v[1].x += lead == 3 ? r.fold : 0.f;
    float d = 0.f;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (k + kAhead < R) {
            g[(k + kAhead) % kBuf] = table4(ta + 32u * (k + kAhead));
            iv[(k + kAhead) % kBuf] = table4(ta + 32u * (k + kAhead) + 16u);
        }
        const float dn = fwd4(v[k], g[k % kBuf], iv[k % kBuf], d);
        d = k + 1 < R || cnt == R ? dn : d;
    }
    const float dp = __shfl_xor_sync(0xffffffffu, d, 16);
    const float* tj = tab + sp.middle();
    float x = fmaf(tj[right ? 0 : 1], d, dp) * tj[2];
#pragma unroll
    for (int k = R - 1; k >= 0; --k) {
        if (k >= kAhead) g[(k - kAhead) % kBuf] = table4(ta + 32u * (k - kAhead));
        const float xn = bwd4(v[k], g[k % kBuf], x);
        x = k + 1 < R || cnt == R ? xn : x;
        if (k == 0) put_end(v[0], lead, end);
        if (act && (k + 1 < R || cnt == R)) st(k, v[k]);
    }
}

// The body for the line's number of chunks per half (2 .. R).
template <int R, bool ROW>
__device__ __forceinline__ void lane_half_pick(int hl, const float* tab, const LineRule& r, float* p, int P, bool act)
{
    if constexpr (R <= 2) {
        lane_half<2, ROW>(tab, r, p, P, act);
    } else {
        if (hl == R) lane_half<R, ROW>(tab, r, p, P, act);
        else lane_half_pick<R - 1, ROW>(hl, tab, r, p, P, act);
    }
}

// A line by one thread.
template <bool ROW>
__device__ __forceinline__ void whole_line(const float* tab, const LineRule& r, float* p, int P)
{
    if (ROW) row_line(p, r, tab);
    else plane_col(p, P, r, tab);
}

// The rows or columns of the plane: R > 0: 16 lines per warp at a time, two
// lanes a line; R = 0: one thread a line.
template <int R, bool ROW>
__device__ __forceinline__ void lane_lines(float* pl, int P, uint32_t nlines, const LineRule& r, const float* tab)
{
    if constexpr (R == 0) {
        for (uint32_t l = threadIdx.x; l < nlines; l += blockDim.x)
            whole_line<ROW>(tab, r, pl + static_cast<int>(l) * (ROW ? P : 1), P);
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, nwarps = blockDim.x >> 5;
    const int n = static_cast<int>(r.n);
    for (uint32_t l0 = 16u * (threadIdx.x >> 5); l0 < nlines; l0 += 16u * nwarps) {
        const uint32_t l = l0 + (lane & 15u);
        const bool act = l < nlines;
        float* p = pl + static_cast<int>(act ? l : nlines - 1) * (ROW ? P : 1);
        if (n >= 13) lane_half_pick<(R > 0 ? R : 2), ROW>(SplitTable(n).hl, tab, r, p, P, act);
        else if (act && lane < 16u) whole_line<ROW>(tab, r, p, P);   // short lines
    }
}

// A run's voxel as its place in the plane: row off / px (exact: off < 2^16).
__device__ __forceinline__ uint32_t plane_place(uint32_t off, uint32_t px, float inv_px, uint32_t P)
{
    const uint32_t j = static_cast<uint32_t>((static_cast<float>(off) + 0.5f) * inv_px);
    return j * P + (off - j * px);
}

// The CTA's copy of the instance's runs and of its substrate's terms: run r
// covers cells [start[r], start[r + 1]) of 'terms' (c2, 1 / c2, then c0 and
// c1 where the instance has them, 'cap' cells each).
struct StagedRuns {
    double* terms;
    uint32_t *start, *place;
    uint32_t cap, n, f;
};

__device__ __forceinline__ void stage_runs(StagedRuns& sr, uint32_t* count, uint32_t P, uint32_t ii, uint32_t sub,
                                           uint32_t nruns, const RunArgs& a)
{
    const CellInst& in = a.insts[ii];
    const uint32_t S = in.S, px = in.px, T = blockDim.x, off0 = in.cell_off;
    const float inv_px = 1.0f / static_cast<float>(px);
    const double* c0a = a.cs + in.rate_off + sub;
    sr.f = a.flags[ii];
    if (threadIdx.x == 0) *count = 0;
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < nruns; r += T) {
        const uint64_t w = a.run_word[r];
        const uint32_t p0 = a.run_start[r], p1 = a.run_start[r + 1];
        if (static_cast<uint32_t>(w >> kRunDensBits) != ii) break;
        sr.place[r] = plane_place(static_cast<uint32_t>((w & kRunDensMask) - in.dens_off), px, inv_px, P);
        sr.start[r] = p0 - off0;
        sr.start[r + 1] = p1 - off0;   // the next run's thread writes the same
        atomicMax(count, r + 1);
        for (uint32_t q = p0 - off0; q < p1 - off0; ++q) {
            const uint64_t o = static_cast<uint64_t>(q) * S;
            const double c2 = c0a[2 * a.cap + o];
            sr.terms[q] = c2;
            sr.terms[sr.cap + q] = __ddiv_rn(1.0, c2);
            if (sr.f & 1u) sr.terms[2 * sr.cap + q] = c0a[o];
            if (sr.f & 2u) sr.terms[3 * sr.cap + q] = c0a[a.cap + o];
        }
    }
    __syncthreads();
    sr.n = *count;
}

// Secretion of the substrate on the plane: k_secrete's operations in its
// order, B runs per thread side by side, so that their FP64 chains overlap.
__device__ __forceinline__ void secrete_staged(float* pl, const StagedRuns& sr)
{
    constexpr int B = 2;
    const uint32_t T = blockDim.x;
    for (uint32_t r = threadIdx.x; r < sr.n; r += B * T) {
        uint32_t q[B], len[B], e[B], most = 0;
        float rho[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const uint32_t rb = r + b * T;
            const bool ok = rb < sr.n;
            q[b] = ok ? sr.start[rb] : 0u;
            len[b] = ok ? sr.start[rb + 1] - q[b] : 0u;
            e[b] = ok ? sr.place[rb] : 0u;
            rho[b] = pl[e[b]];
            most = max(most, len[b]);
        }
        for (uint32_t k = 0; k < most; ++k) {
            double c0[B], c1[B], c2[B], y[B];
            bool act[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                act[b] = k < len[b];
                const uint32_t o = q[b] + k;
                c2[b] = act[b] ? sr.terms[o] : 1.0;
                y[b] = act[b] ? sr.terms[sr.cap + o] : 1.0;
                c0[b] = act[b] && (sr.f & 1u) ? sr.terms[2 * sr.cap + o] : 0.0;
                c1[b] = act[b] && (sr.f & 2u) ? sr.terms[3 * sr.cap + o] : 0.0;
            }
            secrete_side_by_side<B>(rho, c0, c1, c2, y, act);
        }
#pragma unroll
        for (int b = 0; b < B; ++b)
            if (len[b]) pl[e[b]] = rho[b];
    }
}

// One CTA per (2-D instance, substrate): n_steps sub-steps.  apply_faces:
// with the Dirichlet reset (x faces; the y faces are the lines' ends);
// a.run_word null: no secretion; else shared memory holds the runs and terms
// of the instance's up to stage_cells cells from the stage_off-th 8 bytes on.
template <int R>
__global__ void __launch_bounds__(kSteps2dThreads) k_steps_2d(const PlaneJob* __restrict__ jobs,
                                                                 const float* __restrict__ tab,
                                                                 const void* __restrict__ tmaps, RunArgs a, int n_steps,
                                                                 int apply_faces, uint32_t stage_cells,
                                                                 uint32_t stage_off, unsigned* __restrict__ status)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
    float* pl = reinterpret_cast<float*>(smem + 128);
    const PlaneJob jb = jobs[blockIdx.x];
    const uint32_t ii = jb.inst & kPlaneInstMask;
    const uint32_t nx = jb.nx, ny = jb.ny, P = plane_pitch(nx, false);
    float* tx = pl + plane_data_floats(nx, ny);
    float* ty = tx + tab_floats(nx);
    const void* map = static_cast<const unsigned char*>(tmaps) + static_cast<size_t>(jb.map) * 128;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    }
    if (!await_predecessors()) return;
    dependents_may_launch();
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t tbx = tab_floats(nx) * 4u, tby = tab_floats(ny) * 4u;
        mbar_arrive_expect_tx(bar, P * ny * 4u + tbx + tby);   // the whole box, fill included
        tensor_load2(pl, map, 0, 0, bar);
        bulk_load(tx, tab + jb.tab_x, tbx, bar);
        bulk_load(ty, tab + jb.tab_y, tby, bar);
    }
    // the runs, if any cell secretes (the first one is then a voxel's: those
    // of non-secreting cells come last)
    uint32_t nruns = 0;
    if (a.run_word) {
        const uint64_t w = a.run_word[0];
        nruns = *a.n_runs;
        if (static_cast<uint32_t>(w >> kRunDensBits) != ii) nruns = 0;
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
    const bool faces = apply_faces && (jb.inst & kPlaneFaces) != 0;
    StagedRuns sr{};
    if (nruns) {
        sr.terms = reinterpret_cast<double*>(smem + 128) + stage_off;
        sr.cap = stage_cells;
        sr.start = reinterpret_cast<uint32_t*>(sr.terms + kStageTerms * static_cast<size_t>(stage_cells));
        sr.place = sr.start + stage_cells + 1;
        stage_runs(sr, reinterpret_cast<uint32_t*>(smem + 64), P, ii, jb.sub, nruns, a);
    }
    for (int step = 0; step < n_steps; ++step) {
        lane_lines<R, true>(pl, static_cast<int>(P), ny, rx, tx);
        __syncthreads();
        lane_lines<R, false>(pl, static_cast<int>(P), nx, ry, ty);
        __syncthreads();
        if (faces) {
            for (uint32_t j = threadIdx.x; j < ny; j += blockDim.x) {
                pl[j * P] = ry.T;
                pl[j * P + nx - 1] = ry.T;
            }
            __syncthreads();
        }
        if (nruns) {
            secrete_staged(pl, sr);
            __syncthreads();
        }
    }
    fence_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
        tensor_store2(map, 0, 0, pl);
        bulk_commit();
        bulk_wait_read<0>();   // shared memory may be released once the store has read it
    }
}

}  // namespace

size_t steps2d_smem(uint32_t floats, uint32_t stage_cells)
{
    const size_t plane = 128 + (static_cast<size_t>(floats) + 1) / 2 * 8;
    return stage_cells ? plane + (8 * kStageTerms + 8) * static_cast<size_t>(stage_cells) + 8 : plane;
}

using StepsKernel = void (*)(const PlaneJob*, const float*, const void*, RunArgs, int, int, uint32_t, uint32_t, unsigned*);

static StepsKernel steps2d_kernel(int cls) { return cls == 8 ? k_steps_2d<8> : cls == 16 ? k_steps_2d<16> : k_steps_2d<0>; }

cudaError_t steps2d_prepare(int cls) { return allow_max_smem(reinterpret_cast<const void*>(steps2d_kernel(cls))); }

cudaError_t launch_steps2d(cudaStream_t st, int cls, const PlaneJob* jobs, uint32_t njobs, const float* tab,
                           const void* tmaps, uint32_t floats, const RunArgs& a, int n_steps, int apply_faces,
                           uint32_t stage_cells, unsigned* status)
{
    if (njobs == 0 || n_steps <= 0) return cudaSuccess;
    return launch_chained(st, steps2d_kernel(cls), njobs, kSteps2dThreads, steps2d_smem(floats, stage_cells), jobs, tab,
                          tmaps, a, n_steps, apply_faces, stage_cells, (floats + 1) / 2, status);
}

}  // namespace pcg
