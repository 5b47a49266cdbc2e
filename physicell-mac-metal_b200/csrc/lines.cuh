// lines.cuh — device helpers shared by the kernels that solve Thomas lines in
// shared memory: tensor copies with their bounded waits, and the solve of one
// line from both ends.
#pragma once

#include "pcg_kernels.cuh"

namespace pcg {

// ------------------------------------------------------------------ TMA / mbarrier helpers

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// One bounded try: the thread may be suspended for up to kSuspendNs while
// the phase is incomplete, so a waiting warp does not spin on the issue
// slots of the warps that are computing.
constexpr uint32_t kSuspendNs = 20000;

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return done != 0;
}

// Bounded wait: about one second of SM clock, then PCG_DEV_TIMEOUT.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned* status)
{
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > (2ll << 30)) {
            atomicOr(status, PCG_DEV_TIMEOUT);
            return false;
        }
    }
    return true;
}

// global -> shared, completion counted on 'bar' (16-byte aligned, size % 16 == 0)
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// 3-D tensor-map copies of a whole column tile (one instruction each way)
__device__ __forceinline__ void tensor_load3(void* smem_dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}
// 2-D tensor-map copies of a whole x tile
__device__ __forceinline__ void tensor_load2(void* smem_dst, const void* tmap, int c0, int c1, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(smem_dst)),
        "l"(tmap), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}
// L2 prefetch of a tensor box (no shared memory, no barrier): the box a
// later CTA will load then comes from L2.
__device__ __forceinline__ void tensor_prefetch2(const void* tmap, int c0, int c1)
{
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tmap), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void tensor_prefetch3(const void* tmap, int c0, int c1, int c2)
{
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(tmap), "r"(c0), "r"(c1),
                 "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void tensor_store2(const void* tmap, int c0, int c1, const void* smem_src)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(tmap), "r"(c0),
                 "r"(c1), "r"(smem_u32(smem_src))
                 : "memory");
}
__device__ __forceinline__ void tensor_store3(const void* tmap, int c0, int c1, int c2, const void* smem_src)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(tmap),
                 "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(smem_src))
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ------------------------------------------------------------------ solves in shared memory

// Coefficient table of one rule, staged in shared memory next to its lines
// (layout: SplitTable).  A half's chunk k holds the coefficients of its 4
// positions in the order the half is walked in, {g[4], inv[4]} (32-byte
// aligned), g_i = c / den_i, inv_i = 1 / den_i; zero at the end node and past
// the line.
__device__ __forceinline__ float tab_g(const float* t, int i) { return t[((i >> 2) << 3) + (i & 3)]; }
__device__ __forceinline__ float tab_inv(const float* t, int i) { return t[((i >> 2) << 3) + 4 + (i & 3)]; }
__device__ __forceinline__ float4 tab_g4(const float* t, int q) { return *reinterpret_cast<const float4*>(t + (q << 3)); }
__device__ __forceinline__ float4 tab_inv4(const float* t, int q)
{
    return *reinterpret_cast<const float4*>(t + (q << 3) + 4);
}

// One chunk of the forward / backward pass, in walking order.
__device__ __forceinline__ float fwd1(float g, float iv, float d, float& v)
{
    d = fmaf(g, d, v * iv);
    v = d;
    return d;
}
__device__ __forceinline__ float bwd1(float g, float x, float& v)
{
    x = fmaf(g, x, v);
    v = x;
    return x;
}
__device__ __forceinline__ float fwd4(float4& v, float4 g, float4 iv, float d)
{
    d = fwd1(g.x, iv.x, d, v.x);
    d = fwd1(g.y, iv.y, d, v.y);
    d = fwd1(g.z, iv.z, d, v.z);
    return fwd1(g.w, iv.w, d, v.w);
}
__device__ __forceinline__ float bwd4(float4& v, float4 g, float x)
{
    x = bwd1(g.w, x, v.w);
    x = bwd1(g.z, x, v.z);
    x = bwd1(g.y, x, v.y);
    return bwd1(g.x, x, v.x);
}
__device__ __forceinline__ float4 reversed(float4 v) { return make_float4(v.w, v.z, v.y, v.x); }

// The end node of a half leaves its first chunk (with what lies before it,
// 'lead' places past the line) and the first interior node takes the fold,
// unless it lies in the next chunk (lead == 3).  Returns the end node.
__device__ __forceinline__ float take_end(float4& a, int lead, float fold)
{
    const float end = lead == 0 ? a.x : lead == 1 ? a.y : lead == 2 ? a.z : a.w;
    a.x = 0.f;
    a.y = lead == 0 ? a.y + fold : 0.f;
    a.z = lead == 0 ? a.z : lead == 1 ? a.z + fold : 0.f;
    a.w = lead <= 1 ? a.w : lead == 2 ? a.w + fold : 0.f;
    return end;
}
__device__ __forceinline__ void put_end(float4& a, int lead, float end)
{
    if (lead == 0) a.x = end;
    else if (lead == 1) a.y = end;
    else if (lead == 2) a.z = end;
    else a.w = end;
}

// Both halves of one line by one thread, in shared memory, over positions
// 1..n-2 (n >= 3): ld(q) returns chunk q (positions 4q..4q+3), st(q, v)
// writes it back; the end nodes keep their values.  The left half is the
// first SplitTable(n).hl chunks.  Each pass takes a chunk of either half at
// a time, the next ones loaded while the current ones' chains run.
template <class LD, class ST>
__device__ __forceinline__ void split_line(const float* t, int n, float fold, LD ld, ST st)
{
    const SplitTable sp(n);
    const int nq = sp.nq, hl = sp.hl, hr = nq - hl;
    const float* tr = t + sp.right();
    if (!sp.right_has_interior()) {   // n = 3, 4, 5 or 9: the left half alone
        float4 c0 = ld(0), c1 = hl > 1 ? ld(1) : make_float4(0.f, 0.f, 0.f, 0.f);
        float a[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        float d = 0.f, x = 0.f;
#pragma unroll
        for (int i = 1; i < 8; ++i)
            if (i <= n - 2) {
                if (i == 1 || i == n - 2) a[i] += fold;
                d = fwd1(tab_g(t, i), tab_inv(t, i), d, a[i]);
            }
#pragma unroll
        for (int i = 7; i >= 1; --i)
            if (i <= n - 2) x = bwd1(tab_g(t, i), x, a[i]);
        st(0, make_float4(a[0], a[1], a[2], a[3]));
        if (hl > 1) st(1, make_float4(a[4], a[5], a[6], a[7]));
        return;
    }
    const int lead = 4 * nq - n;
    const float fold1 = lead == 3 ? fold : 0.f;
    const float* tj = t + sp.middle();
    const int kc = min(__float_as_int(tj[3]), hr);   // chunks [kc, ..) of both halves: one g, one inv
    float4 a = ld(0), b = reversed(ld(nq - 1));
    const float4 b0 = b;
    float4 gl = tab_g4(t, 0), il = tab_inv4(t, 0), gr = tab_g4(tr, 0), ir = tab_inv4(tr, 0);
    const float lo = take_end(a, 0, fold);
    take_end(b, lead, fold);
    float dl = 0.f, dr = 0.f;
    int k = 0;
    for (; k < kc && k + 1 < hr; ++k) {
        const float4 an = ld(k + 1), gln = tab_g4(t, k + 1), iln = tab_inv4(t, k + 1);
        float4 bn = reversed(ld(nq - 2 - k));
        const float4 grn = tab_g4(tr, k + 1), irn = tab_inv4(tr, k + 1);
        if (k == 0) bn.x += fold1;
        dl = fwd4(a, gl, il, dl);
        dr = fwd4(b, gr, ir, dr);
        st(k, a);
        st(nq - 1 - k, reversed(b));
        a = an;
        b = bn;
        gl = gln;
        il = iln;
        gr = grn;
        ir = irn;
    }
    for (; k + 1 < hr; ++k) {   // gl, il: the constants from here on
        const float4 an = ld(k + 1), bn = reversed(ld(nq - 2 - k));
        dl = fwd4(a, gl, il, dl);
        dr = fwd4(b, gl, il, dr);
        st(k, a);
        st(nq - 1 - k, reversed(b));
        a = an;
        b = bn;
    }
    // the innermost chunks stay in registers
    dl = fwd4(a, gl, il, dl);
    dr = fwd4(b, gr, ir, dr);
    float4 g = gl;
    if (hl > hr) {
        const float4 an = ld(hr);
        st(hr - 1, a);
        a = an;
        g = tab_g4(t, hr);
        dl = fwd4(a, g, tab_inv4(t, hr), dl);
    }
    float xl = fmaf(tj[1], dl, dr) * tj[2];   // the right half's first value, from both sides
    float xr = fmaf(tj[0], dr, dl) * tj[2];   // the left half's last
    if (hl > hr) {
        const float4 an = ld(hr - 1);
        xl = bwd4(a, g, xl);
        st(hr, a);
        a = an;
    }
    k = hr - 1;
    for (; k > 0 && k >= kc; --k) {
        const float4 an = ld(k - 1), bn = reversed(ld(nq - k));
        xl = bwd4(a, gl, xl);
        xr = bwd4(b, gl, xr);
        st(k, a);
        st(nq - 1 - k, reversed(b));
        a = an;
        b = bn;
    }
    gl = tab_g4(t, k);
    gr = tab_g4(tr, k);
    for (; k > 0; --k) {
        const float4 an = ld(k - 1), bn = reversed(ld(nq - k)), gln = tab_g4(t, k - 1), grn = tab_g4(tr, k - 1);
        xl = bwd4(a, gl, xl);
        xr = bwd4(b, gr, xr);
        st(k, a);
        st(nq - 1 - k, reversed(b));
        a = an;
        b = bn;
        gl = gln;
        gr = grn;
    }
    bwd4(a, gl, xl);
    bwd4(b, gr, xr);
    a.x = lo;
    b.x = b0.x;   // the places up to the end node as they were
    b.y = lead >= 1 ? b0.y : b.y;
    b.z = lead >= 2 ? b0.z : b.z;
    b.w = lead == 3 ? b0.w : b.w;
    st(0, a);
    st(nq - 1, reversed(b));
}

// x tile through the row tensor map: lane t solves line t stored at
// st + t * P, P = row_smem_pitch(n).  All lanes sit at the same position, so
// the coefficients are one broadcast load, and each lane moves 4 values with
// one 16-byte shared access; P / 4 is odd, so the 8 lanes of each quarter
// warp hit 8 different 16-byte bank groups (no conflicts).
__device__ __forceinline__ void row_line(float* row, const LineRule& r, const float* t)
{
    const int n = static_cast<int>(r.n);
    if (n >= 3)
        split_line(
            t, n, r.fold, [row](int q) { return *reinterpret_cast<const float4*>(row + 4 * q); },
            [row](int q, float4 v) { *reinterpret_cast<float4*>(row + 4 * q) = v; });
    if (r.dir) {
        row[0] = r.T;
        row[n - 1] = r.T;
    }
}

// Column line of a plane in shared memory (rows P floats apart): the steps
// of solve_cols with row stride P.
__device__ __forceinline__ void plane_col(float* c, int P, const LineRule& r, const float* t)
{
    const int n = static_cast<int>(r.n);
    if (n >= 3)
        split_line(
            t, n, r.fold,
            [c, P](int q) {
                const float* p = c + 4 * q * P;
                return make_float4(p[0], p[P], p[2 * P], p[3 * P]);
            },
            [c, P](int q, float4 v) {
                float* p = c + 4 * q * P;
                p[0] = v.x;
                p[P] = v.y;
                p[2 * P] = v.z;
                p[3 * P] = v.w;
            });
    if (r.dir) {
        c[0] = r.T;
        c[(n - 1) * P] = r.T;
    }
}

}  // namespace pcg
