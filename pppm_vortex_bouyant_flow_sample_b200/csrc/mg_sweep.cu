// A whole red-black sweep (both half sweeps) of a level in one pass over it.
//
// A pass over one colour streams x and b once and x back, 12 B a cell, so a
// sweep of two would move 24 B a cell, 1.2 GB at 256^3 with three components
// (HBM bounds the smoother there), and be two launches where the level lies in
// L2 (64^3, 128^3).  This kernel reads x and b once and writes x once for both.
//
// A CTA owns TY whole rows (in y) and a chunk of planes, and walks the chunk
// upwards.  A thread holds a group of 4 consecutive cells of two rows, for
// the planes around the current one, in registers.  At step z it updates the
// first colour (i + j + k odd) of plane z, then the second colour of plane
// z - 1, whose neighbours of the first colour are final by then, and stores
// that plane.  Neighbours along z are the thread's own; those along y and x
// come from the planes in shared memory, where a plane arrives by cp.async two
// steps before it is needed, takes its first colour in place and is read once
// more for the second, so that a step has one barrier and never waits for
// memory it has just asked for.  Which cells have the colour depends on z and
// the thread's row only, so the steps come in two kinds without a select.
// Measured on B200, three components: 106 us a sweep at 256^3 and 14.6 us at
// 128^3, against 188 us and 26.4 us for two passes of one colour each.  A 128^3
// solve holds 40 sweeps, 16 of them at 128^3 and 24 at 64^3.  The 30 that read x
// and add no correction take 314 us; with the loads in registers one step ahead
// they took 396 us, with a select per cell 332 us.  At 64^3 a sweep takes 4.4 to
// 5.7 us for about 1 us of data: its chunks are no thinner than 4 planes, each
// walks 4 more, and few blocks run.
// The rows and planes next to a CTA's own are updated by it too (the first
// colour: one row or plane each side, from values two away), which costs 4
// extra rows and 4 extra planes of reads but no exchange.  Since neighbours
// still read the old values, the result goes to the level's second copy of x.
//
// Each cell gets the terms of a pass over one colour in the same order, so the
// values are the same bit for bit (tests compare the blocked smoother's).
//
// The start of a smoothing can be folded into the reads: x = 0 (nothing is
// read or cleared), and the coarser level's correction added.  The end of a
// cycle can be folded into the writes: the result is added to the FP64 iterate
// and not stored.
//
// The same walk serves the corrected cycle (mg.cu): another relaxation factor,
// a diagonal that counts the cell's boundary faces, and the correction
// interpolated trilinearly instead of injected.
#include <algorithm>
#include <type_traits>

#include "pppm_internal.cuh"

namespace pppm {

namespace {

constexpr int kSweepThreads = 640;
constexpr int kRows = 2;      // rows of a thread
constexpr int kSweepTY = 16;  // rows of a CTA, at most
constexpr int kAhead = 2;     // planes asked for beyond the next one
constexpr int kXSlots = kAhead + 3, kBSlots = kAhead + 2;
static_assert(kRows == 2 && kAhead == 2, "the walk names its rows and slots");

struct SweepArgs {
    const float *x, *b, *xc;
    float *out;
    double *psi;
    int set_psi;
    int d, ty, zc;
    float inv0, inv1, inv2, inv3;  // corrected: 1 / diagonal by the number of boundary faces
    float gc;      // corrected: ghost factor of the coarser level
};

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// The group's 2 cells of a colour: ODD, ODD + 2.
template <bool CORR, bool ODD>
__device__ __forceinline__ float4 update_group(float4 v, float xl, float xr, const float4 up, const float4 dn,
                                               const float4 fr, const float4 bk, const float4 bb, float inv_lo,
                                               float inv_hi) {
    if (ODD) {
        const float lo = ((v.x + v.z) + (up.y + dn.y)) + (fr.y + bk.y);
        const float hi = ((v.z + xr) + (up.w + dn.w)) + (fr.w + bk.w);
        v.y = CORR ? mg_corr_update(v.y, lo, bb.y, inv_lo) : mg_sor_update(v.y, lo, bb.y);
        v.w = CORR ? mg_corr_update(v.w, hi, bb.w, inv_hi) : mg_sor_update(v.w, hi, bb.w);
    } else {
        const float lo = ((xl + v.y) + (up.x + dn.x)) + (fr.x + bk.x);
        const float hi = ((v.y + v.w) + (up.z + dn.z)) + (fr.z + bk.z);
        v.x = CORR ? mg_corr_update(v.x, lo, bb.x, inv_lo) : mg_sor_update(v.x, lo, bb.x);
        v.z = CORR ? mg_corr_update(v.z, hi, bb.z, inv_hi) : mg_sor_update(v.z, hi, bb.z);
    }
    return v;
}

__device__ __forceinline__ void copy16(float *to, const float *from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// LOADX: x is read (else it is zero); INJECT: plus the coarser level's xc, of
// the parent cell or (CORR) interpolated.
template <bool LOADX, bool INJECT, bool CORR>
__global__ void __launch_bounds__(kSweepThreads) sweep_kernel(const SweepArgs a) {
    extern __shared__ __align__(16) float sweep_smem[];
    const int d = a.d, q = d >> 2, rows = a.ty + 4, stride = d + 8, plane = rows * stride;
    const int g = (int)threadIdx.x % q, rr0 = ((int)threadIdx.x / q) * kRows;  // first of this thread's rows
    const int y0 = (int)blockIdx.x * a.ty - 2 + rr0;                           // its y
    const int zs = (int)blockIdx.y * a.zc, ze = min(zs + a.zc, d);
    const size_t dd = (size_t)d * d, cells = dd * d, comp = blockIdx.z;
    const float *x = a.x + comp * cells;
    const float *b = a.b + comp * cells;
    const int dc = d >> 1;
    const float *xc = INJECT ? a.xc + comp * (size_t)dc * dc * dc : nullptr;
    float *out = a.out + comp * cells;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);

    // the zero columns either side of each row, and the rows beyond the grid
    for (int q4 = (int)threadIdx.x; q4 < kXSlots * plane / 4; q4 += (int)blockDim.x)
        *reinterpret_cast<float4 *>(sweep_smem + 4 * q4) = z4;
    __syncthreads();

    bool in[kRows], red[kRows], own[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int rr = rr0 + r, y = y0 + r;
        in[r] = y >= 0 && y < d;
        red[r] = in[r] && rr >= 1 && rr <= a.ty + 2;
        own[r] = in[r] && rr >= 2 && rr <= a.ty + 1;
    }
    // the coarser level's correction at a group
    auto correction = [&](int r, int z) {
        float4 v = z4;
        if (INJECT && CORR) {
            // 3/4 of the parent and 1/4 of its neighbour on the cell's
            // side along each axis; beyond the grid the neighbour's value
            // is the parent's times the ghost factor
            const int y = y0 + r, cz = z >> 1, cy = y >> 1, cx = 2 * g;
            const int nz = cz + ((z & 1) ? 1 : -1), ny = cy + ((y & 1) ? 1 : -1);
            const bool oz = nz < 0 || nz >= dc, oy = ny < 0 || ny >= dc;
            const float wz[2] = {oz ? 0.75f + 0.25f * a.gc : 0.75f, oz ? 0.f : 0.25f};
            const float wy[2] = {oy ? 0.75f + 0.25f * a.gc : 0.75f, oy ? 0.f : 0.25f};
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;  // parents cx - 1 .. cx + 2
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int zz = (q & 2) ? (oz ? cz : nz) : cz, yy = (q & 1) ? (oy ? cy : ny) : cy;
                const float w = wz[q >> 1] * wy[q & 1];
                const float *row = xc + ((size_t)zz * dc + yy) * dc + cx;
                const float2 c = *reinterpret_cast<const float2 *>(row);
                s1 = fmaf(w, c.x, s1);
                s2 = fmaf(w, c.y, s2);
                s0 = fmaf(w, cx > 0 ? row[-1] : a.gc * c.x, s0);
                s3 = fmaf(w, cx + 2 < dc ? row[2] : a.gc * c.y, s3);
            }
            v.x += fmaf(0.25f, s0, 0.75f * s1);
            v.y += fmaf(0.25f, s2, 0.75f * s1);
            v.z += fmaf(0.25f, s1, 0.75f * s2);
            v.w += fmaf(0.25f, s3, 0.75f * s2);
        } else if (INJECT) {
            const float2 c = *reinterpret_cast<const float2 *>(
                xc + ((size_t)(z >> 1) * dc + ((y0 + r) >> 1)) * dc + 2 * g);
            v.x += c.x;
            v.y += c.x;
            v.z += c.y;
            v.w += c.y;
        }
        return v;
    };
    // This thread's first group in the slots of shared memory and in global
    // memory, as running positions: a step moves them on by one plane.
    const int at = rr0 * stride + 4 + 4 * g, bat = kXSlots * plane + rr0 * d + 4 * g, bplane = rows * d;
    int xm = at, x0 = at + plane, xp = at + 2 * plane, xq = at + 3 * plane, xf = at + 4 * plane;  // z - 1 .. z + 3
    int b0s = bat, b1s = bat + bplane, b2s = bat + 2 * bplane, b3s = bat + 3 * bplane;            // z .. z + 3
    const size_t cell0 = (size_t)(y0 < 0 ? 0 : y0) * d + 4 * g;  // (rows below the grid are never read)
    const int skip = y0 < 0 ? 0 : d;  // from the first row to the second
    // asks for plane z of x and b, at positions xs and bs
    auto fetch = [&](int z, int xs, int bs) {
        if (z >= 0 && z < d && z <= ze + 1) {
            const size_t c = (size_t)z * dd + cell0;
#pragma unroll
            for (int r = 0; r < kRows; r++) {
                if (LOADX && in[r]) copy16(sweep_smem + xs + r * stride, x + c + r * skip);
                if (red[r] && z <= ze) copy16(sweep_smem + bs + r * d, b + c + r * skip);
            }
        }
        copies_commit();
    };
    // plane z of x at position xs, its copies done: this thread's groups, the
    // correction added (and put back for the neighbours)
    auto arrive = [&](int z, int xs, float4 (&v)[kRows]) {
        const bool inside = z >= 0 && z < d;
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            v[r] = z4;
            if (!in[r] || !inside) continue;
            if (LOADX) v[r] = ld4(sweep_smem + xs + r * stride);
            if (INJECT) {
                const float4 c = correction(r, z);
                v[r].x += c.x;
                v[r].y += c.y;
                v[r].z += c.z;
                v[r].w += c.w;
            }
            if (INJECT || !LOADX) *reinterpret_cast<float4 *>(sweep_smem + xs + r * stride) = v[r];
        }
    };

    // planes z - 2 (final), z - 1 (first colour done), z and z + 1 (old)
    float4 pf[kRows], pm[kRows], p0[kRows], pp[kRows], bm[kRows];
    fetch(zs - 1, x0, b0s);
    fetch(zs, xp, b1s);
    fetch(zs + 1, xq, b2s);
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        pf[r] = bm[r] = pm[r] = z4;
        if (in[r] && zs >= 2) {
            if (LOADX) pm[r] = ld4(x + (size_t)(zs - 2) * dd + (size_t)(y0 + r) * d + 4 * g);
            if (INJECT) {
                const float4 c = correction(r, zs - 2);
                pm[r].x += c.x;
                pm[r].y += c.y;
                pm[r].z += c.z;
                pm[r].w += c.w;
            }
        }
    }
    copies_wait<kAhead>();
    arrive(zs - 1, x0, p0);

    auto step = [&](auto parity, int z) {
        constexpr int ZP = decltype(parity)::value;  // z & 1; y0 is even
        copies_wait<kAhead - 1>();
        arrive(z + 1, xp, pp);
        __syncthreads();
        fetch(z + 1 + kAhead, xf, b3s);
        const float *sa = sweep_smem + x0, *sb = sweep_smem + xm, *bs = sweep_smem + b0s;
        float4 b0[kRows] = {z4, z4};
        auto inverse = [&](int r, int zz, bool odd, float &lo, float &hi) {
            const int y = y0 + r, f = (y == 0) + (y == d - 1) + (zz == 0) + (zz == d - 1);
            const float i0 = f == 0 ? a.inv0 : (f == 1 ? a.inv1 : a.inv2), i1 = f == 0 ? a.inv1 : (f == 1 ? a.inv2 : a.inv3);
            lo = (g == 0 && !odd) ? i1 : i0;
            hi = (g == q - 1 && odd) ? i1 : i0;
        };
        auto one = [&](auto rc, const float4 (&v)[kRows], const float *rows_at, const float4 fr, const float4 bk,
                       const float4 bb, auto oddc, int zz) {
            constexpr int r = decltype(rc)::value;
            constexpr bool odd = decltype(oddc)::value;
            const float *row = rows_at + r * stride;
            const float4 up = r + 1 < kRows ? v[r + 1 < kRows ? r + 1 : r] : ld4(row + stride);
            const float4 dn = r > 0 ? v[r > 0 ? r - 1 : r] : ld4(row - stride);
            float lo = 0.f, hi = 0.f;
            if (CORR) inverse(r, zz, odd, lo, hi);
            return update_group<CORR, odd>(v[r], odd ? 0.f : row[-1], odd ? row[4] : 0.f, up, dn, fr, bk, bb, lo, hi);
        };
        if (z >= 0 && z < d) {
            float4 nw[kRows];
            auto first = [&](auto rc) {
                constexpr int r = decltype(rc)::value;
                nw[r] = p0[r];
                b0[r] = z4;
                if (red[r]) {
                    b0[r] = ld4(bs + r * d);
                    nw[r] = one(rc, p0, sa, pm[r], pp[r], b0[r],
                                std::integral_constant<bool, ((r + ZP + 1) & 1) != 0>{}, z);
                }
            };
            first(std::integral_constant<int, 0>{});
            first(std::integral_constant<int, 1>{});
#pragma unroll
            for (int r = 0; r < kRows; r++) {
                p0[r] = nw[r];
                if (red[r]) *reinterpret_cast<float4 *>(sweep_smem + x0 + r * stride) = nw[r];
            }
        }
        if (z > zs) {
            float4 nw[kRows];
            auto second = [&](auto rc) {
                constexpr int r = decltype(rc)::value;
                nw[r] = pm[r];
                if (!own[r]) return;
                nw[r] = one(rc, pm, sb, pf[r], p0[r], bm[r], std::integral_constant<bool, ((r + ZP + 1) & 1) != 0>{},
                            z - 1);
                const size_t c = (size_t)(z - 1) * dd + cell0 + r * skip;
                if (a.psi) {
                    double2 *to = reinterpret_cast<double2 *>(a.psi + comp * cells + c);
                    double2 u = make_double2(0.0, 0.0), w = u;
                    if (!a.set_psi) {
                        u = to[0];
                        w = to[1];
                    }
                    to[0] = make_double2(u.x + (double)nw[r].x, u.y + (double)nw[r].y);
                    to[1] = make_double2(w.x + (double)nw[r].z, w.y + (double)nw[r].w);
                } else {
                    *reinterpret_cast<float4 *>(out + c) = nw[r];
                }
            };
            second(std::integral_constant<int, 0>{});
            second(std::integral_constant<int, 1>{});
#pragma unroll
            for (int r = 0; r < kRows; r++) pm[r] = nw[r];
        }
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            pf[r] = pm[r];
            pm[r] = p0[r];
            p0[r] = pp[r];
            bm[r] = b0[r];
        }
        const int xo = xf, bo = b0s;
        xf = xm;
        xm = x0;
        x0 = xp;
        xp = xq;
        xq = xo;
        b0s = b1s;
        b1s = b2s;
        b2s = b3s;
        b3s = bo;
    };
    int z = zs - 1;
    if (z & 1) step(std::integral_constant<int, 1>{}, z++);
    for (; z + 1 <= ze; z += 2) {
        step(std::integral_constant<int, 0>{}, z);
        step(std::integral_constant<int, 1>{}, z + 1);
    }
    if (z <= ze) step(std::integral_constant<int, 0>{}, z);
    copies_wait<0>();
}

}  // namespace

// Rows of a CTA for a level of edge d (a multiple of 8): 16, or as many as
// its threads allow.
static int sweep_rows(int d) {
    const int q = d / 4;
    return std::min(kSweepTY, std::max(2, kRows * (kSweepThreads / q) - 4));
}

static size_t sweep_bytes(int d, int ty) {
    return sizeof(float) * (size_t)(ty + 4) * (kXSlots * (d + 8) + kBSlots * d);
}

cudaError_t mg_sweep_prepare() {
    size_t most = 0;
    for (int d = 40; d <= 512; d += 8) most = std::max(most, sweep_bytes(d, sweep_rows(d)));
    const void *k[] = {(const void *)sweep_kernel<true, false, false>, (const void *)sweep_kernel<true, true, false>,
                       (const void *)sweep_kernel<false, true, false>, (const void *)sweep_kernel<false, false, false>,
                       (const void *)sweep_kernel<true, false, true>, (const void *)sweep_kernel<true, true, true>,
                       (const void *)sweep_kernel<false, false, true>};
    for (const void *f : k) PPPM_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    return cudaSuccess;
}

// One sweep of a level of edge d > 32 (such an edge is a multiple of 8).
cudaError_t mg_sweep(const SweepSpec &sp, cudaStream_t st) {
    const int d = sp.d, comps = sp.comps;
    SweepArgs a;
    a.x = sp.x;
    a.b = sp.b;
    a.xc = sp.xc;
    a.out = sp.out;
    a.psi = sp.psi;
    a.set_psi = sp.set_psi ? 1 : 0;
    a.gc = 0.f;
    a.inv0 = a.inv1 = a.inv2 = a.inv3 = 0.f;
    if (sp.corrected >= 0) {
        const float gh = mg_ghost_factor(sp.corrected);
        a.inv0 = 1.0f / 6.0f;
        a.inv1 = 1.0f / (6.0f - gh);
        a.inv2 = 1.0f / (6.0f - 2.0f * gh);
        a.inv3 = 1.0f / (6.0f - 3.0f * gh);
        a.gc = mg_ghost_factor(sp.corrected + 1);
    }
    a.d = d;
    a.ty = sweep_rows(d);
    const int threads = (a.ty + 4) / kRows * (d / 4);
    const size_t smem = sweep_bytes(d, a.ty);
    // chunks of planes: fill the resident CTAs in whole waves, each chunk
    // paying 4 planes more than its own
    const int per_sm = std::max(1, std::min({2048 / threads, 65536 / (96 * threads), (int)(227 * 1024 / (smem + 1024))}));
    const int tiles = (d + a.ty - 1) / a.ty * comps, slots = kSMs * per_sm;
    int best = 1;
    long cost = -1;
    for (int c = 1; c <= d / 4; c++) {
        const long len = (d + c - 1) / c, t = (long)((tiles * c + slots - 1) / slots) * (len + 4);
        if (cost < 0 || t < cost) {
            cost = t;
            best = c;
        }
    }
    a.zc = (d + best - 1) / best;
    const dim3 grid((d + a.ty - 1) / a.ty, (d + a.zc - 1) / a.zc, comps);
    ::pppm::note_launch();
    auto *k = sp.corrected >= 0 ? (sp.x ? (sp.xc ? sweep_kernel<true, true, true> : sweep_kernel<true, false, true>)
                                        : sweep_kernel<false, false, true>)
                                : (sp.x ? (sp.xc ? sweep_kernel<true, true, false> : sweep_kernel<true, false, false>)
                                        : (sp.xc ? sweep_kernel<false, true, false> : sweep_kernel<false, false, false>));
    k<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace pppm
