// A whole red-black sweep (both half sweeps) of a level in one pass over it.
//
// A half sweep by itself streams x and b once and x back, 12 B a cell, so a
// sweep of two moves 24 B a cell: 1.2 GB at 256^3 with three components, which
// is what bounds the smoother there, and at 64^3 and 128^3 (in L2) two
// launches.  This kernel reads x and b once and writes x once for the two.
//
// A CTA owns TY whole rows (in y) and a chunk of planes, and walks the chunk
// upwards.  A thread holds a group of 4 consecutive cells of two rows, for
// the planes around the current one, in registers.  At step z it updates the
// first colour (i + j + k odd) of plane z, then the second colour of plane
// z - 1, whose neighbours of the first colour are final by then, and stores
// that plane.  Neighbours along z are the thread's own; those along y and x
// come from two planes in shared memory, the old plane z and plane z - 1 after
// its first colour, in alternating buffers, so that a step has one barrier.
// The rows and planes next to a CTA's own are updated by it too (the first
// colour: one row or plane each side, from values two away), which costs 4
// extra rows and 4 extra planes of reads but no exchange.  Since neighbours
// still read the old values, the result goes to the level's second copy of x.
//
// Each cell gets the terms of the one-colour kernel in its order, so the
// values are the same bit for bit.
//
// The start of a smoothing can be folded into the reads: x = 0 (nothing is
// read or cleared), and the coarser level's correction injected.
#include <algorithm>

#include "pppm_internal.cuh"

namespace pppm {

namespace {

constexpr int kSweepThreads = 640;
constexpr int kRows = 2;      // rows of a thread
constexpr int kSweepTY = 16;  // rows of a CTA, at most

struct SweepArgs {
    const float *x, *b, *xc;
    float *out;
    int d, ty, zc;
};

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// The group's 2 cells of a colour: first + 2 e + odd with e = 0, 1.
__device__ __forceinline__ float4 update_group(float4 v, float xl, float xr, const float4 up, const float4 dn,
                                               const float4 fr, const float4 bk, const float4 bb, bool odd) {
    const float nb_lo = (((odd ? v.x : xl) + (odd ? v.z : v.y)) + ((odd ? up.y : up.x) + (odd ? dn.y : dn.x))) +
                        ((odd ? fr.y : fr.x) + (odd ? bk.y : bk.x));
    const float nb_hi = (((odd ? v.z : v.y) + (odd ? xr : v.w)) + ((odd ? up.w : up.z) + (odd ? dn.w : dn.z))) +
                        ((odd ? fr.w : fr.z) + (odd ? bk.w : bk.z));
    const float lo = mg_sor_update(odd ? v.y : v.x, nb_lo, odd ? bb.y : bb.x);
    const float hi = mg_sor_update(odd ? v.w : v.z, nb_hi, odd ? bb.w : bb.z);
    if (odd) {
        v.y = lo;
        v.w = hi;
    } else {
        v.x = lo;
        v.z = hi;
    }
    return v;
}

// LOADX: x is read (else it is zero); INJECT: plus the coarser level's xc of
// the parent cell.
template <bool LOADX, bool INJECT>
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

    // the zero columns either side of each row of the four planes
    for (int r = (int)threadIdx.x; r < 4 * rows; r += (int)blockDim.x) {
        *reinterpret_cast<float4 *>(sweep_smem + r * stride) = z4;
        *reinterpret_cast<float4 *>(sweep_smem + r * stride + 4 + d) = z4;
    }

    bool in[kRows], red[kRows], own[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int rr = rr0 + r, y = y0 + r;
        in[r] = y >= 0 && y < d;
        red[r] = in[r] && rr >= 1 && rr <= a.ty + 2;
        own[r] = in[r] && rr >= 2 && rr <= a.ty + 1;
    }
    auto load_x = [&](int r, int z) {
        float4 v = z4;
        if (in[r] && z >= 0 && z < d) {
            if (LOADX) v = ld4(x + (size_t)z * dd + (size_t)(y0 + r) * d + 4 * g);
            if (INJECT) {
                const float2 c = *reinterpret_cast<const float2 *>(
                    xc + ((size_t)(z >> 1) * dc + ((y0 + r) >> 1)) * dc + 2 * g);
                v.x += c.x;
                v.y += c.x;
                v.z += c.y;
                v.w += c.y;
            }
        }
        return v;
    };
    auto load_b = [&](int r, int z) {
        return red[r] && z >= 0 && z < d ? ld4(b + (size_t)z * dd + (size_t)(y0 + r) * d + 4 * g) : z4;
    };

    // planes z - 2 (final), z - 1 (first colour done), z and z + 1 (old)
    float4 pf[kRows], pm[kRows], p0[kRows], pp[kRows], bm[kRows], b0[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        pf[r] = z4;
        bm[r] = z4;
        pm[r] = load_x(r, zs - 2);
        p0[r] = load_x(r, zs - 1);
        pp[r] = load_x(r, zs);
        b0[r] = load_b(r, zs - 1);
    }
    const int at = rr0 * stride + 4 + 4 * g;  // this thread's group in a shared plane
    for (int z = zs - 1; z <= ze; z++) {
        float4 nx[kRows], nb[kRows];
#pragma unroll
        for (int r = 0; r < kRows; r++) {  // the next step's planes, in flight meanwhile
            nx[r] = z < ze ? load_x(r, z + 2) : z4;
            nb[r] = z < ze ? load_b(r, z + 1) : z4;
        }
        float *sa = sweep_smem + ((z & 1) ? 2 * plane : 0), *sb = sa + plane;
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            *reinterpret_cast<float4 *>(sa + at + r * stride) = p0[r];
            *reinterpret_cast<float4 *>(sb + at + r * stride) = pm[r];
        }
        __syncthreads();
        if (z >= 0 && z < d) {
            float4 old[kRows];
#pragma unroll
            for (int r = 0; r < kRows; r++) old[r] = p0[r];
#pragma unroll
            for (int r = 0; r < kRows; r++) {
                if (!red[r]) continue;
                const float *row = sa + at + r * stride;
                const float4 up = r + 1 < kRows ? old[r + 1 < kRows ? r + 1 : r] : ld4(row + stride);
                const float4 dn = r > 0 ? old[r > 0 ? r - 1 : r] : ld4(row - stride);
                p0[r] = update_group(old[r], row[-1], row[4], up, dn, pm[r], pp[r], b0[r],
                                     ((y0 + r + z + 1) & 1) != 0);
            }
        }
        if (z > zs) {
            float4 half[kRows];
#pragma unroll
            for (int r = 0; r < kRows; r++) half[r] = pm[r];
#pragma unroll
            for (int r = 0; r < kRows; r++) {
                if (!own[r]) continue;
                const float *row = sb + at + r * stride;
                const float4 up = r + 1 < kRows ? half[r + 1 < kRows ? r + 1 : r] : ld4(row + stride);
                const float4 dn = r > 0 ? half[r > 0 ? r - 1 : r] : ld4(row - stride);
                pm[r] = update_group(half[r], row[-1], row[4], up, dn, pf[r], p0[r], bm[r],
                                     ((y0 + r + z - 1) & 1) != 0);
                *reinterpret_cast<float4 *>(out + (size_t)(z - 1) * dd + (size_t)(y0 + r) * d + 4 * g) = pm[r];
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            pf[r] = pm[r];
            pm[r] = p0[r];
            p0[r] = pp[r];
            pp[r] = nx[r];
            bm[r] = b0[r];
            b0[r] = nb[r];
        }
    }
}

}  // namespace

// Rows of a CTA for a level of edge d (a multiple of 8): 16, or as many as
// its threads allow.
static int sweep_rows(int d) {
    const int q = d / 4;
    return std::min(kSweepTY, std::max(2, kRows * (kSweepThreads / q) - 4));
}

static size_t sweep_bytes(int d, int ty) { return sizeof(float) * 4 * (size_t)(ty + 4) * (d + 8); }

cudaError_t mg_sweep_prepare() {
    size_t most = 0;
    for (int d = 40; d <= 512; d += 8) most = std::max(most, sweep_bytes(d, sweep_rows(d)));
    PPPM_CUDA_TRY(cudaFuncSetAttribute(sweep_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    PPPM_CUDA_TRY(cudaFuncSetAttribute(sweep_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    PPPM_CUDA_TRY(cudaFuncSetAttribute(sweep_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    return cudaFuncSetAttribute(sweep_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// One sweep of a level of edge d > 32 (such an edge is a multiple of 8):
// out = sweep(x + injected xc); x null: from zero; xc may be null.
cudaError_t mg_sweep(const float *x, const float *b, const float *xc, float *out, int d, int comps, cudaStream_t st) {
    SweepArgs a;
    a.x = x;
    a.b = b;
    a.xc = xc;
    a.out = out;
    a.d = d;
    a.ty = sweep_rows(d);
    const int threads = (a.ty + 4) / kRows * (d / 4);
    const size_t smem = sweep_bytes(d, a.ty);
    // chunks of planes: fill the resident CTAs in whole waves, each chunk
    // paying 4 planes more than its own
    const int per_sm = std::max(1, std::min({2048 / threads, 65536 / (104 * threads), (int)(227 * 1024 / (smem + 1024))}));
    const int tiles = (d + a.ty - 1) / a.ty * comps, slots = 148 * per_sm;
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
    if (x && xc) sweep_kernel<true, true><<<grid, threads, smem, st>>>(a);
    else if (x) sweep_kernel<true, false><<<grid, threads, smem, st>>>(a);
    else if (xc) sweep_kernel<false, true><<<grid, threads, smem, st>>>(a);
    else sweep_kernel<false, false><<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace pppm
