// Particle-to-mesh vorticity spreading (HFS/GPU_kernel.cu:218-294 with the
// nearest-grid-point weight of :31-50, then ComputeRHS :524-543 called with
// G = -1 at HFS/BiotSavartSolverImp.cpp:552-559).
//
// The reference gathers, for every grid cell, over the 5^3 hash cells around
// it and keeps the particles whose NGP cell is that cell.  Here the vortices
// are already sorted by hash cell, so a cell's particles are one contiguous
// run: a warp walks a cell's run with coalesced loads and reduces with a fixed
// xor-butterfly (deterministic, no atomics on the sums).  A particle whose FP64 NGP
// cell differs from its FP32 hash cell (a rounding tie at a cell face) has
// flagged its NGP cell; only flagged cells also walk their 26 neighbouring
// runs, which is the exact set the reference's 5^3 window can reach.
#include "pppm_internal.cuh"

namespace pppm {

namespace {

constexpr int kP2MThreads = 128;
constexpr int kP2MCells = 128;  // cells of a block

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void run_sum(const float4 *__restrict__ vrec, const float4 *__restrict__ valf,
                                        uint32_t s, uint32_t e, uint32_t cell, int lane, float &ax, float &ay,
                                        float &az) {
    // unrolled, and the strength loaded whether or not it counts, so that a
    // dense cell's loads are in flight together (each lane's records are still
    // added in order)
#pragma unroll 4
    for (uint32_t p = s + lane; p < e; p += 32) {
        const uint32_t at = __float_as_uint(vrec[p].w);
        const float4 a = valf[p];
        if (at == cell) {
            ax += a.x;
            ay += a.y;
            az += a.z;
        }
    }
}

// A block takes 128 consecutive cells.  Their runs differ widely (a ring fills
// a few thousand cells of two million, ten or more in a row, with hundreds of
// records each), so the block lists its non-empty cells and its warps take
// them in turn: with a warp for its own 32 cells the longest of them set the
// time.  1M ring at 128^3: 178 to 127 us; 262,144 points spread over 256^3,
// bound by the cell bounds and the six grids (134 MB + 400 MB), 152 and 157 us.
__global__ void __launch_bounds__(kP2MThreads)
p2m_kernel(const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
           const float4 *__restrict__ vrec, const float4 *__restrict__ valf, const uint32_t *__restrict__ mflag,
           uint32_t epoch, const DevParams *__restrict__ P, uint32_t n, float *__restrict__ vort,
           float *__restrict__ rhs) {
    __shared__ uint32_t cs[kP2MCells], ce[kP2MCells];
    __shared__ unsigned char list[kP2MCells], flist[kP2MCells];
    __shared__ int busy, flagged;
    __shared__ float sum[3][kP2MCells];
    const uint32_t C = n * n * n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t base = blockIdx.x * kP2MCells, cell = base + tid;
    const bool inb = tid < kP2MCells && cell < C;
    if (tid == 0) busy = flagged = 0;
    __syncthreads();
    const uint32_t s = inb ? start[cell] : kEmpty;
    const bool fl = inb && mflag[cell] == epoch;
    if (tid < kP2MCells) sum[0][tid] = sum[1][tid] = sum[2][tid] = 0.f;
    if (s != kEmpty) {
        cs[tid] = s;
        ce[tid] = end[cell];
        list[atomicAdd(&busy, 1)] = (unsigned char)tid;  // any order: each cell is summed by itself
    }
    if (fl) flist[atomicAdd(&flagged, 1)] = (unsigned char)tid;
    __syncthreads();
    for (int q = warp; q < busy; q += kP2MThreads / 32) {
        const int b = list[q];
        float ax = 0.f, ay = 0.f, az = 0.f;
        run_sum(vrec, valf, cs[b], ce[b], base + b, lane, ax, ay, az);
        ax = warp_sum(ax);
        ay = warp_sum(ay);
        az = warp_sum(az);
        if (lane == 0) {
            sum[0][b] = ax;
            sum[1][b] = ay;
            sum[2][b] = az;
        }
    }
    __syncthreads();
    for (int q = warp; q < flagged; q += kP2MThreads / 32) {
        const int b = flist[q];
        const uint32_t c = base + b;
        const int ci = (int)(c % n), cj = (int)((c / n) % n), ck = (int)(c / (n * n));
        float ax = 0.f, ay = 0.f, az = 0.f;
        for (int dk = -1; dk <= 1; dk++)
            for (int dj = -1; dj <= 1; dj++)
                for (int di = -1; di <= 1; di++) {
                    if (!di && !dj && !dk) continue;
                    const int ii = ci + di, jj = cj + dj, kk = ck + dk;
                    if (ii < 0 || jj < 0 || kk < 0 || ii >= (int)n || jj >= (int)n || kk >= (int)n) continue;
                    const uint32_t nb = ((uint32_t)kk * n + (uint32_t)jj) * n + (uint32_t)ii;
                    const uint32_t ns = start[nb];
                    if (ns == kEmpty) continue;
                    run_sum(vrec, valf, ns, end[nb], c, lane, ax, ay, az);
                }
        ax = warp_sum(ax);
        ay = warp_sum(ay);
        az = warp_sum(az);
        if (lane == 0) {
            sum[0][b] += ax;
            sum[1][b] += ay;
            sum[2][b] += az;
        }
    }
    __syncthreads();
    if (inb) {
        const float s3 = P->invh3_f, h2 = P->h2f;
        const float wx = sum[0][tid] * s3, wy = sum[1][tid] * s3, wz = sum[2][tid] * s3;
        vort[cell] = wx;
        vort[C + cell] = wy;
        vort[2 * (size_t)C + cell] = wz;
        rhs[cell] = -(wx * h2);
        rhs[C + cell] = -(wy * h2);
        rhs[2 * (size_t)C + cell] = -(wz * h2);
    }
}

}  // namespace

cudaError_t launch_p2m(pppm_scene *s) {
    const unsigned blocks = (s->C + kP2MCells - 1) / kP2MCells;
    ::pppm::note_launch();
    p2m_kernel<<<blocks, kP2MThreads, 0, s->stream>>>(s->cell_start, s->cell_end, s->vrec, s->valf, s->mflag,
                                                      s->epoch, s->dparams, s->n, s->vort, s->lv[0].b);
    return cudaGetLastError();
}

}  // namespace pppm
