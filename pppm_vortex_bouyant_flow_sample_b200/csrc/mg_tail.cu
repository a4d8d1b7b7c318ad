// The small levels of the multigrid in one launch.
//
// A V-cycle visits every level of edge <= 32 with a handful of short kernels
// (eight half sweeps, a restriction and a prolongation each way, the coarsest
// solve).  Each of those moves at most 0.4 MB, so it lasts as long as a launch
// does (1.5 to 2 us inside a graph) whatever it computes, and a full multigrid
// solve holds about 150 of them.  Here one thread-block cluster of 8 CTAs per
// component keeps those levels in shared memory and runs the whole cycle (or
// the whole full multigrid) over them:
//   A  the level with 16 < edge <= 32, in slabs of 4 planes, one per CTA.
//      After a half sweep a CTA stores the planes next to its neighbours'
//      into their halo planes (distributed shared memory), then the cluster
//      synchronises.
//   B  the level with 8 < edge <= 16, in CTA 0 alone: a block barrier costs
//      less than a cluster barrier there.
//   C  the coarsest level (edge <= 8), in CTA 0.  Its solve is a fixed linear
//      map that a separable eigenbasis diagonalises: three 1-D transforms of
//      at most 8 points, one factor per mode, three transforms back, in FP64.
//      The reference schedule's 100 Jacobi sweeps from zero are the factor
//      -(1 - mu^100) / (6 (1 - mu)) with mu the mode's eigenvalue of the
//      sweep (sine modes); the stored 512 x 512 operator that the one-level
//      kernels apply would have to be read by one CTA, 2 MB of it.
// Edges: the levels halve, every level above the coarsest is even, and the
// coarsest is the first with at most 512 cells, so a hierarchy has at most
// one level of each kind; grids of edge 9 to 16 start at B.
//
// Sums are taken in the order of the one-level kernels, so A and B hold the
// same values bit for bit; the coarsest solve agrees with the stored operator
// to FP64 rounding.
#include <cooperative_groups.h>

#include <cmath>

#include "pppm_internal.cuh"

namespace cg = cooperative_groups;

namespace pppm {

namespace {

constexpr int kTailThreads = 512;
constexpr int kTailCtas = 8;
constexpr int kSlab = 4;      // planes of level A per CTA
constexpr int kMaxA = 32, kMaxB = 16, kMaxC = 8;
constexpr int kItems = kSlab * kMaxA * kMaxA / 2 / kTailThreads;  // cell pairs of A per thread
constexpr int kItemsB = kMaxB * kMaxB * kMaxB / 2 / kTailThreads;  // cell pairs of B per thread

struct TailShared {
    float xa[(kSlab + 2) * (kMaxA + 2) * (kMaxA + 2)];  // with halo planes and a zero border
    float ba[kSlab * kMaxA * kMaxA];
    float xb[(kMaxB + 2) * (kMaxB + 2) * (kMaxB + 2)];
    float bb[kMaxB * kMaxB * kMaxB];
    float xc[(kMaxC + 2) * (kMaxC + 2) * (kMaxC + 2)];
    float bc[kMaxC * kMaxC * kMaxC];
    double t0[kMaxC * kMaxC * kMaxC], t1[kMaxC * kMaxC * kMaxC];
    double q[kMaxC * kMaxC];
};

// A cell pair (2 ih, 2 ih + 1) of row (j, z): offset into the padded x, the
// parity of j + z, and (level A) whether its plane is a neighbour's halo.
struct Pair {
    int off;
    int par;
    bool on, first, last;
};

__device__ __forceinline__ float nb6(const float *__restrict__ x, int o, int P) {
    return ((x[o - 1] + x[o + 1]) + (x[o + P] + x[o - P])) + (x[o - P * P] + x[o + P * P]);
}

// b restricted to the coarse cell whose first child sits at padded offset o
// of x and at ob of b: 0.5 * sum of the children's residuals (of b itself
// when x is zero), in the one-level kernels' order.
__device__ __forceinline__ float restrict8(const float *__restrict__ x, const float *__restrict__ b, int o, int ob,
                                           int d, bool x_zero) {
    const int P = d + 2;
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int c = o + (q & 1) + ((q >> 1) & 1) * P + (q >> 2) * P * P;
        float r = b[ob + (q & 1) + ((q >> 1) & 1) * d + (q >> 2) * d * d];
        if (!x_zero) r -= nb6(x, c, P) - 6.f * x[c];
        sum += r;
    }
    return sum * 0.5f;
}

// x_C = the coarsest solve of b_C (all threads; edge d).
__device__ void coarse_modes(TailShared &S, int d, double factor, int tid) {
    const int cells = d * d * d;
    const int i = tid % d, j = (tid / d) % d, k = tid / (d * d);
    const bool on = tid < cells;
    if (on) S.t0[tid] = (double)S.bc[tid];
    __syncthreads();
    double *src = S.t0, *dst = S.t1;
#pragma unroll
    for (int pass = 0; pass < 6; pass++) {
        const int axis = pass % 3;
        if (on) {
            const int st = axis == 0 ? 1 : (axis == 1 ? d : d * d);
            const int me = axis == 0 ? i : (axis == 1 ? j : k);
            const double *v = src + (tid - me * st);
            double acc = 0.0;
            for (int m = 0; m < d; m++)  // back-transform: the basis transposed
                acc = fma(pass < 3 ? S.q[me * kMaxC + m] : S.q[m * kMaxC + me], v[m * st], acc);
            if (pass == 2) acc *= factor;
            dst[tid] = acc;
        }
        __syncthreads();
        double *t = src;
        src = dst;
        dst = t;
    }
    if (on) S.xc[((k + 1) * (d + 2) + (j + 1)) * (d + 2) + i + 1] = (float)src[tid];
    __syncthreads();
}

// Eight half sweeps of level B (CTA 0).
__device__ __forceinline__ void smooth_b(float *__restrict__ x, const Pair (&it)[kItemsB], const float2 (&bv)[kItemsB],
                                         int d) {
    const int P = d + 2;
    for (int h = 0; h < 8; h++) {
        const int color = (h & 1) ^ 1;
#pragma unroll
        for (int q = 0; q < kItemsB; q++) {
            if (it[q].on) {
                const int e = (it[q].par + color) & 1;
                const int o = it[q].off + e;
                x[o] = mg_sor_update(x[o], nb6(x, o, P), e ? bv[q].y : bv[q].x);
            }
        }
        __syncthreads();
    }
}

// One V(4,4) cycle on B and C in CTA 0, b_B given, x_B zero or given.
__device__ void cycle_b(TailShared &S, const Pair (&it)[kItemsB], int dB, int dC, double factor, int tid) {
    const int P = dB + 2, PC = dC + 2;
    float2 bv[kItemsB];
#pragma unroll
    for (int q = 0; q < kItemsB; q++) {
        bv[q] = make_float2(0.f, 0.f);
        const int p = tid + q * kTailThreads;
        if (it[q].on) bv[q] = make_float2(S.bb[2 * p], S.bb[2 * p + 1]);
    }
    smooth_b(S.xb, it, bv, dB);
    const int cells = dC * dC * dC;
    const int ic = tid % dC, jc = (tid / dC) % dC, kc = tid / (dC * dC);
    if (tid < cells)
        S.bc[tid] = restrict8(S.xb, S.bb, ((2 * kc + 1) * P + 2 * jc + 1) * P + 2 * ic + 1,
                              (2 * kc * dB + 2 * jc) * dB + 2 * ic, dB, false);
    __syncthreads();
    coarse_modes(S, dC, factor, tid);
    if (tid < cells) {
        const float v = S.xc[((kc + 1) * PC + jc + 1) * PC + ic + 1];
        const int o = ((2 * kc + 1) * P + 2 * jc + 1) * P + 2 * ic + 1;
#pragma unroll
        for (int q = 0; q < 8; q++) S.xb[o + (q & 1) + ((q >> 1) & 1) * P + (q >> 2) * P * P] += v;
    }
    __syncthreads();
    smooth_b(S.xb, it, bv, dB);
}

// FMG: the full multigrid of the levels from b (x from the coarse solution);
// otherwise one V(4,4) cycle from x = 0.
template <bool FMG>
__global__ void __cluster_dims__(kTailCtas, 1, 1) __launch_bounds__(kTailThreads)
mg_tail_kernel(const TailArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    TailShared &S = *reinterpret_cast<TailShared *>(smem);
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x;
    const int rank = (int)cl.block_rank();
    const int comp = blockIdx.y;
    const int dA = a.dA, dB = a.dB, dC = a.dC, PA = dA + 2, PB = dB + 2;
    if (dA == 0 && rank != 0) return;  // level B is the top: one CTA does it all, nothing is shared

    // the coarsest level's basis, this thread's mode factor
    double factor = 0.0;
    if (rank == 0) {
        if (tid < kMaxC * kMaxC) S.q[tid] = a.basis[tid];
        if (tid < dC * dC * dC) {
            const double mu = (6.0 + a.lambda[tid % dC] + a.lambda[(tid / dC) % dC] + a.lambda[tid / (dC * dC)]) / 6.0;
            const double m2 = mu * mu, m4 = m2 * m2, m8 = m4 * m4, m16 = m8 * m8, m32 = m16 * m16, m64 = m32 * m32;
            factor = -(1.0 - m64 * m32 * m4) / (6.0 * (1.0 - mu));
        }
        for (int q = tid; q < (kMaxC + 2) * (kMaxC + 2) * (kMaxC + 2); q += kTailThreads) S.xc[q] = 0.f;
    }
    // level B's cell pairs of this thread
    Pair itb[kItemsB];
#pragma unroll
    for (int q = 0; q < kItemsB; q++) {
        const int p = tid + q * kTailThreads, hb = dB >> 1;
        const int ih = p % hb, j = (p / hb) % dB, k = p / (hb * dB);
        itb[q].on = p < hb * dB * dB;
        itb[q].off = ((k + 1) * PB + j + 1) * PB + 2 * ih + 1;
        itb[q].par = (j + k) & 1;
        itb[q].first = itb[q].last = false;
    }
    for (int q = tid; q < PB * PB * PB; q += kTailThreads) S.xb[q] = 0.f;

    // this CTA's slab of A: planes [z0, z1)
    const int z0 = min(rank * kSlab, dA), z1 = min(z0 + kSlab, dA);
    const int own = (z1 - z0) * dA * dA;
    Pair ita[kItems];
    float2 bva[kItems];
    const size_t cellsA = (size_t)dA * dA * dA;
    if (dA) {
        const float *bg = a.b + comp * cellsA + (size_t)z0 * dA * dA;
        for (int q = tid; q < (kSlab + 2) * PA * PA; q += kTailThreads) S.xa[q] = 0.f;
#pragma unroll
        for (int q = 0; q < kItems; q++) {
            const int p = tid + q * kTailThreads, ha = dA >> 1;
            const int ih = p % ha, j = (p / ha) % dA, kl = p / (ha * dA);
            ita[q].on = 2 * p < own;
            ita[q].off = ((kl + 1) * PA + j + 1) * PA + 2 * ih + 1;
            ita[q].par = (j + z0 + kl) & 1;
            ita[q].first = kl == 0 && rank > 0;
            ita[q].last = z0 + kl == z1 - 1 && z1 < dA;
            bva[q] = make_float2(0.f, 0.f);
            if (ita[q].on) {
                bva[q] = *reinterpret_cast<const float2 *>(bg + 2 * p);
                *reinterpret_cast<float2 *>(&S.ba[2 * p]) = bva[q];
            }
        }
    } else {
        const float *bg = a.b + comp * (size_t)dB * dB * dB;
        for (int q = tid; q < dB * dB * dB; q += kTailThreads) S.bb[q] = bg[q];
    }
    float *bb0 = nullptr, *xb0 = nullptr, *up = nullptr, *down = nullptr;
    if (dA) {
        bb0 = cl.map_shared_rank(S.bb, 0);
        xb0 = cl.map_shared_rank(S.xb, 0);
        // the neighbours' halo planes that this CTA's first plane (padded
        // plane 1) and last plane (padded plane kSlab: a CTA with another
        // above it has a whole slab) fill, both indexed by the cell's own
        // padded offset
        if (rank > 0) down = cl.map_shared_rank(S.xa, rank - 1) + kSlab * PA * PA;
        if (z1 < dA) up = cl.map_shared_rank(S.xa, rank + 1) - kSlab * PA * PA;
        cl.sync();  // every CTA runs and has set its planes up
    } else {
        __syncthreads();
    }
    // b_B of CTA 0 from this CTA's planes
    auto restrict_a = [&](bool x_zero) {
        for (int q = tid; q < own / 8; q += kTailThreads) {
            const int ic = q % dB, jc = (q / dB) % dB, kl = q / (dB * dB);
            bb0[((z0 >> 1) + kl) * dB * dB + jc * dB + ic] =
                restrict8(S.xa, S.ba, ((2 * kl + 1) * PA + 2 * jc + 1) * PA + 2 * ic + 1,
                          (2 * kl * dA + 2 * jc) * dA + 2 * ic, dA, x_zero);
        }
    };
    // x_A += x_B injected, on this CTA's planes and its halo planes
    auto inject_a = [&]() {
        const int lo = max(z0 - 1, 0), cnt = (min(z1 + 1, dA) - lo) * dA * dA;
        if (z0 < z1)
            for (int q = tid; q < cnt; q += kTailThreads) {
                const int i = q % dA, j = (q / dA) % dA, z = lo + q / (dA * dA);
                S.xa[((z - z0 + 1) * PA + j + 1) * PA + i + 1] +=
                    xb0[(((z >> 1) + 1) * PB + (j >> 1) + 1) * PB + (i >> 1) + 1];
            }
    };
    auto smooth_a = [&]() {
        for (int h = 0; h < 8; h++) {
            const int color = (h & 1) ^ 1;
#pragma unroll
            for (int q = 0; q < kItems; q++) {
                if (ita[q].on) {
                    const int e = (ita[q].par + color) & 1;
                    const int o = ita[q].off + e;
                    const float v = mg_sor_update(S.xa[o], nb6(S.xa, o, PA), e ? bva[q].y : bva[q].x);
                    S.xa[o] = v;
                    if (ita[q].first) down[o] = v;
                    if (ita[q].last) up[o] = v;
                }
            }
            cl.sync();
        }
    };

    if (FMG) {
        if (dA) {
            restrict_a(true);
            cl.sync();
        }
        if (rank == 0) {
            const int cells = dC * dC * dC, PC = dC + 2;
            const int ic = tid % dC, jc = (tid / dC) % dC, kc = tid / (dC * dC);
            if (tid < cells) S.bc[tid] = restrict8(S.xb, S.bb, 0, (2 * kc * dB + 2 * jc) * dB + 2 * ic, dB, true);
            __syncthreads();
            coarse_modes(S, dC, factor, tid);
            if (tid < cells) {
                const float v = S.xc[((kc + 1) * PC + jc + 1) * PC + ic + 1];
                const int o = ((2 * kc + 1) * PB + 2 * jc + 1) * PB + 2 * ic + 1;
#pragma unroll
                for (int q = 0; q < 8; q++) S.xb[o + (q & 1) + ((q >> 1) & 1) * PB + (q >> 2) * PB * PB] = v;
            }
            __syncthreads();
            cycle_b(S, itb, dB, dC, factor, tid);
        }
        if (dA) {
            cl.sync();
            inject_a();
            cl.sync();  // every CTA has read x_B
        }
    }
    if (dA) {
        if (FMG && rank == 0)
            for (int q = tid; q < PB * PB * PB; q += kTailThreads) S.xb[q] = 0.f;
        smooth_a();
        restrict_a(false);
        cl.sync();
        if (rank == 0) cycle_b(S, itb, dB, dC, factor, tid);
        cl.sync();
        inject_a();
        cl.sync();  // a neighbour's first stores into the halo planes come after they are injected
        smooth_a();
        float *xg = a.x + comp * cellsA + (size_t)z0 * dA * dA;
#pragma unroll
        for (int q = 0; q < kItems; q++)
            if (ita[q].on)
                *reinterpret_cast<float2 *>(xg + 2 * (tid + q * kTailThreads)) =
                    make_float2(S.xa[ita[q].off], S.xa[ita[q].off + 1]);
    } else {
        if (!FMG) cycle_b(S, itb, dB, dC, factor, tid);
        float *xg = a.x + comp * (size_t)dB * dB * dB;
#pragma unroll
        for (int q = 0; q < kItemsB; q++)
            if (itb[q].on)
                *reinterpret_cast<float2 *>(xg + 2 * (tid + q * kTailThreads)) =
                    make_float2(S.xb[itb[q].off], S.xb[itb[q].off + 1]);
    }
}

}  // namespace

// First level of a hierarchy that the launch can take: the first of edge
// <= 32 with a coarser level below it; -1 for a hierarchy without one.
int mg_tail_level(const MGPlan &m) {
    for (int l = 0; l + 1 < m.levels; l++)
        if (m.lv[l].d <= (uint32_t)kMaxA) return l;
    return -1;
}

TailArgs mg_tail_args(const MGPlan &m, int level) {
    TailArgs a;
    int l = level;
    if (m.lv[l].d > (uint32_t)kMaxB) a.dA = (int)m.lv[l++].d;
    a.dB = (int)m.lv[l].d;
    a.dC = (int)m.lv[l + 1].d;
    a.x = m.lv[level].x;
    a.b = m.lv[level].b;
    // sine modes of the one-dimensional second difference with zero ends
    const double pi = 3.14159265358979323846;
    const int n = a.dC;
    for (int i = 0; i < n; i++) {
        a.lambda[i] = -2.0 + 2.0 * std::cos(pi * (i + 1) / (n + 1));
        for (int j = 0; j < n; j++)
            a.basis[i * kMaxC + j] = std::sqrt(2.0 / (n + 1)) * std::sin(pi * (i + 1) * (j + 1) / (n + 1));
    }
    return a;
}

cudaError_t mg_tail_prepare() {
    PPPM_CUDA_TRY(cudaFuncSetAttribute(mg_tail_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(TailShared)));
    return cudaFuncSetAttribute(mg_tail_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(TailShared));
}

// The full multigrid (fmg) of lv[level].b, or one V(4,4) cycle on it from
// zero, over level `level` and every coarser one; the result is lv[level].x.
cudaError_t mg_tail_launch(const MGPlan &m, int level, bool fmg) {
    const TailArgs a = mg_tail_args(m, level);
    const dim3 grid(kTailCtas, m.comps);
    ::pppm::note_launch();
    if (fmg) mg_tail_kernel<true><<<grid, kTailThreads, sizeof(TailShared), m.st>>>(a);
    else mg_tail_kernel<false><<<grid, kTailThreads, sizeof(TailShared), m.st>>>(a);
    return cudaGetLastError();
}

}  // namespace pppm
