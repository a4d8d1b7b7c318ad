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
//      sweep (sine modes).  Applied as a 512 x 512 matrix the same map would
//      have one CTA read 2 MB.
// Edges: the levels halve, every level above the coarsest is even, and the
// coarsest is the first with at most 512 cells, so a hierarchy has at most
// one level of each kind; grids of edge 9 to 16 start at B.
//
// Sums are taken in the order of the larger levels' kernels (mg_sweep.cu,
// mg.cu), so a level holds the same values bit for bit wherever it runs; the
// coarsest solve agrees with 100 sweeps to FP64 rounding.
//
// The basis is formed on the host at each launch: sines, captured once with the
// graph of the fixed schedule, or, for the corrected cycle, an eigenproblem of at
// most 8 points that takes 12 us (5 points) to 45 us (8) of host time.
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
constexpr int kQ = kMaxC + 1;  // row stride of the basis (no bank conflicts either way)
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
    double q[kMaxC * kQ];
};

// p / d for p < 2^16 and d <= 32 by one multiplication (the edges are known
// only at run time, and every index here needs a division or two).
struct Div {
    int d;
    uint32_t m;
    __device__ explicit Div(int v) : d(v), m(v > 1 ? 0xFFFFFFFFu / (uint32_t)v + 1u : 0u) {}
    __device__ __forceinline__ int quot(int p) const { return d > 1 ? (int)__umulhi((uint32_t)p, m) : p; }
    __device__ __forceinline__ int rem(int p, int q) const { return p - q * d; }
};
// p -> (i, j, k) on an a x b x . box, x fastest
__device__ __forceinline__ void split(const Div &a, const Div &b, int p, int &i, int &j, int &k) {
    const int row = a.quot(p);
    i = a.rem(p, row);
    k = b.quot(row);
    j = b.rem(row, k);
}

// A cell pair (2 ih, 2 ih + 1) of row (j, z): offset into the padded x, the
// parity of j + z, and (level A) whether its plane is a neighbour's halo.
struct Pair {
    int off;
    int par;
    bool on, first, last;
    int f0, f1;  // boundary faces of the two cells
};

__device__ __forceinline__ float nb6(const float *__restrict__ x, int o, int P) {
    return ((x[o - 1] + x[o + 1]) + (x[o + P] + x[o - P])) + (x[o - P * P] + x[o + P * P]);
}

__device__ __forceinline__ int faces_of(int i, int d) { return (i == 0) + (i == d - 1); }

__device__ __forceinline__ float pick4(const float4 &v, int i) {
    return i < 2 ? (i == 0 ? v.x : v.y) : (i == 2 ? v.z : v.w);
}

// b restricted to the coarse cell whose first child sits at padded offset o
// of x and at ob of b: 0.5 * sum of the children's residuals (of b itself
// when x is zero), in resid_restrict2_kernel's order (mg.cu).  CORR: (i, j, k)
// is the first child, ghost the level's ghost factor.
template <bool CORR>
__device__ __forceinline__ float restrict8(const float *__restrict__ x, const float *__restrict__ b, int o, int ob,
                                           int d, bool x_zero, float ghost, int i, int j, int k) {
    const int P = d + 2;
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int c = o + (q & 1) + ((q >> 1) & 1) * P + (q >> 2) * P * P;
        float r = b[ob + (q & 1) + ((q >> 1) & 1) * d + (q >> 2) * d * d];
        if (!x_zero) {
            float diag = 6.f;
            if (CORR)
                diag -= ghost * (float)(faces_of(i + (q & 1), d) + faces_of(j + ((q >> 1) & 1), d) +
                                        faces_of(k + (q >> 2), d));
            r -= nb6(x, c, P) - diag * x[c];
        }
        sum += r;
    }
    return sum * 0.5f;
}

// The ghost cells of a padded x: its boundary cells times the ghost factor,
// along each axis in turn (all threads).
__device__ void fill_ghosts(float *__restrict__ x, int d, float ghost, int tid) {
    const int P = d + 2;
    for (int axis = 0; axis < 3; axis++) {
        const int st = axis == 0 ? 1 : (axis == 1 ? P : P * P);
        for (int q = tid; q < P * P; q += kTailThreads) {
            const int u = q % P, v = q / P;
            const int o = axis == 0 ? (v * P + u) * P : (axis == 1 ? v * P * P + u : v * P + u);
            x[o] = ghost * x[o + st];
            x[o + (d + 1) * st] = ghost * x[o + d * st];
        }
        __syncthreads();
    }
}

// Trilinear interpolation of a padded coarse x (ghosts filled) at fine cell
// (i, j, k): 3/4 of the parent and 1/4 of its neighbour on the cell's side
// along each axis.
__device__ __forceinline__ float trilinear(const float *__restrict__ x, int P, int i, int j, int k) {
    const int o = (((k >> 1) + 1) * P + (j >> 1) + 1) * P + (i >> 1) + 1;
    const int sx = (i & 1) ? 1 : -1, sy = (j & 1) ? P : -P, sz = (k & 1) ? P * P : -P * P;
    auto line = [&](int at) { return fmaf(0.25f, x[at + sx], 0.75f * x[at]); };
    auto face = [&](int at) { return fmaf(0.25f, line(at + sy), 0.75f * line(at)); };
    return fmaf(0.25f, face(o + sz), 0.75f * face(o));
}

// x_C = the coarsest solve of b_C (all threads; edge d).  The transforms run
// over 8 points whatever d is, the basis being zero beyond it: loads ahead of
// the sums and no loop control, which is all a pass of one term in eight lasts.
__device__ __forceinline__ void coarse_modes(TailShared &S, int d, double factor, int tid, int i, int j, int k) {
    const bool on = tid < d * d * d;
    if (on) S.t0[tid] = (double)S.bc[tid];
    __syncthreads();
#pragma unroll
    for (int pass = 0; pass < 6; pass++) {
        const double *src = (pass & 1) ? S.t1 : S.t0;
        double *dst = (pass & 1) ? S.t0 : S.t1;
        const int axis = pass % 3;
        if (on) {
            const int st = axis == 0 ? 1 : (axis == 1 ? d : d * d);
            const int me = axis == 0 ? i : (axis == 1 ? j : k);
            const double *v = src + (tid - me * st);
            double x[kMaxC], q[kMaxC];
#pragma unroll
            for (int m = 0; m < kMaxC; m++) {
                x[m] = m < d ? v[m * st] : 0.0;
                q[m] = pass < 3 ? S.q[me * kQ + m] : S.q[m * kQ + me];  // back-transform: transposed
            }
            double a0 = q[0] * x[0], a1 = q[1] * x[1];
#pragma unroll
            for (int m = 2; m < kMaxC; m += 2) {
                a0 = fma(q[m], x[m], a0);
                a1 = fma(q[m + 1], x[m + 1], a1);
            }
            const double acc = a0 + a1;
            dst[tid] = pass == 2 ? acc * factor : acc;
        }
        __syncthreads();
    }
    if (on) S.xc[((k + 1) * (d + 2) + (j + 1)) * (d + 2) + i + 1] = (float)S.t0[tid];
    __syncthreads();
}

// Eight half sweeps of level B (CTA 0); CORR: four.
template <bool CORR>
__device__ __forceinline__ void smooth_b(float *__restrict__ x, const Pair (&it)[kItemsB], const float2 (&bv)[kItemsB],
                                         int d, const float4 inv) {
    const int P = d + 2;
    for (int h = 0; h < (CORR ? 4 : 8); h++) {
        const int color = (h & 1) ^ 1;
#pragma unroll
        for (int q = 0; q < kItemsB; q++) {
            if (it[q].on) {
                const int e = (it[q].par + color) & 1;
                const int o = it[q].off + e;
                const float nb = nb6(x, o, P), b = e ? bv[q].y : bv[q].x;
                x[o] = CORR ? mg_corr_update(x[o], nb, b, pick4(inv, e ? it[q].f1 : it[q].f0)) : mg_sor_update(x[o], nb, b);
            }
        }
        __syncthreads();
    }
}

// One V(4,4) cycle on B and C in CTA 0, b_B given, x_B zero or given; CORR:
// one corrected V(2,2) cycle from zero, the ghosts of x_B filled after it.
template <bool CORR>
__device__ void cycle_b(TailShared &S, const Pair (&it)[kItemsB], const TailArgs &a, double factor, int tid) {
    const int dB = a.dB, dC = a.dC;
    const int P = dB + 2, PC = dC + 2;
    float2 bv[kItemsB];
#pragma unroll
    for (int q = 0; q < kItemsB; q++) {
        bv[q] = make_float2(0.f, 0.f);
        const int p = tid + q * kTailThreads;
        if (it[q].on) bv[q] = make_float2(S.bb[2 * p], S.bb[2 * p + 1]);
    }
    smooth_b<CORR>(S.xb, it, bv, dB, a.invB);
    const int cells = dC * dC * dC;
    const Div vB(dB), vC(dC);
    int ic, jc, kc;
    split(vC, vC, tid, ic, jc, kc);
    if (tid < cells)
        S.bc[tid] = restrict8<CORR>(S.xb, S.bb, ((2 * kc + 1) * P + 2 * jc + 1) * P + 2 * ic + 1,
                                    (2 * kc * dB + 2 * jc) * dB + 2 * ic, dB, false, a.gB, 2 * ic, 2 * jc, 2 * kc);
    __syncthreads();
    coarse_modes(S, dC, factor, tid, ic, jc, kc);
    if (CORR) {
        fill_ghosts(S.xc, dC, a.gC, tid);
        for (int q = tid; q < dB * dB * dB; q += kTailThreads) {
            int i, j, k;
            split(vB, vB, q, i, j, k);
            S.xb[((k + 1) * P + j + 1) * P + i + 1] += trilinear(S.xc, PC, i, j, k);
        }
    } else if (tid < cells) {
        const float v = S.xc[((kc + 1) * PC + jc + 1) * PC + ic + 1];
        const int o = ((2 * kc + 1) * P + 2 * jc + 1) * P + 2 * ic + 1;
#pragma unroll
        for (int q = 0; q < 8; q++) S.xb[o + (q & 1) + ((q >> 1) & 1) * P + (q >> 2) * P * P] += v;
    }
    __syncthreads();
    smooth_b<CORR>(S.xb, it, bv, dB, a.invB);
    if (CORR) fill_ghosts(S.xb, dB, a.gB, tid);
}

// kTailFull: the full multigrid of the levels from b (x from the coarse
// solution); otherwise one cycle from x = 0, V(4,4) or the corrected V(2,2).
template <TailMode MODE>
__global__ void __cluster_dims__(kTailCtas, 1, 1) __launch_bounds__(kTailThreads)
mg_tail_kernel(const TailArgs a) {
    constexpr bool FMG = MODE == kTailFull, CORR = MODE == kTailCorrected;
    extern __shared__ __align__(16) unsigned char smem[];
    TailShared &S = *reinterpret_cast<TailShared *>(smem);
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x;
    const int rank = (int)cl.block_rank();
    const int comp = blockIdx.y;
    const int dA = a.dA, dB = a.dB, dC = a.dC, PA = dA + 2, PB = dB + 2;
    if (dA == 0 && rank != 0) return;  // level B is the top: one CTA does it all, nothing is shared

    const Div vA(dA), vB(dB), vC(dC);
    // the coarsest level's basis, this thread's mode factor
    double factor = 0.0;
    if (rank == 0) {
        if (tid < kMaxC * kMaxC) S.q[(tid >> 3) * kQ + (tid & 7)] = a.basis[tid];
        if (tid < dC * dC * dC) {
            int ic, jc, kc;
            split(vC, vC, tid, ic, jc, kc);
            const double sum = a.lambda[ic] + a.lambda[jc] + a.lambda[kc];
            const double mu = (6.0 + sum) / 6.0;
            const double m2 = mu * mu, m4 = m2 * m2, m8 = m4 * m4, m16 = m8 * m8, m32 = m16 * m16, m64 = m32 * m32;
            factor = CORR ? 1.0 / sum : -(1.0 - m64 * m32 * m4) / (6.0 * (1.0 - mu));
        }
        for (int q = tid; q < (kMaxC + 2) * (kMaxC + 2) * (kMaxC + 2); q += kTailThreads) S.xc[q] = 0.f;
    }
    const Div vHA(dA >> 1), vHB(dB >> 1);
    // level B's cell pairs of this thread
    Pair itb[kItemsB];
#pragma unroll
    for (int q = 0; q < kItemsB; q++) {
        const int p = tid + q * kTailThreads, hb = dB >> 1;
        int ih, j, k;
        split(vHB, vB, p, ih, j, k);
        itb[q].on = p < hb * dB * dB;
        itb[q].off = ((k + 1) * PB + j + 1) * PB + 2 * ih + 1;
        itb[q].par = (j + k) & 1;
        itb[q].first = itb[q].last = false;
        itb[q].f0 = faces_of(j, dB) + faces_of(k, dB) + (ih == 0);
        itb[q].f1 = faces_of(j, dB) + faces_of(k, dB) + (ih == hb - 1);
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
            int ih, j, kl;
            split(vHA, vA, p, ih, j, kl);
            ita[q].on = 2 * p < own;
            ita[q].off = ((kl + 1) * PA + j + 1) * PA + 2 * ih + 1;
            ita[q].par = (j + z0 + kl) & 1;
            ita[q].first = kl == 0 && rank > 0;
            ita[q].last = z0 + kl == z1 - 1 && z1 < dA;
            ita[q].f0 = faces_of(j, dA) + faces_of(z0 + kl, dA) + (ih == 0);
            ita[q].f1 = faces_of(j, dA) + faces_of(z0 + kl, dA) + (ih == ha - 1);
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
            int ic, jc, kl;
            split(vB, vB, q, ic, jc, kl);
            bb0[((z0 >> 1) + kl) * dB * dB + jc * dB + ic] =
                restrict8<CORR>(S.xa, S.ba, ((2 * kl + 1) * PA + 2 * jc + 1) * PA + 2 * ic + 1,
                                (2 * kl * dA + 2 * jc) * dA + 2 * ic, dA, x_zero, a.gA, 2 * ic, 2 * jc, z0 + 2 * kl);
        }
    };
    // x_A += x_B injected (CORR: interpolated), on this CTA's planes and its
    // halo planes
    auto inject_a = [&]() {
        const int lo = max(z0 - 1, 0), cnt = (min(z1 + 1, dA) - lo) * dA * dA;
        if (CORR) {
            // the coarse planes around them first, into this CTA's own x_B
            const int c0 = (lo >> 1), c1 = ((min(z1 + 1, dA) - 1) >> 1) + 2;  // padded planes
            if (z0 < z1 && rank != 0)
                for (int q = c0 * PB * PB + tid; q < (c1 + 1) * PB * PB; q += kTailThreads) S.xb[q] = xb0[q];
            __syncthreads();
            if (z0 < z1)
                for (int q = tid; q < cnt; q += kTailThreads) {
                    int i, j, z;
                    split(vA, vA, q, i, j, z);
                    z += lo;
                    S.xa[((z - z0 + 1) * PA + j + 1) * PA + i + 1] += trilinear(S.xb, PB, i, j, z);
                }
        } else if (z0 < z1)
            for (int q = tid; q < cnt; q += kTailThreads) {
                int i, j, z;
                split(vA, vA, q, i, j, z);
                z += lo;
                S.xa[((z - z0 + 1) * PA + j + 1) * PA + i + 1] +=
                    xb0[(((z >> 1) + 1) * PB + (j >> 1) + 1) * PB + (i >> 1) + 1];
            }
    };
    auto smooth_a = [&]() {
        for (int h = 0; h < (CORR ? 4 : 8); h++) {
            const int color = (h & 1) ^ 1;
#pragma unroll
            for (int q = 0; q < kItems; q++) {
                if (ita[q].on) {
                    const int e = (ita[q].par + color) & 1;
                    const int o = ita[q].off + e;
                    const float nb = nb6(S.xa, o, PA), b = e ? bva[q].y : bva[q].x;
                    const float v = CORR ? mg_corr_update(S.xa[o], nb, b, pick4(a.invA, e ? ita[q].f1 : ita[q].f0))
                                         : mg_sor_update(S.xa[o], nb, b);
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
            int ic, jc, kc;
            split(vC, vC, tid, ic, jc, kc);
            if (tid < cells) S.bc[tid] = restrict8<false>(S.xb, S.bb, 0, (2 * kc * dB + 2 * jc) * dB + 2 * ic, dB, true, 0.f, 0, 0, 0);
            __syncthreads();
            coarse_modes(S, dC, factor, tid, ic, jc, kc);
            if (tid < cells) {
                const float v = S.xc[((kc + 1) * PC + jc + 1) * PC + ic + 1];
                const int o = ((2 * kc + 1) * PB + 2 * jc + 1) * PB + 2 * ic + 1;
#pragma unroll
                for (int q = 0; q < 8; q++) S.xb[o + (q & 1) + ((q >> 1) & 1) * PB + (q >> 2) * PB * PB] = v;
            }
            __syncthreads();
            cycle_b<CORR>(S, itb, a, factor, tid);
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
        if (rank == 0) cycle_b<CORR>(S, itb, a, factor, tid);
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
        if (!FMG) cycle_b<CORR>(S, itb, a, factor, tid);
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

// Eigenvectors (rows of q) and eigenvalues of the symmetric n x n matrix t,
// by cyclic Jacobi rotations.
static void small_eigen(int n, double t[8][8], double q[8][8], double *lambda) {
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++) q[i][j] = i == j ? 1.0 : 0.0;
    for (int round = 0; round < 30; round++)
        for (int i = 0; i < n; i++)
            for (int j = i + 1; j < n; j++) {
                if (std::fabs(t[i][j]) < 1e-300) continue;
                const double th = 0.5 * (t[j][j] - t[i][i]) / t[i][j];
                const double tn = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
                const double c = 1.0 / std::sqrt(tn * tn + 1.0), s = tn * c;
                for (int k = 0; k < n; k++) {
                    const double u = t[k][i], v = t[k][j];
                    t[k][i] = c * u - s * v;
                    t[k][j] = s * u + c * v;
                }
                for (int k = 0; k < n; k++) {
                    const double u = t[i][k], v = t[j][k];
                    t[i][k] = c * u - s * v;
                    t[j][k] = s * u + c * v;
                    const double x = q[i][k], y = q[j][k];
                    q[i][k] = c * x - s * y;
                    q[j][k] = s * x + c * y;
                }
            }
    for (int i = 0; i < n; i++) lambda[i] = t[i][i];
}

TailArgs mg_tail_args(const MGPlan &m, int level, bool corrected) {
    TailArgs a;
    int l = level;
    if (m.lv[l].d > (uint32_t)kMaxB) a.dA = (int)m.lv[l++].d;
    a.dB = (int)m.lv[l].d;
    a.dC = (int)m.lv[l + 1].d;
    a.x = m.lv[level].x;
    a.b = m.lv[level].b;
    const int n = a.dC;
    if (corrected) {
        // the coarsest operator with its ghost factor, one-dimensional part
        const float g = mg_ghost_factor(m.levels - 1);
        double t[8][8] = {}, q[8][8];
        for (int i = 0; i < n; i++) {
            t[i][i] = -2.0 + ((i == 0) + (i == n - 1)) * (double)g;
            if (i) t[i][i - 1] = t[i - 1][i] = 1.0;
        }
        small_eigen(n, t, q, a.lambda);
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++) a.basis[i * kMaxC + j] = q[i][j];
        a.gC = g;
        a.gB = mg_ghost_factor(m.levels - 2);
        a.gA = a.dA ? mg_ghost_factor(m.levels - 3) : 0.f;
        auto inv = [](float gh) {
            return make_float4(1.0f / 6.0f, 1.0f / (6.0f - gh), 1.0f / (6.0f - 2.0f * gh), 1.0f / (6.0f - 3.0f * gh));
        };
        a.invA = inv(a.gA);
        a.invB = inv(a.gB);
        return a;
    }
    // sine modes of the one-dimensional second difference with zero ends
    const double pi = 3.14159265358979323846;
    for (int i = 0; i < n; i++) {
        a.lambda[i] = -2.0 + 2.0 * std::cos(pi * (i + 1) / (n + 1));
        for (int j = 0; j < n; j++)
            a.basis[i * kMaxC + j] = std::sqrt(2.0 / (n + 1)) * std::sin(pi * (i + 1) * (j + 1) / (n + 1));
    }
    return a;
}

cudaError_t mg_tail_prepare() {
    const void *k[] = {(const void *)mg_tail_kernel<kTailCycle>, (const void *)mg_tail_kernel<kTailFull>,
                       (const void *)mg_tail_kernel<kTailCorrected>};
    for (const void *f : k)
        PPPM_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TailShared)));
    return cudaSuccess;
}

// The full multigrid of lv[level].b, or one cycle on it from zero, over level
// `level` and every coarser one; the result is lv[level].x.
cudaError_t mg_tail_launch(const MGPlan &m, int level, TailMode mode) {
    const TailArgs a = mg_tail_args(m, level, mode == kTailCorrected);
    const dim3 grid(kTailCtas, m.comps);
    ::pppm::note_launch();
    auto *k = mode == kTailFull ? mg_tail_kernel<kTailFull>
                                : (mode == kTailCorrected ? mg_tail_kernel<kTailCorrected> : mg_tail_kernel<kTailCycle>);
    k<<<grid, kTailThreads, sizeof(TailShared), m.st>>>(a);
    return cudaGetLastError();
}

}  // namespace pppm
