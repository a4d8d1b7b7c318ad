// Curl of the vector potential fused with the far-field correction
// (HFS/GPU_kernel.cu:1750-1805 getCurl, 2487-2564 Step1, 1976-2001 diagonal
// potential, 2566-2630 diagonal subtraction, host table 2646-2692):
//
//   U(c)   = curl(psi)(c), central differences / (2h), clamped sampling
//   far(c) = U(c) - sum_{c' != c, |c'-c|_inf <= K, c' in grid} D[c'-c] x omega(c') h^3
//                 - curl(0.250580605913965 * omega * h^2)(c)     (clamped)
//
// D[off] is the central-difference gradient (step h) of 1/(4 pi |X - X'|)
// between the cell centre and the cell at offset `off`, a coincident pair
// reading 1/1e24 (HFS/GPU_kernel.cu:11-17).  Each block evaluates the
// (2K+1)^3 table in FP64 from the device cell size into shared memory, so the
// reference's per-call host build, cudaMalloc and copy disappear, as does the
// grid-velocity round trip through the host (HFS/BiotSavartSolverImp.cpp:
// 779-781, 811-813).  The curl reads the FP64 potential; the omega stencil
// runs in FP32.
#include <algorithm>

#include "pppm_internal.cuh"

namespace pppm {

namespace {

constexpr int kFFThreads = 256;
constexpr int kMaxTable = (2 * kMaxK + 1) * (2 * kMaxK + 1) * (2 * kMaxK + 1);

__device__ double inv4pi_r(double ax, double ay, double az, double bx, double by, double bz) {
    const double r_sqr = (ax - bx) * (ax - bx) + (ay - by) * (ay - by) + (az - bz) * (az - bz);
    const double r = (r_sqr > 1e-12) ? kFourPi * sqrt(r_sqr) : 1e+24;
    return 1.0 / r;
}

// The (2K+1)^3 table of D into shared memory (one float4 per offset).
__device__ void green_table(float4 *__restrict__ table, double h, int K, int tid, int threads) {
    const int W = 2 * K + 1;
    const int T = W * W * W;
    for (int q = tid; q < T; q += threads) {
        const int ii = q % W - K, jj = (q / W) % W - K, kk = q / (W * W) - K;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ii || jj || kk) {
            const double Xpx = ((double)ii + 0.5) * h, Xpy = ((double)jj + 0.5) * h, Xpz = ((double)kk + 0.5) * h;
            const double X = 0.5 * h;
            v.x = (float)(0.5 * (inv4pi_r(X + h, X, X, Xpx, Xpy, Xpz) - inv4pi_r(X - h, X, X, Xpx, Xpy, Xpz)) / h);
            v.y = (float)(0.5 * (inv4pi_r(X, X + h, X, Xpx, Xpy, Xpz) - inv4pi_r(X, X - h, X, Xpx, Xpy, Xpz)) / h);
            v.z = (float)(0.5 * (inv4pi_r(X, X, X + h, Xpx, Xpy, Xpz) - inv4pi_r(X, X, X - h, Xpx, Xpy, Xpz)) / h);
        }
        table[q] = v;
    }
}

__global__ void __launch_bounds__(kFFThreads)
farfield_kernel(const double *__restrict__ psi, const float *__restrict__ vort, float *__restrict__ far,
                const DevParams *__restrict__ P, int n, int K) {
    __shared__ float4 table[kMaxTable];
    const int W = 2 * K + 1;
    green_table(table, P->cell_h, K, threadIdx.x, blockDim.x);
    __syncthreads();
    const uint32_t C = (uint32_t)n * n * n;
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int i = (int)(c % n), j = (int)((c / n) % n), k = (int)(c / ((uint32_t)n * n));
    const int im = max(i - 1, 0), ip = min(i + 1, n - 1);
    const int jm = max(j - 1, 0), jp = min(j + 1, n - 1);
    const int km = max(k - 1, 0), kp = min(k + 1, n - 1);
    auto at = [n](int x, int y, int z) { return ((size_t)z * n + y) * n + x; };
    const double *Fx = psi, *Fy = psi + C, *Fz = psi + 2 * (size_t)C;
    const float *Wx = vort, *Wy = vort + C, *Wz = vort + 2 * (size_t)C;

    // curl(psi), HFS/GPU_kernel.cu:1770-1793
    const double invh = P->invh;
    const double ux = 0.5 * invh * (Fz[at(i, jp, k)] - Fz[at(i, jm, k)] + Fy[at(i, j, km)] - Fy[at(i, j, kp)]);
    const double uy = 0.5 * invh * (Fx[at(i, j, kp)] - Fx[at(i, j, km)] + Fz[at(im, j, k)] - Fz[at(ip, j, k)]);
    const double uz = 0.5 * invh * (Fy[at(ip, j, k)] - Fy[at(im, j, k)] + Fx[at(i, jm, k)] - Fx[at(i, jp, k)]);

    // mesh's own near-field contribution, HFS/GPU_kernel.cu:2533-2556
    float mx = 0.f, my = 0.f, mz = 0.f;
    for (int dk = -K; dk <= K; dk++) {
        const int kk = k + dk;
        if (kk < 0 || kk >= n) continue;
        for (int dj = -K; dj <= K; dj++) {
            const int jj = j + dj;
            if (jj < 0 || jj >= n) continue;
            for (int di = -K; di <= K; di++) {
                const int ii = i + di;
                if (ii < 0 || ii >= n || (!di && !dj && !dk)) continue;
                const size_t s = at(ii, jj, kk);
                const float4 D = table[((dk + K) * W + (dj + K)) * W + (di + K)];
                const float ox = Wx[s], oy = Wy[s], oz = Wz[s];
                mx += D.y * oz - D.z * oy;
                my += D.z * ox - D.x * oz;
                mz += D.x * oy - D.y * ox;
            }
        }
    }
    const float vh3 = P->vh3_f;
    mx *= vh3;
    my *= vh3;
    mz *= vh3;

    // curl of the diagonal self-potential 0.250580605913965 * omega * h^2
    const float kd = P->kdiag_f;
    const float dx = kd * (Wz[at(i, jp, k)] - Wz[at(i, jm, k)] + Wy[at(i, j, km)] - Wy[at(i, j, kp)]);
    const float dy = kd * (Wx[at(i, j, kp)] - Wx[at(i, j, km)] + Wz[at(im, j, k)] - Wz[at(ip, j, k)]);
    const float dz = kd * (Wy[at(ip, j, k)] - Wy[at(im, j, k)] + Wx[at(i, jm, k)] - Wx[at(i, jp, k)]);

    far[c] = (float)(ux - (double)mx) - dx;
    far[C + c] = (float)(uy - (double)my) - dy;
    far[2 * (size_t)C + c] = (float)(uz - (double)mz) - dz;
}

// The same with a thread per group of 4 consecutive cells of a row (edge a
// multiple of 4), the terms in the one-cell kernel's order.  A group reads each
// of its (2K+1)^2 neighbour rows once with 128-bit loads, 4 + 2K values that
// serve its 4 cells, instead of 2K+1 scalars a cell, and each table entry once;
// the one-cell kernel issues 81 loads and 26 table reads a cell at K = 1 and is
// bound by them.  K = 1 on B200: 1206 to 437 us at 256^3 (its 48 bytes a cell
// take 123 us at the copy rate), 156 to 57 us at 128^3; small grids: see
// launch_farfield.
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

__device__ __forceinline__ void load_row(const double *__restrict__ row, double *v) {
    const double2 a = *reinterpret_cast<const double2 *>(row), b = *reinterpret_cast<const double2 *>(row + 2);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}

template <int K>
__global__ void __launch_bounds__(kFFThreads)
farfield4_kernel(const double *__restrict__ psi, const float *__restrict__ vort, float *__restrict__ far,
                 const DevParams *__restrict__ P, int n) {
    constexpr int W = 2 * K + 1;
    constexpr int R = (K + 3) / 4 * 4;  // values loaded either side of the group
    __shared__ float4 table[W * W * W];
    green_table(table, P->cell_h, K, (int)(threadIdx.y * blockDim.x + threadIdx.x), (int)(blockDim.x * blockDim.y));
    __syncthreads();
    const int g = (int)(blockIdx.x * blockDim.x + threadIdx.x), jt = (int)(blockIdx.y * blockDim.y + threadIdx.y);
    const int k = (int)blockIdx.z;
    // threads beyond the grid follow the last row or group (the lanes exchange
    // values) and store nothing
    const bool on = 4 * g < n && jt < n;
    const int i0 = min(4 * g, n - 4), j = min(jt, n - 1);
    if (K > 1 && !on) return;
    const int tid = (int)(threadIdx.y * blockDim.x + threadIdx.x), lane = tid & 31;
    const int rest = (int)(blockDim.x * blockDim.y) - (tid - lane);  // a block's last warp may not be whole
    const unsigned lanes = rest >= 32 ? 0xffffffffu : (1u << rest) - 1u;
    // whether the lane before / after holds the group before / after
    const bool left = threadIdx.x > 0 && lane > 0, right = threadIdx.x + 1 < blockDim.x && lane < 31 && 4 * g + 4 < n;
    const size_t C = (size_t)n * n * n;
    const float *Wx = vort, *Wy = vort + C, *Wz = vort + 2 * C;
    float mx[4] = {}, my[4] = {}, mz[4] = {};
    // K <= 1: every row in line, without the components of D that vanish on a
    // plane of symmetry, and the two outer values of a row from the lanes that
    // hold them (a load of one value per lane, 16 bytes apart, costs the cache
    // as much as the group's own 128-bit load)
    constexpr bool kSmall = K <= 1;
#pragma unroll (kSmall ? W : 1)
    for (int dk = -K; dk <= K; dk++) {
        const int kk = k + dk;
        if (kk < 0 || kk >= n) continue;
#pragma unroll (kSmall ? W : 1)
        for (int dj = -K; dj <= K; dj++) {
            const int jj = j + dj;
            const bool row_in = jj >= 0 && jj < n;
            if (!kSmall && !row_in) continue;
            const size_t row = ((size_t)kk * n + jj) * n + i0;
            float ox[4 + 2 * R], oy[4 + 2 * R], oz[4 + 2 * R];
#pragma unroll
            for (int q = -R; q < 4 + R; q += 4) {
                if (kSmall && q != 0) continue;
                const bool in = row_in && i0 + q >= 0 && i0 + q < n;
                const int o = q + R;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, c = a;
                if (in) {
                    a = ld4(Wx + row + q);
                    b = ld4(Wy + row + q);
                    c = ld4(Wz + row + q);
                }
                ox[o] = a.x; ox[o + 1] = a.y; ox[o + 2] = a.z; ox[o + 3] = a.w;
                oy[o] = b.x; oy[o + 1] = b.y; oy[o + 2] = b.z; oy[o + 3] = b.w;
                oz[o] = c.x; oz[o + 1] = c.y; oz[o + 2] = c.z; oz[o + 3] = c.w;
            }
            if constexpr (K == 1) {
                auto edges = [&](float (&v)[4 + 2 * R], const float *w) {
                    const float l = __shfl_up_sync(lanes, v[R + 3], 1), r = __shfl_down_sync(lanes, v[R], 1);
                    v[R - 1] = left ? l : (row_in && i0 > 0 ? w[row - 1] : 0.f);
                    v[R + 4] = right ? r : (row_in && i0 + 4 < n ? w[row + 4] : 0.f);
                };
                edges(ox, Wx);
                edges(oy, Wy);
                edges(oz, Wz);
            }
#pragma unroll
            for (int di = -K; di <= K; di++) {
                if (!di && !dj && !dk) continue;
                const float4 D = table[((dk + K) * W + (dj + K)) * W + (di + K)];
                const bool dx = !kSmall || di != 0, dy = !kSmall || dj != 0, dz = !kSmall || dk != 0;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int o = e + di + R;
                    if (dy && dz) mx[e] += D.y * oz[o] - D.z * oy[o];
                    else if (dy) mx[e] += D.y * oz[o];
                    else if (dz) mx[e] -= D.z * oy[o];
                    if (dz && dx) my[e] += D.z * ox[o] - D.x * oz[o];
                    else if (dz) my[e] += D.z * ox[o];
                    else if (dx) my[e] -= D.x * oz[o];
                    if (dx && dy) mz[e] += D.x * oy[o] - D.y * ox[o];
                    else if (dx) mz[e] += D.x * oy[o];
                    else if (dy) mz[e] -= D.y * ox[o];
                }
            }
        }
    }
    const int im = max(i0 - 1, 0), ip = min(i0 + 4, n - 1);
    const int jm = max(j - 1, 0), jp = min(j + 1, n - 1);
    const int km = max(k - 1, 0), kp = min(k + 1, n - 1);
    auto at = [n](int x, int y, int z) { return ((size_t)z * n + y) * n + x; };
    const double *Fx = psi, *Fy = psi + C, *Fz = psi + 2 * C;
    // curl(psi), HFS/GPU_kernel.cu:1770-1793
    const double hh = 0.5 * P->invh;
    double u[4], v[4], w[4];
    {
        double a[4], b[4], c[4], d[4];
        load_row(Fz + at(i0, jp, k), a);
        load_row(Fz + at(i0, jm, k), b);
        load_row(Fy + at(i0, j, km), c);
        load_row(Fy + at(i0, j, kp), d);
#pragma unroll
        for (int e = 0; e < 4; e++) u[e] = hh * (a[e] - b[e] + c[e] - d[e]);
        double z[6], y[6];
        load_row(Fz + at(i0, j, k), z + 1);
        load_row(Fy + at(i0, j, k), y + 1);
        z[0] = im == i0 ? z[1] : Fz[at(im, j, k)];
        z[5] = Fz[at(ip, j, k)];
        y[0] = im == i0 ? y[1] : Fy[at(im, j, k)];
        y[5] = Fy[at(ip, j, k)];
        load_row(Fx + at(i0, j, kp), a);
        load_row(Fx + at(i0, j, km), b);
        load_row(Fx + at(i0, jm, k), c);
        load_row(Fx + at(i0, jp, k), d);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            v[e] = hh * (a[e] - b[e] + z[e] - z[e + 2]);
            w[e] = hh * (y[e + 2] - y[e] + c[e] - d[e]);
        }
    }
    // curl of the diagonal self-potential 0.250580605913965 * omega * h^2
    const float vh3 = P->vh3_f, kd = P->kdiag_f;
    const float4 zjp = ld4(Wz + at(i0, jp, k)), zjm = ld4(Wz + at(i0, jm, k)), ykm = ld4(Wy + at(i0, j, km)),
                 ykp = ld4(Wy + at(i0, j, kp)), xkp = ld4(Wx + at(i0, j, kp)), xkm = ld4(Wx + at(i0, j, km)),
                 xjm = ld4(Wx + at(i0, jm, k)), xjp = ld4(Wx + at(i0, jp, k)), zc = ld4(Wz + at(i0, j, k)),
                 yc = ld4(Wy + at(i0, j, k));
    const float zr[6] = {Wz[at(im, j, k)], zc.x, zc.y, zc.z, zc.w, Wz[at(ip, j, k)]};
    const float yr[6] = {Wy[at(im, j, k)], yc.x, yc.y, yc.z, yc.w, Wy[at(ip, j, k)]};
    const float a0[4] = {zjp.x, zjp.y, zjp.z, zjp.w}, a1[4] = {zjm.x, zjm.y, zjm.z, zjm.w};
    const float a2[4] = {ykm.x, ykm.y, ykm.z, ykm.w}, a3[4] = {ykp.x, ykp.y, ykp.z, ykp.w};
    const float b0[4] = {xkp.x, xkp.y, xkp.z, xkp.w}, b1[4] = {xkm.x, xkm.y, xkm.z, xkm.w};
    const float c0[4] = {xjm.x, xjm.y, xjm.z, xjm.w}, c1[4] = {xjp.x, xjp.y, xjp.z, xjp.w};
    float fx[4], fy[4], fz[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float dx = kd * (a0[e] - a1[e] + a2[e] - a3[e]);
        const float dy = kd * (b0[e] - b1[e] + zr[e] - zr[e + 2]);
        const float dz = kd * (yr[e + 2] - yr[e] + c0[e] - c1[e]);
        fx[e] = (float)(u[e] - (double)(mx[e] * vh3)) - dx;
        fy[e] = (float)(v[e] - (double)(my[e] * vh3)) - dy;
        fz[e] = (float)(w[e] - (double)(mz[e] * vh3)) - dz;
    }
    if (!on) return;
    const size_t c = at(i0, j, k);
    *reinterpret_cast<float4 *>(far + c) = make_float4(fx[0], fx[1], fx[2], fx[3]);
    *reinterpret_cast<float4 *>(far + C + c) = make_float4(fy[0], fy[1], fy[2], fy[3]);
    *reinterpret_cast<float4 *>(far + 2 * C + c) = make_float4(fz[0], fz[1], fz[2], fz[3]);
}

__global__ void __launch_bounds__(kFFThreads)
curl_only_kernel(const double *__restrict__ psi, float *__restrict__ far, const DevParams *__restrict__ P, int n) {
    const uint32_t C = (uint32_t)n * n * n;
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int i = (int)(c % n), j = (int)((c / n) % n), k = (int)(c / ((uint32_t)n * n));
    const int im = max(i - 1, 0), ip = min(i + 1, n - 1);
    const int jm = max(j - 1, 0), jp = min(j + 1, n - 1);
    const int km = max(k - 1, 0), kp = min(k + 1, n - 1);
    auto at = [n](int x, int y, int z) { return ((size_t)z * n + y) * n + x; };
    const double *Fx = psi, *Fy = psi + C, *Fz = psi + 2 * (size_t)C;
    const double invh = P->invh;
    far[c] = (float)(0.5 * invh * (Fz[at(i, jp, k)] - Fz[at(i, jm, k)] + Fy[at(i, j, km)] - Fy[at(i, j, kp)]));
    far[C + c] = (float)(0.5 * invh * (Fx[at(i, j, kp)] - Fx[at(i, j, km)] + Fz[at(im, j, k)] - Fz[at(ip, j, k)]));
    far[2 * (size_t)C + c] =
        (float)(0.5 * invh * (Fy[at(ip, j, k)] - Fy[at(im, j, k)] + Fx[at(i, jm, k)] - Fx[at(i, jp, k)]));
}

}  // namespace

cudaError_t launch_farfield(pppm_scene *s) {
    const unsigned blocks = (s->C + kFFThreads - 1) / kFFThreads;
    ::pppm::note_launch();
    const int n = (int)s->n, K = s->prm.K;
    // K = 0 reads no neighbours beside the two curls', so that below edge 48 there
    // are too few groups of 4 for their longer threads to pay: 2.5 to 3.4 us from
    // 12^3 to 40^3 with a cell a thread, 2.8 to 3.6 us with four; 3.8 and 3.7 at
    // 48^3.  With K = 1 four take 8.0, 8.3 and 9.1 us at 8^3, 12^3 and 20^3 where
    // one takes 8.3, 8.8 and 9.8 (16^3: 8.9 and 8.5), and 12.3 to 13.5 against
    // 19.3 to 21.2 with K = 2.
    if (n % 4 == 0 && (K > 0 || (K == 0 && n >= 48))) {
        const int bx = std::min(32, n / 4);
        const dim3 block(bx, kFFThreads / bx), grid((n / 4 + block.x - 1) / block.x, (n + block.y - 1) / block.y, n);
        auto *f = K == 0 ? farfield4_kernel<0>
                         : (K == 1 ? farfield4_kernel<1>
                                   : (K == 2 ? farfield4_kernel<2> : (K == 3 ? farfield4_kernel<3> : farfield4_kernel<4>)));
        f<<<grid, block, 0, s->stream>>>(s->psi, s->vort, s->far, s->dparams, n);
    } else if (K >= 0)
        farfield_kernel<<<blocks, kFFThreads, 0, s->stream>>>(s->psi, s->vort, s->far, s->dparams, (int)s->n,
                                                              s->prm.K);
    else  // BiotSavartComputeFarField is a no-op for K < 0: far = curl(psi)
        curl_only_kernel<<<blocks, kFFThreads, 0, s->stream>>>(s->psi, s->far, s->dparams, (int)s->n);
    return cudaGetLastError();
}

}  // namespace pppm
