// Velocity evaluation: far-field interpolation + near-field smoothed
// Biot-Savart correction + scatter back to the caller's order, one fused
// kernel (HFS/GPU_kernel.cu:2886-2976 BiotSavartInterpolate_far_field_kernel2,
// :2262-2485 BiotSavartPPCorrScaleMN_kernel, PH/particle_hash_kernel.cu:
// 160-188 removeReorder).
//
// Evaluation points are visited along a Hilbert curve, so that the threads of a
// warp walk the same neighbour cells and read the same vortex records.  Per
// point:
//   * relative position rounded to float from the FP64 difference with the
//     domain origin, NGP cell floor(rel * invh) in FP64 (reference rounding);
//   * far field: hat weights 1 - |cell centre - rel/h| on the 8 surrounding
//     cell centres, cells outside the grid skipped, no write when the point's
//     own cell is outside the grid;
//   * near field: hash cells [i-K-1, i+K+1]^3; a vortex counts when its float
//     coordinate differences are all below (K+0.5)h (the float test is exact:
//     |d| <= largest float below the double bound); contribution
//     (alpha x d) * phi((r/a)^3) / (4 pi a^3) with phi(t) = (1 - e^-t)/t,
//     which equals (1 - e^-(r/a)^3) / (4 pi r^3); pairs with r = 0, or (for
//     segments) a zero distance to the other end, are skipped.
// Pair arithmetic is FP32 (r^3 = r^2 sqrt.approx(r^2) in the warp-uniform walk,
// r^2 rsqrt(r^2) in a lane's own walk; ~1 ulp).  phi in the warp-uniform walk:
// when no pair of the scene can reach t = 0.25, a degree-4 polynomial (Chebyshev
// interpolant on [0, 0.25], relative error 5e-9); when none can reach t = 2, a
// degree-7 one on [0, 2] (relative error 2e-7, below that of the exp form near
// t = 0.25).  No cancellation in either polynomial.  When some pair can reach
// t = 2 (a smoothing radius of about a cell or less), the exp form
// (1 - e^-t) / (4 pi r^3) for every pair, r^-1 from rsqrt.approx and e^-t from
// ex2.approx, with a degree-5 polynomial of phi below t = 1/64, where 1 - e^-t
// would cancel.  A lane's own walk takes the degree-4 polynomial below t = 0.25
// and (1 - exp(-t)) / t above.
#include <climits>
#include <cstring>
#include <cmath>
#include <type_traits>
#include <utility>

#include "pppm_internal.cuh"

namespace pppm {

namespace {

constexpr int kEvalThreads = 128;
// 72 registers.  The pair loop is bound by issue slots and the latency of its
// special functions: 1M points on 128^3 with a of a cell (exp form) take 12.2 ms
// with 7 blocks, 12.3 with 6 (80 registers), 12.5 with 8 (64); 2M segment ends on
// 256^3 (polynomial) 1.30 ms with 7, 1.39 with 6, 1.43 with 8.
constexpr int kEvalBlocksPerSM = 7;

__device__ __forceinline__ float3 rel_pos(float4 p, const DevParams *__restrict__ P) {
    return make_float3((float)((double)p.x - P->origin[0]), (float)((double)p.y - P->origin[1]),
                       (float)((double)p.z - P->origin[2]));
}

// Evaluation order: along a Hilbert curve through the quarter cells of the
// grid (half cells where four times the edge needs more than 10 bits), points
// outside at the nearest one.  32 consecutive points then lie close together
// on all three axes whatever the density, so that the union of their
// near-field boxes, over which a warp walks, exceeds each point's own box by
// little.  Rows of cells, however ordered inside, string the points of a
// sparse scene out along x: 32 of them spanned 20 cells of a 256^3 grid with
// 1.5 vortices a cell.  The order is internal: results return in caller order.
// The curve's index by Skilling's transform (AIP Conf. Proc. 707, 381, 2004):
// undo the rotations from the top bit down, then take the Gray code.
__device__ __forceinline__ uint32_t hilbert_index(uint32_t x, uint32_t y, uint32_t z, int bits) {
    uint32_t v[3] = {x, y, z};
    for (int b = bits - 1; b > 0; b--) {
        const uint32_t q = 1u << b, low = q - 1u;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (v[a] & q) {
                v[0] ^= low;
            } else {
                const uint32_t t = (v[0] ^ v[a]) & low;
                v[0] ^= t;
                v[a] ^= t;
            }
        }
    }
    v[1] ^= v[0];
    v[2] ^= v[1];
    uint32_t t = 0;
    for (int b = bits - 1; b > 0; b--)
        if (v[2] & (1u << b)) t ^= (1u << b) - 1u;
    uint32_t key = 0;
    for (int b = bits - 1; b >= 0; b--)
#pragma unroll
        for (int a = 0; a < 3; a++) key = (key << 1) | (((v[a] ^ t) >> b) & 1u);
    return key;
}

__global__ void eval_keys_kernel(const float4 *__restrict__ eval_a, uint32_t M, const DevParams *__restrict__ P,
                                 int per_cell, int bits, uint32_t *__restrict__ key, uint32_t *__restrict__ idx) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= M) return;
    const float3 r = rel_pos(eval_a[t], P);
    const double scale = P->invh * (double)per_cell, top = (double)(P->n * (uint32_t)per_cell - 1u);
    // (a coordinate that is not a number goes to 0)
    const uint32_t ux = (uint32_t)fmin(fmax((double)r.x * scale, 0.0), top),
                   uy = (uint32_t)fmin(fmax((double)r.y * scale, 0.0), top),
                   uz = (uint32_t)fmin(fmax((double)r.z * scale, 0.0), top);
    key[t] = hilbert_index(ux, uy, uz, bits);
    idx[t] = t;
}

struct PairAcc {
    float x = 0.f, y = 0.f, z = 0.f;
    unsigned long long n = 0;
};

// phi(t) = (1 - e^-t) / t, scaled by 1/(4 pi a^3).  Below t = 0.25 a degree-4
// polynomial (the interpolant at the 5 Chebyshev nodes of [0, 0.25], relative
// error below 5e-9 with float coefficients) needs no special function; its
// coefficients arrive pre-scaled by 1/(4 pi a^3) in cf[0..4].  Above it
// (1 - exp(-t)) / t, where the scene can get there (need_exp).
__device__ __forceinline__ float smooth_coeff(float t, const float *cf, float inv4pia3, bool need_exp) {
    float p = cf[4];
    p = fmaf(p, t, cf[3]);
    p = fmaf(p, t, cf[2]);
    p = fmaf(p, t, cf[1]);
    p = fmaf(p, t, cf[0]);
    if (need_exp) {
        const bool big = t >= 0.25f;
        if (big) {
            const float e = __fdividef(1.0f - __expf(-t), fmaxf(t, 0.25f)) * inv4pia3;
            p = big ? e : p;
        }
    }
    return p;
}

// One candidate pair, branch free: the box test, the lane's cell range and
// the zero-distance exclusions become a zero coefficient.  SEG: test the
// segment's other end; COUNT: count the pairs inside the box.
template <bool SEG, bool COUNT>
__device__ __forceinline__ void pair_term(const float4 r, const float4 al, bool lane_ok, const float3 ra,
                                          const float3 rb, float cr, float inv_a3, const float *cf, float inv4pia3,
                                          bool need_exp, PairAcc &acc) {
    const float dx = ra.x - r.x, dy = ra.y - r.y, dz = ra.z - r.z;
    const float m = fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz)));
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const bool inbox = lane_ok && m <= cr;
    if (COUNT) acc.n += inbox ? 1ull : 0ull;
    bool ok = inbox && !(r2 < 1e-24f);
    if (SEG) {
        const float ex = rb.x - r.x, ey = rb.y - r.y, ez = rb.z - r.z;
        ok = ok && !(fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < 1e-24f);
    }
    const float rr = r2 * rsqrtf(fmaxf(r2, 1e-30f));
    const float c = smooth_coeff(r2 * rr * inv_a3, cf, inv4pia3, need_exp);
    const float coeff = ok ? c : 0.0f;
    acc.x = fmaf(al.y * dz - al.z * dy, coeff, acc.x);
    acc.y = fmaf(al.z * dx - al.x * dz, coeff, acc.y);
    acc.z = fmaf(al.x * dy - al.y * dx, coeff, acc.z);
}

// Near-field sum over one hash cell's vortices for one point (own walk).
template <bool SEG, bool COUNT>
__device__ __forceinline__ void cell_pairs(const float4 *__restrict__ vrec, const float4 *__restrict__ valf,
                                           uint32_t ps, uint32_t pe, bool lane_ok, const float3 ra, const float3 rb,
                                           float cr, float inv_a3, const float *cf, float inv4pia3, bool need_exp,
                                           PairAcc &acc) {
    for (uint32_t p = ps; p < pe; p++)
        pair_term<SEG, COUNT>(vrec[p], valf[p], lane_ok, ra, rb, cr, inv_a3, cf, inv4pia3, need_exp, acc);
}

// The near-field sum of a target,
//   sum_p c_p alpha_p x (ra - r_p),
// is kept as  A x (ra - o) - B  with  A = sum_p c_p alpha_p  and
// B = sum_p c_p alpha_p x (r_p - o), o the middle of the warp's targets: the
// per-source moment alpha_p x (r_p - o) is formed once when the record is
// staged, so a pair costs 6 multiply-adds for the accumulation instead of 9 for
// a cross product per pair.  With o within a few cells of both points, the two
// terms are of the size of the result (no cancellation beyond a few ulp).
struct PairSums {
    float2 ax = {0.f, 0.f}, ay = {0.f, 0.f}, az = {0.f, 0.f};  // .x half: even records, .y half: odd ones
    float2 bx = {0.f, 0.f}, by = {0.f, 0.f}, bz = {0.f, 0.f};
    unsigned long long n = 0;
};

// Ring of a warp: 64 records as 32 record pairs, so that one Blackwell f32x2
// instruction (FADD2 / FMUL2 / FFMA2) works on two records and a lane on its
// own target: slot p holds records 2p (.x, .z halves) and 2p+1 (.y, .w halves).
// Planes: A {-x, -y}, B {-z, alpha_x}, C {alpha_y, alpha_z}, D {m_x, m_y},
// E {m_z, index} with m = alpha x (r - o).
// The sums are a contraction, coefficients (targets x sources) times source
// columns (alpha, m), but as one it is slower: with the coefficients in the
// layout of m16n8k8, split into two TF32 parts to keep FP32's digits, 1M points
// on 128^3 with a of a cell took 15.0 ms against 12.2 ms here, and 262,144
// segments' ends 2.35 ms against 1.78 ms.  The product frees 12 of the 53 issue slots of
// two pairs, the split and the layout take 8 back, and 4 targets x 8 sources of
// coefficients a lane leave too few registers to hide the special functions.
constexpr int kRingSlots = 32;
constexpr int kRingPlanes = 5;
constexpr uint32_t kBlockRecs = 32;  // records per block of the pair loop
// What a warp's walk needs per chunk of records but not per pair, kept out of
// the registers of the pair block.
struct WarpBox {
    float4 lo, hi;   // the targets' boxes' union; lo.w: margin of the near test
    float4 mid;      // origin of the moments; w: the lanes with a near field, as bits
    int4 cells, size;  // first cell x, half-cells y, z and x; cells x, half-cells y, z and last half-cell x
};
struct WarpMem {
    float4 ring[kRingPlanes * kRingSlots];
    WarpBox box;
};

struct Ring {
    uint32_t fill = 0;  // records staged so far
    uint32_t head = 0;  // records evaluated so far (a multiple of kBlockRecs)
    bool near = false;  // a waiting record may lie within a / 4 of a target (exp form)
};

// max(|a|, |b|, |c|) in one instruction: the three-input max.abs of PTX ISA 8.8
// (sm_100 and later).
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float r;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// sqrt.approx.ftz.f32: one special-function op, sqrt(+0) = +0, so
// r^3 = r^2 sqrt(r^2) needs no guard at r = 0 (where rsqrt would give infinity);
// a subnormal r^2 (r < 1e-19) flushes to 0, where phi is its value at 0.
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// rsqrt.approx.ftz.f32 and ex2.approx.ftz.f32: one special-function op each.
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Exp-form constants of the warp-uniform walk for scenes whose pairs reach
// t = (r/a)^3 >= 2 (smoothing radius of about a cell or less).
struct ExpForm {
    float2 inv_a3;   // {1/a^3, 1/a^3}
    float2 nl2a3;    // {-log2(e)/a^3, ...}: the exponent of e^-t in base 2, per r^3
    float tsmall;    // below it phi comes from the polynomial (1 - e^-t cancels)
    float r3small;   // r^3 above tsmall * a^3 by a margin: the warp's trigger
};

// Switch point of the exp form to the polynomial.  ex2.approx has a relative
// error of about 2^-22 (the PTX ISA's bound), so near 1 the absolute error of
// e^-t is about 2^-22 and 1 - e^-t carries a relative error of about
// 2^-22 / t: 1.5e-5 at t = 1/64 (r = a / 4), falling as 1 / t, on pairs whose
// terms are a small part of the sum.  A low switch point keeps the polynomial
// branch rare: with a = h and K = 1 about 0.2 % of a lane's pairs have
// t < 1/64, against 5 % below t = 0.5, where some lane of the warp needed the
// branch on nearly every step.
constexpr float kExpSmallT = 1.0f / 64.0f;

// The exp form of two pairs at (dx, dy, dz): c * 4 pi = (1 - e^-t) / r^3 with
// t = r^3 / a^3: r^-1 from rsqrt, e^-t from ex2 (two special-function ops).
// r^2 gets 1e-30 in its chain, so that rsqrt stays finite at r = 0.  Where some
// lane has t < tsmall (1 - e^-t cancels, or r = 0) the degree-5 polynomial
// phi(t) / a^3 replaces it; CHECK: whether it is looked for.  The trigger
// r^3 < r3small is a superset of t < tsmall, and a pair outside its box may
// trigger it (its coefficient is dropped either way).
template <bool CHECK>
__device__ __forceinline__ float2 exp_coeff(float2 dx, float2 dy, float2 dz, const float2 *cf, const ExpForm &xf) {
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, make_float2(1e-30f, 1e-30f))));
    const float2 rs = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const float2 r3 = __fmul2_rn(r2, __fmul2_rn(r2, rs));
    const float2 ri3 = __fmul2_rn(__fmul2_rn(rs, rs), rs);
    const float2 ex = __fmul2_rn(r3, xf.nl2a3);
    const float2 e = make_float2(ex2_approx(ex.x), ex2_approx(ex.y));
    float2 c = __ffma2_rn(make_float2(-e.x, -e.y), ri3, ri3);
    if (CHECK && __any_sync(0xffffffffu, fminf(r3.x, r3.y) < xf.r3small)) {
        const float2 t = __fmul2_rn(r3, xf.inv_a3);
        float2 p = __ffma2_rn(cf[5], t, cf[4]);
#pragma unroll
        for (int q = 3; q >= 0; q--) p = __ffma2_rn(p, t, cf[q]);
        p = __fmul2_rn(p, xf.inv_a3);
        c.x = t.x < xf.tsmall ? p.x : c.x;
        c.y = t.y < xf.tsmall ? p.y : c.y;
    }
    return c;
}

// phi of two pairs at (dx, dy, dz): the degree-DEG polynomial cf (DEG 4 for
// scenes that never leave [0, 0.25], DEG 7 for those that stay below t = 2), or
// (DEG 0) the exp form.  FOLD: the coefficients carry the powers of 1/a^3, so
// the polynomial takes r^3 directly.
template <bool FOLD, int DEG, bool CHECK>
__device__ __forceinline__ float2 phi_coeff(float2 dx, float2 dy, float2 dz, float2 inv_a3, const float2 *cf,
                                            const ExpForm &xf) {
    float2 c;
    if constexpr (DEG == 0) {
        c = exp_coeff<CHECK>(dx, dy, dz, cf, xf);
    } else {
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        const float2 r3 = __fmul2_rn(r2, make_float2(sqrt_approx(r2.x), sqrt_approx(r2.y)));
        const float2 t3 = FOLD ? r3 : __fmul2_rn(r3, inv_a3);
        c = __ffma2_rn(cf[DEG], t3, cf[DEG - 1]);
#pragma unroll
        for (int q = DEG - 2; q >= 0; q--) c = __ffma2_rn(c, t3, cf[q]);
    }
    return c;
}

// Puts a record (position r, strength a, moments about o) at place e of a ring.
__device__ __forceinline__ void stage_record(WarpMem &W, uint32_t e, float4 r, float4 a, float3 o, uint32_t ridx) {
    const uint32_t slot = (e >> 1) & (kRingSlots - 1), half = e & 1u;
    float *A = reinterpret_cast<float *>(&W.ring[slot]) + half;
    constexpr int kPlane = 4 * kRingSlots;
    const float sx = r.x - o.x, sy = r.y - o.y, sz = r.z - o.z;
    A[0] = -r.x;
    A[2] = -r.y;
    A[kPlane] = -r.z;
    A[kPlane + 2] = a.x;
    A[2 * kPlane] = a.y;
    A[2 * kPlane + 2] = a.z;
    A[3 * kPlane] = fmaf(a.y, sz, -(a.z * sy));
    A[3 * kPlane + 2] = fmaf(a.z, sx, -(a.x * sz));
    A[4 * kPlane] = fmaf(a.x, sy, -(a.y * sx));
    A[4 * kPlane + 2] = __uint_as_float(ridx);
}

// np slots of the ring from slot s0 (FULL: one whole block of 16 slots,
// unrolled into straight-line code with constant offsets): every lane takes
// the records two at a time (broadcast reads).  cr_lane: the half-width of the
// box, or -1 for a lane without a point.  OTHER: the other-end test of segments,
// 1 by position (|rb - r_p|^2 < 1e-24), 2 by record index (the one vortex at rb,
// pstar, found beforehand), 0 none.  The r = 0 exclusion needs no test: the
// pair's ra - r_p is zero.
template <int OTHER, bool COUNT, bool FOLD, int DEG, bool FULL, bool CHECK>
__device__ __forceinline__ void pair_block(const WarpMem &W, uint32_t s0, uint32_t np, float cr_lane,
                                             const float3 ra, const float3 rb, uint32_t pstar, float2 inv_a3,
                                             const float2 *cf, const ExpForm &xf, PairSums &acc) {
    const float2 tx = make_float2(ra.x, ra.x), ty = make_float2(ra.y, ra.y), tz = make_float2(ra.z, ra.z);
    const uint32_t cnt = FULL ? kBlockRecs / 2 : np;
#pragma unroll (FULL ? kBlockRecs / 2 : 2)
    for (uint32_t i = 0; i < cnt; i++) {
        const float4 *pk = &W.ring[s0 + i];
        const float4 A = pk[0], B = pk[kRingSlots], Cc = pk[2 * kRingSlots];
        const float4 D = pk[3 * kRingSlots], E = pk[4 * kRingSlots];
        const float2 nx = make_float2(A.x, A.y), ny = make_float2(A.z, A.w), nz = make_float2(B.x, B.y);
        const float2 dx = __fadd2_rn(tx, nx), dy = __fadd2_rn(ty, ny), dz = __fadd2_rn(tz, nz);
        bool ok0 = max3_abs(dx.x, dy.x, dz.x) <= cr_lane, ok1 = max3_abs(dx.y, dy.y, dz.y) <= cr_lane;
        if (COUNT) acc.n += (ok0 ? 1ull : 0ull) + (ok1 ? 1ull : 0ull);
        if (OTHER == 2) {
            ok0 = ok0 && __float_as_uint(E.z) != pstar;
            ok1 = ok1 && __float_as_uint(E.w) != pstar;
        }
        if (OTHER == 1) {
            const float2 ex = __fadd2_rn(make_float2(rb.x, rb.x), nx);
            const float2 ey = __fadd2_rn(make_float2(rb.y, rb.y), ny);
            const float2 ez = __fadd2_rn(make_float2(rb.z, rb.z), nz);
            const float2 e2 = __ffma2_rn(ex, ex, __ffma2_rn(ey, ey, __fmul2_rn(ez, ez)));
            ok0 = ok0 && !(e2.x < 1e-24f);
            ok1 = ok1 && !(e2.y < 1e-24f);
        }
        const float2 c = phi_coeff<FOLD, DEG, CHECK>(dx, dy, dz, inv_a3, cf, xf);
        // the exp form's c is finite for every pair of a lane with a point (r = 0
        // takes the polynomial), so the box mask can multiply it; the polynomials
        // can overflow on the padding record
        const float2 coeff = (DEG == 0 && OTHER != 1 && !COUNT)
                                 ? __fmul2_rn(c, make_float2(ok0 ? 1.0f : 0.0f, ok1 ? 1.0f : 0.0f))
                                 : make_float2(ok0 ? c.x : 0.0f, ok1 ? c.y : 0.0f);
        acc.ax = __ffma2_rn(coeff, make_float2(B.z, B.w), acc.ax);
        acc.ay = __ffma2_rn(coeff, make_float2(Cc.x, Cc.y), acc.ay);
        acc.az = __ffma2_rn(coeff, make_float2(Cc.z, Cc.w), acc.az);
        acc.bx = __ffma2_rn(coeff, make_float2(D.x, D.y), acc.bx);
        acc.by = __ffma2_rn(coeff, make_float2(D.z, D.w), acc.by);
        acc.bz = __ffma2_rn(coeff, make_float2(E.x, E.y), acc.bz);
    }
}

// Warp-uniform walk up to this many half-cells (a sparse scene's 32 targets
// span several cells); beyond, scattered targets walk their own boxes.
constexpr int kUniformMaxSub = 4096;
// ... and while the targets span no more than this many cells: the moments
// about their middle lose digits to the distance from there, and with a few
// vortices a cell most of the pairs of a block would lie outside the targets'
// boxes.
constexpr double kMaxSpread = 2.5;

// SEG: is_segment == 1 with a distinct other-end array (with eval_b == eval_a
// the other-end test is the r = 0 test itself, so SEG is off).
// Series coefficients of the smoothing kernel, known on the host from a alone;
// passed by value so they sit in the constant bank.
// Polynomials of phi, scaled by 1/(4 pi a^3).  The packed forms hold each
// coefficient twice ({c, c}): the f32x2 multiply-add then reads them straight
// from the kernel's parameter bank.  With fold they are in r^3 (c_q / a^(3q)),
// otherwise in t = (r/a)^3.
struct SmoothSeries {
    float c[5];    // degree 4 on [0, 0.25], in t (a lane's own walk)
    float2 p4[5];  // degree 4 on [0, 0.25], packed
    float2 p7[8];  // degree 7 on [0, 2], packed
    float2 p5[6];  // degree 5 on [0, 0.5] in t, unit scale (exp-form walk)
};

// One block of evaluation points of one scene: kEvalThreads consecutive points
// in the evaluation order, or (SPLIT) 32 points, whose walk the block's four
// warps share.
template <bool SEG, bool COUNT, bool FOLD, bool SPLIT>
__device__ __forceinline__ void eval_points(const SmoothSeries &sc, const EvalArgs &ea, uint32_t block,
                                            WarpMem *__restrict__ stage) {
    const uint32_t *__restrict__ eidx = ea.eidx;
    const uint32_t M = ea.M;
    const float4 *__restrict__ eval_a = ea.eval_a;
    const float4 *__restrict__ eval_b = ea.eval_b;
    const float *__restrict__ far = ea.far;
    const uint32_t *__restrict__ start = ea.start;
    const uint32_t *__restrict__ end = ea.end;
    const uint32_t *__restrict__ sub_start = ea.sub_start;
    const float4 *__restrict__ vrec = ea.vrec;
    const float4 *__restrict__ valf = ea.valf;
    const DevParams *__restrict__ P = ea.P;
    const int n = ea.n, K = ea.K;
    double *__restrict__ u = ea.u;
    double *__restrict__ v = ea.v;
    double *__restrict__ w = ea.w;
    float *__restrict__ uf = ea.uf;
    unsigned long long *__restrict__ pair_count = ea.pair_count;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    WarpMem &W = stage[warp];
    const uint32_t s = SPLIT ? block * 32 + lane : block * blockDim.x + threadIdx.x;
    const bool act = s < M;
    const double invh = P->invh;
    const uint32_t C = (uint32_t)n * n * n;
    PairAcc acc;
    PairSums sums;
    // some pair can reach t = 2: the exp-form walk (its sums carry 4 pi)
    const bool tier0 = P->need_exp2 != 0;
    unsigned near_lanes = 0;
    if (K >= 0) {
        float3 ra = make_float3(0.f, 0.f, 0.f), rb = make_float3(0.f, 0.f, 0.f);
        if (act) {
            const uint32_t q = eidx[s];
            ra = rel_pos(eval_a[q], P);
            if (SEG) rb = rel_pos(eval_b[q], P);
        }
        const double qx = (double)ra.x * invh, qy = (double)ra.y * invh, qz = (double)ra.z * invh;
        const int i = (int)floor(qx), j = (int)floor(qy), k = (int)floor(qz);
        // FOLD: coefficients carry 1/(4 pi a^3); otherwise they have unit
        // scale and the sums are scaled once per point below
        const float cr = P->cr_f, inv_a3 = P->inv_a3_f, inv4pia3 = FOLD ? P->inv4pia3_f : 1.0f;
        const bool need_exp = P->need_exp != 0;
        const float *cf = sc.c;
        // some pair can reach t = 0.25 (but not 2): the degree-7 polynomial
        const bool tier7 = need_exp && !tier0;
        ExpForm xf;
        xf.inv_a3 = make_float2(inv_a3, inv_a3);
        xf.nl2a3 = make_float2(-1.4426950408889634f * inv_a3, -1.4426950408889634f * inv_a3);
        xf.tsmall = kExpSmallT;
        xf.r3small = 1.001f * kExpSmallT / inv_a3;
        const float2 inv_a3_2 = make_float2(inv_a3, inv_a3);
        // The reference walks hash cells [i-K-1, i+K+1]^3.  Only the half-cells
        // (cell, octant runs of the vortex order) that can hold a vortex inside
        // the point's box are visited: the box spans K+0.5 cells either side,
        // widened by the hash/NGP rounding bound.  Coordinates below are in
        // half cells.
        const double R = (double)K + 0.5 + P->prune_cells;
        int lo[3], hi[3], rlo[3], rhi[3];
        const double qq[3] = {qx, qy, qz};
        const int cc[3] = {i, j, k};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            rlo[a] = cc[a] - K - 1;
            rhi[a] = cc[a] + K + 1;
            lo[a] = max(max(2 * rlo[a], 0), (int)floor(2.0 * (qq[a] - R)));
            hi[a] = min(min(2 * rhi[a] + 1, 2 * n - 1), (int)floor(2.0 * (qq[a] + R)));
        }
        // A target without a near field (outside the grid and its margin, at
        // infinity, not a number) has no say in the warp's walk: it would
        // stretch the others' box, and an infinite one would put their moments'
        // origin at infinity.  It follows one of them through the walk, and its
        // sums are dropped at the end (a mask of its own in the pair loop made
        // the 1M ring's evaluation 1.5 % longer).
        const bool box = act && lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2] && !isnan(ra.x + ra.y + ra.z);
#pragma unroll
        for (int a = 0; a < 3; a++)
            if (!box) { lo[a] = INT_MAX; hi[a] = INT_MIN; }
        near_lanes = __ballot_sync(0xffffffffu, box);
        {
            const int from = near_lanes ? __ffs(near_lanes) - 1 : 0;
            const float3 other = make_float3(__shfl_sync(0xffffffffu, ra.x, from), __shfl_sync(0xffffffffu, ra.y, from),
                                             __shfl_sync(0xffffffffu, ra.z, from));
            if (!box) ra = other;
        }
        // the warp's box: every such target's box, widened by far more than
        // the rounding of these float bounds (2^-18 of the coordinates' size)
        float spread;  // largest extent of the targets (none: negative)
        {
            float lx = box ? ra.x : INFINITY, ly = box ? ra.y : INFINITY, lz = box ? ra.z : INFINITY;
            float hx = box ? ra.x : -INFINITY, hy = box ? ra.y : -INFINITY, hz = box ? ra.z : -INFINITY;
#pragma unroll
            for (int s2 = 16; s2 > 0; s2 >>= 1) {
                lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, s2));
                ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, s2));
                lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, s2));
                hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, s2));
                hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, s2));
                hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, s2));
            }
            float3 o = make_float3(0.f, 0.f, 0.f);
            if (lx <= hx) o = make_float3(0.5f * (lx + hx), 0.5f * (ly + hy), 0.5f * (lz + hz));
            spread = fmaxf(hx - lx, fmaxf(hy - ly, hz - lz));
            const float mx = ldexpf(fabsf(lx) + fabsf(hx) + cr, -18), my = ldexpf(fabsf(ly) + fabsf(hy) + cr, -18),
                        mz = ldexpf(fabsf(lz) + fabsf(hz) + cr, -18);
            // exp form: records inside [lo + near, hi - near] may lie within
            // a / 4 of a target (1 % margin on a / 4, far above the trigger's)
            const float near = cr - (float)(0.2525 * P->a);
            if (lane == 0) {
                W.box.lo = make_float4(lx - cr - mx, ly - cr - my, lz - cr - mz, near);
                W.box.hi = make_float4(hx + cr + mx, hy + cr + my, hz + cr + mz, 0.f);
                W.box.mid = make_float4(o.x, o.y, o.z, __uint_as_float(near_lanes));
            }
        }
        int ulo[3], uhi[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            ulo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
            uhi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        }
        long long vol = 1;
#pragma unroll
        for (int a = 0; a < 3; a++) vol *= (uhi[a] >= ulo[a]) ? (long long)(uhi[a] - ulo[a] + 1) : 0ll;
        // warp-uniform walk over half-cells: every lane sees the same vortex at
        // once; DEG picks phi's polynomial (one walk per polynomial, so that
        // only one pair loop is live at a time).  The walk does not test a
        // lane's hash-cell range [i-K-1, i+K+1]^3 per run: a vortex inside the
        // lane's box, (K+0.5)h either side of a point of cell i, lies in that
        // range whenever its hash cell differs from its coordinate by less
        // than half a cell, which the rounding bound prune_cells < 1/4 (far
        // beyond float rounding of the relative coordinates) guarantees;
        // otherwise every lane takes its own walk below.
        // Segments: the pair test on the other end only ever drops a vortex
        // that sits at this lane's other end (|rb - r_p|^2 < 1e-24).  Each lane
        // looks for them among the records of the hash cells its other end can
        // fall in (widened by the rounding bound prune_cells), with the pair
        // loop's own arithmetic.  None: the walk needs no test.  Exactly one
        // (the time step's segments: the other end is the segment's own
        // centre): the pair loop drops that record by its index.  More, or an
        // other end near or beyond the grid's faces (vortices hashed from
        // outside wrap around): the position test.
        int seg_mode = 0;
        uint32_t pstar = 0xFFFFFFFFu;
        if (SEG) {
            int found = 0;
            if (box) {
                const double pr = P->prune_cells + 1e-6;
                const double qb[3] = {(double)rb.x * invh, (double)rb.y * invh, (double)rb.z * invh};
                int clo[3], chi[3];
                bool edge = false;
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    // inside: floor(qb - pr) >= 0 and floor(qb + pr) <= n - 1
                    edge = edge || !(qb[a] >= pr && qb[a] < (double)n - pr);
                    clo[a] = (int)floor(qb[a] - pr);
                    chi[a] = (int)floor(qb[a] + pr);
                }
                if (edge) {
                    found = 2;
                } else {
                    for (int kk = clo[2]; kk <= chi[2] && found < 2; kk++)
                        for (int jj = clo[1]; jj <= chi[1] && found < 2; jj++)
                            for (int ii = clo[0]; ii <= chi[0] && found < 2; ii++) {
                                const uint32_t cell = ((uint32_t)kk * n + (uint32_t)jj) * n + (uint32_t)ii;
                                const uint32_t ps = start[cell];
                                if (ps == kEmpty) continue;
                                const uint32_t pe = end[cell];
                                for (uint32_t p = ps; p < pe && found < 2; p++) {
                                    const float4 r = vrec[p];
                                    const float ex = rb.x + (-r.x), ey = rb.y + (-r.y), ez = rb.z + (-r.z);
                                    if (fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < 1e-24f) {
                                        found++;
                                        pstar = p;
                                    }
                                }
                            }
                }
            }
            seg_mode = __any_sync(0xffffffffu, found >= 2) ? 1 : (__any_sync(0xffffffffu, found == 1) ? 2 : 0);
        }
        if (lane == 0) {
            const int cx0 = ulo[0] >> 1;
            W.box.cells = make_int4(cx0, ulo[1], ulo[2], ulo[0]);
            W.box.size = make_int4((uhi[0] >> 1) - cx0 + 1, uhi[1] - ulo[1] + 1, uhi[2] - ulo[2] + 1, uhi[0]);
        }
        __syncwarp();
        auto uniform_walk = [&](auto deg, auto segc) {
            constexpr int D = decltype(deg)::value;
            constexpr int S = decltype(segc)::value;
            const float2 *cfd = D == 0 ? sc.p5 : (D == 7 ? sc.p7 : sc.p4);
            Ring ring;
            // the targets against `recs` records of the ring from slot s0
            auto block = [&](auto full, auto check, uint32_t s0, uint32_t recs) {
                constexpr bool FULL = decltype(full)::value, CHECK = decltype(check)::value;
                pair_block<S, COUNT, FOLD, D, FULL, CHECK>(W, s0, recs >> 1, (COUNT ? box : act) ? cr : -1.0f, ra, rb, pstar, inv_a3_2,
                                                           cfd, xf, sums);
            };
            // The runs of records, one per (cell, y and z halves): the two x
            // halves of a cell are adjacent.  The lanes look up 32 runs at
            // once, and the records of those runs, laid end to end, are taken
            // 32 at a time, each lane finding its record's run by bisection
            // of the running sum of lengths: short runs (a sparse scene has a
            // record or none in most) fill the lanes as long ones do.
            const int runs = W.box.size.x * W.box.size.y * W.box.size.z;
            constexpr int kStep = SPLIT ? kEvalThreads : 32;  // SPLIT: the warps take turns
            for (int base = SPLIT ? 32 * warp : 0; base < runs; base += kStep) {
                const int id = base + lane;
                uint32_t ps = 0, len = 0;
                if (id < runs) {
                    const int4 c0 = W.box.cells, sz = W.box.size;
                    const int row = id / sz.x, ci = c0.x + (id - row * sz.x), k = row / sz.y;
                    const int j2 = c0.y + (row - k * sz.y), k2 = c0.z + k;
                    const uint32_t cell = ((uint32_t)(k2 >> 1) * n + (uint32_t)(j2 >> 1)) * n + (uint32_t)ci;
                    const uint32_t k0 = (cell << 3) | ((uint32_t)(j2 & 1) << 1) | ((uint32_t)(k2 & 1) << 2);
                    const uint32_t cs = start[cell];
                    const uint2 st = *reinterpret_cast<const uint2 *>(sub_start + k0);
                    const uint32_t after = (k0 & 7u) == 6u ? end[cell] : sub_start[k0 + 2];
                    if (cs != kEmpty) {
                        ps = 2 * ci >= c0.w ? st.x : st.y;
                        len = (2 * ci + 1 <= sz.w ? after : st.y) - ps;
                    }
                }
                uint32_t incl = len;
#pragma unroll
                for (int w = 1; w < 32; w <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, w);
                    if (lane >= w) incl += v;
                }
                const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
                const uint32_t shift = ps - (incl - len);  // record = shift of its run + its place
                for (uint32_t at = 0; at < total; at += 32) {
                    const uint32_t place = at + (uint32_t)lane;
                    int run = 0;
#pragma unroll
                    for (int w = 16; w > 0; w >>= 1)
                        if (__shfl_sync(0xffffffffu, incl, run + w - 1) <= place) run += w;
                    const uint32_t rec = __shfl_sync(0xffffffffu, shift, run & 31) + place;
                    // the strength is loaded with the position (one latency
                    // per chunk, not two), also for records the box tests drop
                    float4 r = make_float4(INFINITY, 0.f, 0.f, 0.f), al = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (place < total) {
                        r = vrec[rec];
                        al = valf[rec];
                    }
                    // records outside the warp's box cannot pass any target's
                    // test
                    const float4 blo = W.box.lo, bhi = W.box.hi;
                    const bool keep = r.x >= blo.x && r.x <= bhi.x && r.y >= blo.y && r.y <= bhi.y && r.z >= blo.z &&
                                      r.z <= bhi.z;
                    const unsigned kept = __ballot_sync(0xffffffffu, keep);
                    if (kept == 0u) continue;
                    // exp form: a record farther than that inside the box on
                    // some axis is more than a / 4 (with a margin) from every
                    // target, so no pair with it needs the small-t polynomial;
                    // a block without another record skips the warp's test
                    bool near_chunk = D != 0;
                    if (D == 0) {
                        const bool nr = keep && r.x >= blo.x + blo.w && r.x <= bhi.x - blo.w && r.y >= blo.y + blo.w &&
                                        r.y <= bhi.y - blo.w && r.z >= blo.z + blo.w && r.z <= bhi.z - blo.w;
                        near_chunk = __any_sync(0xffffffffu, nr);
                    }
                    if (keep) {
                        const float4 o = W.box.mid;
                        const uint32_t e = ring.fill + (uint32_t)__popc(kept & ((1u << lane) - 1u));
                        stage_record(W, e, r, al, make_float3(o.x, o.y, o.z), rec);
                    }
                    ring.fill += (uint32_t)__popc(kept);
                    ring.near = ring.near || near_chunk;
                    // The ring never overwrites a record still waiting: before
                    // a chunk fewer than 32 wait, a chunk adds at most 32, and
                    // it holds 64.  The records still waiting after a block all
                    // come from the chunk just staged, so its flag carries over.
                    if (ring.fill - ring.head >= kBlockRecs) {
                        __syncwarp();
                        const uint32_t s0 = (ring.head >> 1) & (kRingSlots - 1);
                        if (D != 0 || ring.near) block(std::true_type{}, std::true_type{}, s0, kBlockRecs);
                        else block(std::true_type{}, std::false_type{}, s0, kBlockRecs);
                        ring.head += kBlockRecs;
                        ring.near = near_chunk && ring.fill != ring.head;
                        __syncwarp();  // the next records may take the slots just read
                    }
                }
            }
            // what is left (fewer than 32), an odd record paired with one outside
            // every box and without strength
            const uint32_t rem = ring.fill - ring.head;
            if (rem != 0) {
                if (lane == 0 && (rem & 1u))
                    stage_record(W, ring.fill, make_float4(-1e18f, -1e18f, -1e18f, 0.f),
                                 make_float4(0.f, 0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f), 0xFFFFFFFEu);
                __syncwarp();
                block(std::false_type{}, std::true_type{}, (ring.head >> 1) & (kRingSlots - 1), rem + (rem & 1u));
            }
        };
        auto walk = [&](auto deg) {
            if constexpr (SEG) {
                if (seg_mode == 1) uniform_walk(deg, std::integral_constant<int, 1>{});
                else if (seg_mode == 2) uniform_walk(deg, std::integral_constant<int, 2>{});
                else uniform_walk(deg, std::integral_constant<int, 0>{});
            } else {
                uniform_walk(deg, std::integral_constant<int, 0>{});
            }
        };
        const bool close = !(spread > (float)(kMaxSpread / invh));
        if (vol > 0 && vol <= kUniformMaxSub && close && P->prune_cells < 0.25) {
            if (tier0) walk(std::integral_constant<int, 0>{});
            else if (tier7) walk(std::integral_constant<int, 7>{});
            else walk(std::integral_constant<int, 4>{});
        } else if (box) {
            // scattered warp (sparse regions): own walk, by rows of cells,
            // whose records are consecutive (SPLIT: the warps take the rows
            // in turn)
            const int x0 = lo[0] >> 1, x1 = hi[0] >> 1, y0 = lo[1] >> 1, z0 = lo[2] >> 1;
            const int ny = (hi[1] >> 1) - y0 + 1, rows = ny * ((hi[2] >> 1) - z0 + 1);
            for (int row = SPLIT ? warp : 0; row < rows; row += SPLIT ? kEvalThreads / 32 : 1) {
                const int jj = y0 + row % ny, kk = z0 + row / ny;
                const uint32_t cell = ((uint32_t)kk * n + (uint32_t)jj) * n;
                uint32_t ps = kEmpty, pe = 0;
                for (int ii = x0; ii <= x1; ii++) {
                    const uint32_t cs = start[cell + ii];
                    if (cs == kEmpty) continue;
                    ps = min(ps, cs);
                    pe = end[cell + ii];
                }
                if (ps == kEmpty) continue;
                cell_pairs<SEG, COUNT>(vrec, valf, ps, pe, true, ra, rb, cr, inv_a3, cf, inv4pia3, need_exp, acc);
            }
        }
    }
    float ab[6] = {sums.ax.x + sums.ax.y, sums.ay.x + sums.ay.y, sums.az.x + sums.az.y,
                   sums.bx.x + sums.bx.y, sums.by.x + sums.by.y, sums.bz.x + sums.bz.y};
    // (the lanes with a near field: segments keep them in a register, which is up
    // to 4 % faster there than reading them back; other points read them back,
    // which is 1 % faster there)
    float ox = 0.f, oy = 0.f, oz = 0.f;
    bool near = false;
    if (K >= 0) {
        __syncwarp();
        ox = W.box.mid.x;
        oy = W.box.mid.y;
        oz = W.box.mid.z;
        near = (((SEG ? near_lanes : __float_as_uint(W.box.mid.w)) >> lane) & 1u) != 0u;
    }
    if constexpr (SPLIT) {
        // the four warps' sums, added in order
        __syncthreads();  // the rings are done with
        float *part = reinterpret_cast<float *>(stage) + lane;
#pragma unroll
        for (int q = 0; q < 9; q++)
            part[(9 * warp + q) * 32] = q < 6 ? ab[q] : (q == 6 ? acc.x : (q == 7 ? acc.y : acc.z));
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < kEvalThreads / 32; w++) {
                const float *from = part + 9 * w * 32;
#pragma unroll
                for (int q = 0; q < 6; q++) ab[q] += from[q * 32];
                acc.x += from[6 * 32];
                acc.y += from[7 * 32];
                acc.z += from[8 * 32];
            }
        }
    }
    if (!COUNT && (!act || (SPLIT && warp != 0))) return;
    // the far field, after the walk: its registers are the pair block's then
    // (the point is read again)
    const uint32_t q = act ? __ldcg(eidx + s) : 0u;
    float3 ra = make_float3(0.f, 0.f, 0.f);
    if (act) ra = rel_pos(eval_a[q], P);
    float ux = 0.f, uy = 0.f, uz = 0.f;
    const double qx = (double)ra.x * invh, qy = (double)ra.y * invh, qz = (double)ra.z * invh;
    const int i = (int)floor(qx), j = (int)floor(qy), k = (int)floor(qz);
    if (i >= 0 && i < n && j >= 0 && j < n && k >= 0 && k < n) {
        const double tx = qx - 0.5, ty = qy - 0.5, tz = qz - 0.5;
        const double fx0 = floor(tx), fy0 = floor(ty), fz0 = floor(tz);
        const int i0 = (int)fx0, j0 = (int)fy0, k0 = (int)fz0;
        const float fx = (float)(tx - fx0), fy = (float)(ty - fy0), fz = (float)(tz - fz0);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int ii = i0 + (c & 1), jj = j0 + ((c >> 1) & 1), kk = k0 + (c >> 2);
            const float wgt = ((c & 1) ? fx : 1.f - fx) * ((c & 2) ? fy : 1.f - fy) * ((c & 4) ? fz : 1.f - fz);
            if (ii >= 0 && ii < n && jj >= 0 && jj < n && kk >= 0 && kk < n) {
                const size_t g = ((size_t)kk * n + jj) * n + ii;
                ux = fmaf(far[g], wgt, ux);
                uy = fmaf(far[C + g], wgt, uy);
                uz = fmaf(far[2 * (size_t)C + g], wgt, uz);
            }
        }
    }
    if (act && (!SPLIT || warp == 0)) {
        const float Ax = ab[0], Ay = ab[1], Az = ab[2], Bx = ab[3], By = ab[4], Bz = ab[5];
        const float sx = ra.x - ox, sy = ra.y - oy, sz = ra.z - oz;
        const float nx = near ? fmaf(Ay, sz, -(Az * sy)) - Bx : 0.f, ny = near ? fmaf(Az, sx, -(Ax * sz)) - By : 0.f,
                    nz = near ? fmaf(Ax, sy, -(Ay * sx)) - Bz : 0.f;
        if (tier0) {
            // exp-form sums carry 4 pi (the reference's literal); the lane's
            // own walk carries the scale of its coefficients
            const float kown = FOLD ? 1.0f : P->inv4pia3_f;
            const float k4 = (float)(1.0 / kFourPi);
            ux = fmaf(nx, k4, fmaf(acc.x, kown, ux));
            uy = fmaf(ny, k4, fmaf(acc.y, kown, uy));
            uz = fmaf(nz, k4, fmaf(acc.z, kown, uz));
        } else if (FOLD) {
            ux += acc.x + nx;
            uy += acc.y + ny;
            uz += acc.z + nz;
        } else {
            const float k = P->inv4pia3_f;
            ux = fmaf(acc.x + nx, k, ux);
            uy = fmaf(acc.y + ny, k, uy);
            uz = fmaf(acc.z + nz, k, uz);
        }
        if (P->status != 0) {
            // zero or non-finite domain edge (one vortex, or all coincident):
            // the cell size is 0 and the sums above are meaningless; the
            // velocity is defined as 0 and pppm_get_domain reports the domain
            ux = 0.f;
            uy = 0.f;
            uz = 0.f;
        }
        if (u) {
            u[q] = (double)ux;
            v[q] = (double)uy;
            w[q] = (double)uz;
        }
        if (uf) {
            uf[3 * (size_t)q] = ux;
            uf[3 * (size_t)q + 1] = uy;
            uf[3 * (size_t)q + 2] = uz;
        }
    }
    if (COUNT) {
        unsigned long long pairs = acc.n + sums.n;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
        if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(pair_count, pairs);
    }
}

// One scene: block b evaluates points [128 b, 128 b + 128) of the order, or
// (SPLIT) [32 b, 32 b + 32).
template <bool SEG, bool COUNT, bool FOLD, bool SPLIT>
__global__ void __launch_bounds__(kEvalThreads, kEvalBlocksPerSM)
eval_kernel(const SmoothSeries sc, const EvalArgs ea) {
    __shared__ WarpMem stage[kEvalThreads / 32];
    eval_points<SEG, COUNT, FOLD, SPLIT>(sc, ea, blockIdx.x, stage);
}

// Several scenes in one launch: block b takes work item work[b] = (scene,
// block of that scene).  The host orders the list so that the blocks of the
// scenes with the most pairs per point come first, which the block scheduler
// then hands out first (longest work first); each point's arithmetic is the
// one-scene kernel's, so results do not depend on the batch.
template <bool SEG, bool COUNT, bool FOLD, bool SPLIT>
__global__ void __launch_bounds__(kEvalThreads, kEvalBlocksPerSM)
eval_batch_kernel(const SmoothSeries sc, const EvalArgs *__restrict__ scenes, const uint2 *__restrict__ work) {
    __shared__ WarpMem stage[kEvalThreads / 32];
    __shared__ EvalArgs sa;  // the block's scene, read from shared memory where used
    const uint2 it = work[blockIdx.x];
    if (threadIdx.x == 0) sa = scenes[it.x];
    __syncthreads();
    eval_points<SEG, COUNT, FOLD, SPLIT>(sc, sa, it.y, stage);
}

// Monomial coefficients of the degree-deg polynomial that interpolates
// phi(t) = (1 - e^-t) / t at the deg + 1 Chebyshev nodes of [0, T] (a near-best
// uniform approximation: relative error 2.6e-9 for degree 4 on [0, 0.25],
// 2e-8 for degree 7 on [0, 2]), by solving the Vandermonde system in FP64.
void phi_chebyshev(int deg, double T, double *c) {
    const double pi = 3.14159265358979323846;
    const int m = deg + 1;
    double V[8][9];
    for (int k = 0; k < m; k++) {
        const double t = 0.5 * T + 0.5 * T * std::cos((2 * k + 1) * pi / (2.0 * m));
        double pw = 1.0;
        for (int q = 0; q < m; q++) { V[k][q] = pw; pw *= t; }
        V[k][m] = -std::expm1(-t) / t;
    }
    for (int col = 0; col < m; col++) {  // Gauss-Jordan elimination, partial pivoting
        int piv = col;
        for (int r = col + 1; r < m; r++)
            if (std::fabs(V[r][col]) > std::fabs(V[piv][col])) piv = r;
        for (int q = 0; q <= m; q++) std::swap(V[col][q], V[piv][q]);
        for (int r = 0; r < m; r++) {
            if (r == col) continue;
            const double f = V[r][col] / V[col][col];
            for (int q = col; q <= m; q++) V[r][q] -= f * V[col][q];
        }
    }
    for (int q = 0; q < m; q++) c[q] = V[q][m] / V[q][q];
}

}  // namespace

// Evaluation keys of M points and their radix sort (the order the eval
// kernel walks); the sorted original indices land in s->esorted_idx.
cudaError_t launch_eval_sort(pppm_scene *s, const float4 *eval_a, uint32_t M) {
    uint32_t *skey = nullptr, *sidx = nullptr;
    prof_begin(s, kStageEvalSort);
    ::pppm::note_launch();
    const int per_cell = s->n <= 256 ? 4 : 2;
    int side = 1;
    while ((1u << side) < s->n * (uint32_t)per_cell) side++;
    eval_keys_kernel<<<(M + 255) / 256, 256, 0, s->stream>>>(eval_a, M, s->dparams, per_cell, side, s->ekey[0],
                                                             s->eidx[0]);
    PPPM_CUDA_TRY(cudaGetLastError());
    const uint32_t bits = 3u * (uint32_t)side;
    PPPM_CUDA_TRY(radix_sort_pairs(s->stream, M, bits, s->ekey, s->eidx, s->hist, &skey, &sidx));
    prof_end(s, kStageEvalSort);
    s->esorted_idx = sidx;
    return cudaSuccess;
}

// The smoothing series of a scene and whether its coefficients are folded.
// With an absolute a (known here) the packed polynomials are in r^3
// (c_q / a^(3q), scaled by 1/(4 pi a^3)) while every coefficient stays a
// normal float far from overflow.  Otherwise (a tied to the cell size of the
// build, known only on the device, or extreme a) they are in t = (r/a)^3 with
// unit scale, and the kernel applies 1/(4 pi a^3) from the device parameters
// once per point.
static bool make_series(const pppm_scene *s, SmoothSeries &sc) {
    memset(&sc, 0, sizeof(sc));
    bool fold = s->prm.a_cells <= 0.0;
    double f4[5], f7[8], f5[6];
    phi_chebyshev(4, 0.25, f4);
    phi_chebyshev(7, 2.0, f7);
    phi_chebyshev(5, 0.5, f5);
    for (int q = 0; q < 6; q++) sc.p5[q] = make_float2((float)f5[q], (float)f5[q]);
    double u4[5], u7[8], k = 1.0;
    if (fold) {
        const double a = s->prm.a;
        k = 1.0 / (kFourPi * a * a * a);
        const double ia3 = 1.0 / (a * a * a);
        double pw = 1.0;
        for (int q = 0; q < 8; q++, pw *= ia3) {
            if (q < 5) u4[q] = k * f4[q] * pw;
            u7[q] = k * f7[q] * pw;
            for (double x : {q < 5 ? u4[q] : 1.0, u7[q]})
                if (!(std::fabs(x) <= 1e30 && std::fabs(x) >= 1e-30)) fold = false;
        }
    }
    if (!fold) k = 1.0;
    for (int q = 0; q < 8; q++) {
        if (q < 5) {
            sc.c[q] = (float)(k * f4[q]);
            const float v4 = fold ? (float)u4[q] : sc.c[q];
            sc.p4[q] = make_float2(v4, v4);
        }
        const float v7 = fold ? (float)u7[q] : (float)(k * f7[q]);
        sc.p7[q] = make_float2(v7, v7);
    }
    return fold;
}

static EvalArgs make_args(pppm_scene *s, const float4 *eval_a, const float4 *eval_b, uint32_t M, double *u, double *v,
                          double *w, float *uf, unsigned long long *pc) {
    EvalArgs a;
    a.eidx = s->esorted_idx;
    a.M = M;
    a.eval_a = eval_a;
    a.eval_b = eval_b;
    a.far = s->far;
    a.start = s->cell_start;
    a.end = s->cell_end;
    a.sub_start = s->sub_start;
    a.vrec = s->vrec;
    a.valf = s->valf;
    a.P = s->dparams;
    a.n = (int)s->n;
    a.K = s->prm.K;
    a.u = u;
    a.v = v;
    a.w = w;
    a.uf = uf;
    a.pair_count = pc;
    return a;
}

// Whether a scene's points are evaluated 32 to a block, its four warps sharing
// their walk: with fewer than about two warps of points for each that the GPU
// holds, the longest walks (the densest part of a scene) set the time, and a
// quarter of a walk is what each warp then does (65,537 points, K = 3: 5.6 ms
// without, 2.6 ms with it).  Without a near field (K < 0) there is no walk to
// share: the interpolation of 200,000 points took 21 us with three idle warps in
// each block, 17 us in whole blocks.
constexpr uint32_t kSplitMaxPoints = 2 * kSMs * kEvalBlocksPerSM * kEvalThreads;
static bool eval_split(int K, uint32_t M) { return K >= 0 && M <= kSplitMaxPoints; }
uint32_t eval_blocks(int K, uint32_t M) {
    const uint32_t per = eval_split(K, M) ? 32 : kEvalThreads;
    return (M + per - 1) / per;
}

template <class F>
static void pick(bool v, F f) {
    if (v) f(std::true_type{});
    else f(std::false_type{});
}

cudaError_t launch_eval(pppm_scene *s, const float4 *eval_a, const float4 *eval_b, int is_segment, uint32_t M,
                        double *u, double *v, double *w, float *uf, int count_pairs) {
    PPPM_CUDA_TRY(launch_eval_sort(s, eval_a, M));
    if (count_pairs) PPPM_CUDA_TRY(cudaMemsetAsync(s->pair_count, 0, sizeof(unsigned long long), s->stream));
    prof_begin(s, kStageEval);
    ::pppm::note_launch();
    const bool seg = (is_segment == 1) && (eval_b != eval_a);
    const bool split = eval_split(s->prm.K, M);
    const unsigned grid = eval_blocks(s->prm.K, M);
    SmoothSeries sc;
    const bool fold = make_series(s, sc);
    const EvalArgs ea = make_args(s, eval_a, eval_b, M, u, v, w, uf, count_pairs ? s->pair_count : nullptr);
    pick(seg, [&](auto a) {
        pick(count_pairs != 0, [&](auto b) {
            pick(fold, [&](auto c) {
                pick(split, [&](auto d) {
                    eval_kernel<decltype(a)::value, decltype(b)::value, decltype(c)::value, decltype(d)::value>
                        <<<grid, kEvalThreads, 0, s->stream>>>(sc, ea);
                });
            });
        });
    });
    prof_end(s, kStageEval);
    return cudaGetLastError();
}

// Batched evaluation (pppm_batch_run): the arguments of each item's scene
// after its sort, and whether all items can share one launch (the same
// series, segment mode and folding).
cudaError_t eval_batch_prepare(pppm_scene *s, const float4 *eval_a, const float4 *eval_b, int is_segment, uint32_t M,
                               double *u, double *v, double *w, EvalArgs *args, EvalMode *mode) {
    PPPM_CUDA_TRY(launch_eval_sort(s, eval_a, M));
    SmoothSeries sc;
    mode->fold = make_series(s, sc);
    static_assert(sizeof(SmoothSeries) <= sizeof(mode->series), "series bytes");
    memcpy(mode->series, &sc, sizeof(sc));
    mode->seg = (is_segment == 1) && (eval_b != eval_a);
    mode->split = eval_split(s->prm.K, M);
    *args = make_args(s, eval_a, eval_b, M, u, v, w, nullptr, nullptr);
    return cudaSuccess;
}

// One launch over a device work list of `blocks` (scene, block) items for
// scenes that share `mode`.
cudaError_t launch_eval_batch(const EvalMode &mode, const EvalArgs *args_dev, const uint2 *work_dev, uint32_t blocks,
                              cudaStream_t st) {
    if (!blocks) return cudaSuccess;
    SmoothSeries sc;
    memcpy(&sc, mode.series, sizeof(sc));
    ::pppm::note_launch();
    pick(mode.seg, [&](auto a) {
        pick(mode.fold, [&](auto c) {
            pick(mode.split, [&](auto d) {
                eval_batch_kernel<decltype(a)::value, false, decltype(c)::value, decltype(d)::value>
                    <<<blocks, kEvalThreads, 0, st>>>(sc, args_dev, work_dev);
            });
        });
    });
    return cudaGetLastError();
}

}  // namespace pppm
