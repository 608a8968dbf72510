// dev_field.cuh -- fused refractive-index evaluation: n(p) and grad n(p) in one call.
//
// The reference evaluates RIF and dRIF separately, twice per leapfrog step
// (renderer/src/scene.cpp:323-330) plus once more for the optical length (scene.cpp:416).
// All three evaluations after a step are at the same point p', and the next step starts at that
// point again, so the march keeps (n, grad n) of its current position and a step costs one
// fused evaluation.
//
// Gap gating (renderer/include/rif_base.h:104-137, cuda_scene.cuh:463-481): outside
// sgap <= x <= egap the index is n_o and the gradient zero.
#pragma once
#include <climits>

#include "dev_math.cuh"
#include "kparams.h"

namespace smp {

static constexpr float kEps = 1.19209290e-07f;    // M_EPSILON (constants.h)

// Cylindrical Bessel mode about the -x axis (scene.cpp:206-257, fixed axes rif_base.h:146-148):
//   n = n_o + n_max*s*J_m(k r) cos(m phi),  phi = atan2(y, z), r = |(y, z)|
//   dn/dy = n_max*s*(J_m' k y/r cos(m phi) - J_m m sin(m phi) z/r^2)
//   dn/dz = n_max*s*(J_m' k z/r cos(m phi) + J_m m sin(m phi) y/r^2),  J_m' = (m/kr) J_m - J_{m+1}
// cos(m phi), sin(m phi) come from (z/r + i y/r)^m instead of atan2 + sincos.
// Below r = M_EPSILON the gradient uses y = z = r = M_EPSILON as the reference does.
template <int M>
__device__ __forceinline__ void bessel_field_any(const FieldParams &F, const float4 *tab, float3 p, float s, float &n, float3 &g) {
    float y = p.y, z = p.z;
    const float r2 = fmaf(y, y, z * z);
    float rs = rsqrt_fast(r2);                 // +inf at r2 = 0
    const float A = F.amp * s;
    float jm, jm1;
    if (r2 * rs >= kEps) {                     // off the axis (false for r2 = 0: 0 * inf is NaN)
        const float r = r2 * rs;
        bessel_pair_table_t<M>(tab, F.bint, F.kb * r, F.k_r * r, jm, jm1);
        if (M == 0) {
            // grad = A k J_0'(kr) (0, y, z)/r = -A k J_1(kr) (0, y, z)/r
            n = fmaf(A, jm, F.n_o);
            const float w = -(A * F.k_r) * jm1 * rs;
            g = f3(0.0f, w * y, w * z);
        } else if (M == 1) {
            // n = n_o + A J_1(kr) z/r; with J_1' = J_1/(kr) - J_2 the gradient reduces to
            // dn/dy = -A k J_2(kr) y z/r^2,  dn/dz = A J_1(kr)/r - A k J_2(kr) z^2/r^2
            const float aj = A * jm * rs;
            n = fmaf(aj, z, F.n_o);
            const float wz = (A * F.k_r) * jm1 * (rs * rs) * z;
            g = f3(0.0f, -wz * y, fmaf(-wz, z, aj));
        } else {
            const float c = z * rs, sn = y * rs;
            const float cm = fmaf(c, c, -sn * sn), sm = 2.0f * c * sn;
            n = fmaf(A * jm, cm, F.n_o);
            const float djm = fmaf(float(M) * F.inv_k * rs, jm, -jm1);
            const float a1 = A * djm * F.k_r * rs * cm;
            const float a2 = A * jm * float(M) * sm * rs * rs;
            g = f3(0.0f, fmaf(a1, y, -a2 * z), fmaf(a1, z, a2 * y));
        }
        return;
    }
    // on or next to the axis: the value at r, the gradient from y = z = r = M_EPSILON
    // (scene.cpp:229-234); at r = 0, phi = atan2(0, 0) = 0
    float r = r2 > 0.0f ? r2 * rs : 0.0f;
    float cm = 1.0f, sm = 0.0f;
    if (M > 0 && r2 > 0.0f) {
        const float c = z * rs, sn = y * rs;
        if (M == 1) { cm = c; sm = sn; }
        else { cm = fmaf(c, c, -sn * sn); sm = 2.0f * c * sn; }
    }
    bessel_pair_table<M>(tab, F.bint, F.binv_h, F.k_r * r, jm, jm1);
    n = fmaf(A * jm, cm, F.n_o);
    y = kEps; z = kEps; r = kEps; rs = 1.0f / kEps;
    bessel_pair_table<M>(tab, F.bint, F.binv_h, F.k_r * kEps, jm, jm1);
    // J_m'(kr) = (m/kr) J_m - J_{m+1}, with 1/(kr) = rs/k
    const float djm = (M == 0) ? -jm1 : fmaf(float(M) * F.inv_k * rs, jm, -jm1);
    const float a1 = A * djm * F.k_r * rs * cm;            // radial part / r
    const float a2 = (M == 0) ? 0.0f : A * jm * float(M) * sm * rs * rs;
    g = f3(0.0f, fmaf(a1, y, -a2 * z), fmaf(a1, z, a2 * y));
}

template <int M>
static __device__ __noinline__ float4 bessel_field_rare(const FieldParams &F, const float4 *tab, float3 p, float s) {
    float n;
    float3 g;
    bessel_field_any<M>(F, tab, p, s, n, g);
    return make_float4(g.x, g.y, g.z, n);
}

// The Bessel table as the march reads it. A plain pointer: entry i is tab[2i], tab[2i + 1]. RepTable<R>:
// R copies of every 16-byte half side by side in shared memory, lane l reading copy l mod R. The lanes
// of a warp look up unrelated radii, so the plain table's 16-byte loads collide in banks (the eight lanes
// a wavefront serves share four 16-byte groups: about 14 wavefronts a load, and the L1/shared-memory
// path at 86 % of its peak bounded the march kernel). With four copies two of the eight lanes share a
// group: eight wavefronts.
template <int R> struct RepTable {
    const float4 *p;           // this lane's copy of entry 0
};
__device__ __forceinline__ void tab_load(const float4 *tab, unsigned i, float4 &a, float4 &b) {
    a = tab[2 * i];
    b = tab[2 * i + 1];
}
template <int R> __device__ __forceinline__ void tab_load(const RepTable<R> &tab, unsigned i, float4 &a, float4 &b) {
    a = tab.p[2 * R * i];
    b = tab.p[2 * R * i + R];
}
// the plain table, for the rare paths
__device__ __forceinline__ const float4 *tab_plain(const FieldParams &, const float4 *tab) { return tab; }
template <int R> __device__ __forceinline__ const float4 *tab_plain(const FieldParams &F, const RepTable<R> &) { return F.btab; }

// (J_M, J_{M+1}) from the table at the coordinate t = k r / h, with no test on the way: the interval is
// clamped to the table, and the caller redoes a point whose t is not below bend (or not a number).
template <class TAB>
__device__ __forceinline__ void bessel_pair_clamped(const FieldParams &F, const TAB &tab, float t, float &jm, float &jm1) {
    const float tb = __fadd_rd(t, 8388608.0f);
    const unsigned i = min(unsigned(__float_as_int(tb) - 0x4B000000), unsigned(F.bint - 1));
    const float f = t - (tb - 8388608.0f);
    float4 a, b;
    tab_load(tab, i, a, b);
    jm = fmaf(fmaf(fmaf(a.w, f, a.z), f, a.y), f, a.x);
    jm1 = fmaf(fmaf(fmaf(b.w, f, b.z), f, b.y), f, b.x);
}

// n and grad n at (y, z) off the axis from J_M and J_{M+1}, 1/r and A = n_max s
template <int M>
__device__ __forceinline__ void bessel_result(const FieldParams &F, float A, float y, float z, float rs, float jm, float jm1,
                                              float &n, float3 &g) {
    if (M == 0) {
        // grad = A k J_0'(kr) (0, y, z)/r = -A k J_1(kr) (0, y, z)/r
        n = fmaf(A, jm, F.n_o);
        const float w = -(A * F.k_r) * jm1 * rs;
        g = f3(0.0f, w * y, w * z);
    } else if (M == 1) {
        // n = n_o + A J_1(kr) z/r; with J_1' = J_1/(kr) - J_2 the gradient reduces to
        // dn/dy = -A k J_2(kr) y z/r^2,  dn/dz = A J_1(kr)/r - A k J_2(kr) z^2/r^2
        const float aj = A * jm * rs;
        n = fmaf(aj, z, F.n_o);
        const float wz = (A * F.k_r) * jm1 * (rs * rs) * z;
        g = f3(0.0f, -wz * y, fmaf(-wz, z, aj));
    } else {
        const float c = z * rs, sn = y * rs;
        const float cm = fmaf(c, c, -sn * sn), sm = 2.0f * c * sn;
        n = fmaf(A * jm, cm, F.n_o);
        const float djm = fmaf(float(M) * F.inv_k * rs, jm, -jm1);
        const float a1 = A * djm * F.k_r * rs * cm;
        const float a2 = A * jm * float(M) * sm * rs * rs;
        g = f3(0.0f, fmaf(a1, y, -a2 * z), fmaf(a1, z, a2 * y));
    }
}

// The same field in one straight line, for the march. A point off the axis and inside the table --
// practically all of them -- needs no branch; the two tests that find the others are off the step's
// dependency chain and share one branch at its end. (Each test as a branch of its own before the
// lookup held the whole chain up until it resolved: the lone tail photon's step took 295 cycles.)
template <int M, class TAB>
__device__ __forceinline__ void bessel_field_ng(const FieldParams &F, const TAB &tab, float3 p, float s, float &n, float3 &g) {
    const float y = p.y, z = p.z;
    const float r2 = fmaxf(fmaf(y, y, z * z), 1e-20f);       // a point below is rare anyway: r < kEps
    const float rs = rsqrt_fast(r2);
    const float A = F.amp * s;
    const float r = r2 * rs, t = F.kb * r;
    float jm, jm1;
    bessel_pair_clamped(F, tab, t, jm, jm1);
    bessel_result<M>(F, A, y, z, rs, jm, jm1, n, g);
    if (!((r >= kEps) & (t < F.bend))) {
        const float4 q = bessel_field_rare<M>(F, tab_plain(F, tab), p, s);
        n = q.w;
        g = f3(q.x, q.y, q.z);
    }
}

// gap gating (rif_base.h:104-137): n_o and no gradient outside sgap <= x <= egap
__device__ __forceinline__ bool in_gap(const FieldParams &F, float3 p) { return p.x > F.egap || p.x < F.sgap; }

// In the gaps the amplitude is zeroed instead of branching: n = n_o + 0 and grad n = 0 exactly,
// and every lane runs the same instructions.
template <int M, class TAB>
__device__ __forceinline__ void bessel_field(const FieldParams &F, const TAB &tab, float3 p, float s, float &n, float3 &g) {
    bessel_field_ng<M>(F, tab, p, in_gap(F, p) ? 0.0f : s, n, g);
}

// Plane waves (not in the reference): n = n_o + sum_i a_i sin(k_i.p - tau + phase_i)
__device__ __forceinline__ void wave_field_ng(const FieldParams &F, float3 p, float tau, float &n, float3 &g) {
    float acc = 0.0f;
    float3 gg = f3(0.0f, 0.0f, 0.0f);
    // unrolled, so that every wave's constants are operands of their instructions; with a run-time index
    // each is a constant-memory load on the step's dependency chain
#pragma unroll
    for (int i = 0; i < SMP_MAX_WAVES; ++i) {
        if (i >= F.n_waves) break;
        float ph = F.wk[i][0] * p.x + F.wk[i][1] * p.y + F.wk[i][2] * p.z - tau + F.wphase[i];
        float sn, cs;
        sincos_near(ph, sn, cs);
        acc = fmaf(F.wamp[i], sn, acc);
        float ac = F.wamp[i] * cs;
        gg.x = fmaf(ac, F.wk[i][0], gg.x);
        gg.y = fmaf(ac, F.wk[i][1], gg.y);
        gg.z = fmaf(ac, F.wk[i][2], gg.z);
    }
    n = F.n_o + acc;
    g = gg;
}

__device__ __forceinline__ void wave_field(const FieldParams &F, float3 p, float tau, float &n, float3 &g) {
    if (in_gap(F, p)) {
        n = F.n_o;
        g = f3(0.0f, 0.0f, 0.0f);
        return;
    }
    wave_field_ng(F, p, tau, n, g);
}

// Spherical point sources on two arcs (scene.cpp:139-195, rif_sources.h:156-198):
//   n = n_o + n_scaling * sum_c w_c sum_src cos(k r c + phase)/r,  w_c = 4(-1)^(c+1)/((c pi)^2 nsrc)
//   grad = n_scaling * sum_c w_c sum_src -(cos(k r c + ph) + k r c sin(k r c + ph))/r^3 (p - centre)
// All lanes of a warp read the same centre each iteration (broadcast loads through L1).
__device__ __forceinline__ void sources_field(const FieldParams &F, float3 p, float &n, float3 &g) {
    if (p.x > F.egap || p.x < F.sgap) {
        n = F.n_o;
        g = f3(0.0f, 0.0f, 0.0f);
        return;
    }
    float rif = 0.0f;
    float3 dn = f3(0.0f, 0.0f, 0.0f);
    const float pi = 3.14159265358979f;
    for (int c = 1; c <= F.n_coeff; ++c) {
        float sf = ((c & 1) ? 4.0f : -4.0f) / (float(c) * pi * float(c) * pi * float(F.nsources));
        float trif = 0.0f;
        float3 tdn = f3(0.0f, 0.0f, 0.0f);
        for (int arc = 0; arc < 2; ++arc) {
            if (!(arc == 0 ? F.active1 : F.active2)) continue;
            const float ph = arc == 0 ? F.phase1 : F.phase2;
            const float4 *cen = F.centers + arc * F.nsources;
            for (int k = 0; k < F.nsources; ++k) {
                float4 q = __ldg(cen + k);
                float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                float rr2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                float ir = rsqrtf(rr2);
                float r = rr2 * ir;
                float krc = F.k_r * r * float(c);
                float sn, cs;
                sincos_near(krc + ph, sn, cs);
                trif = fmaf(cs, ir, trif);
                float ct = -fmaf(krc, sn, cs) * ir * ir * ir;
                tdn.x = fmaf(ct, dx, tdn.x);
                tdn.y = fmaf(ct, dy, tdn.y);
                tdn.z = fmaf(ct, dz, tdn.z);
            }
        }
        rif = fmaf(trif, sf, rif);
        dn = add(dn, mul(tdn, sf));
    }
    n = fmaf(F.n_scaling, rif, F.n_o);
    g = mul(dn, F.n_scaling);
}

// Tricubic B-spline (spline.h:33-62 kernels, :308-356 value/gradient) with the mirror rule of the
// reference's 1-D/2-D evaluators for taps outside the grid. The B-spline weights sum to 1 and
// their derivatives to 0, so the coefficients are stored as offsets from their mean:
// n = base + sum(delta w), grad n = sum(delta w'). Summing the raw coefficients (~1.33) in FP32,
// as the reference does, cancels about four digits of a 1e-3 gradient signal.
__device__ __forceinline__ int spline_wrap(int i, int n) {
    if (unsigned(i) < unsigned(n)) return i;     // inside the grid: the common case
    int m = 2 * n - 2;
    int w = i % m;
    if (w < 0) w += m;
    return w >= n ? m - w : w;
}
// f = t - floor(t): taps at floor(t)-1 .. floor(t)+2, offsets d = t - i in (1,2], (0,1], (-1,0], (-2,-1]
__device__ __forceinline__ void bspline_weights_f(float f, float w[4], float dw[4]) {
    float f2 = f * f, f3v = f2 * f;
    float g = 1.0f - f;
    w[0] = g * g * g * (1.0f / 6.0f);
    w[1] = (2.0f / 3.0f) - f2 + 0.5f * f3v;
    w[2] = (2.0f / 3.0f) - g * g + 0.5f * g * g * g;
    w[3] = f3v * (1.0f / 6.0f);
    dw[0] = -0.5f * g * g;
    dw[1] = (1.5f * f - 2.0f) * f;
    dw[2] = -(1.5f * g - 2.0f) * g;
    dw[3] = 0.5f * f2;
}
__device__ __forceinline__ void bspline_weights(float t, float w[4], float dw[4]) {
    bspline_weights_f(t - floorf(t), w, dw);
}
// Cell and offset of a grid coordinate without conversions: a round-down add of 2^23 + 64 leaves
// floor(t) + 64 in the low bits. A t outside [-64, 2^23) or not a number gives a cell far off any grid.
__device__ __forceinline__ int spline_cell_of(float t, float &f) {
    const float tb = __fadd_rd(t, 8388672.0f);
    f = t - (tb - 8388672.0f);
    return __float_as_int(tb) - (0x4B000000 + 64);
}
// The march kernel of the slot pool stages one brick of the coefficient grid in shared memory (the
// x-tap quads of kSplineBrick^3 cells and their rows' one-cell apron below and two-cell apron above
// in y and z: kSplineBrick x (kSplineBrick + 3)^2 quads) and passes it as `brick`: entry 0 holds the
// brick's first cell (x, y, z) as ints and a valid flag, the quads follow, x fastest. A point whose
// 4x4x4 taps lie in the brick reads them there; any other point (and every kernel without a brick,
// brick == nullptr) reads the global quads. The values and sums are the same either way.
static constexpr int kSplineBrick = 16;
static constexpr int kSplineBrickRows = kSplineBrick + 3;
static constexpr int kSplineBrickQuads = kSplineBrick * kSplineBrickRows * kSplineBrickRows;

// One (y, z) row of the 4x4x4 taps: its four x taps times the x weights, into the value and gradient
// sums. Every spline evaluation adds its sixteen rows through here in the same order.
struct SplineW { float wx[4], dx[4], wy[4], dy[4], wz[4], dz[4]; };
struct SplineSum { float v, gx, gy, gz; };
__device__ __forceinline__ void spline_row(const SplineW &w, int b, int c, float r0, float r1, float r2, float r3,
                                           SplineSum &s) {
    const float sv = r0 * w.wx[0] + r1 * w.wx[1] + r2 * w.wx[2] + r3 * w.wx[3];
    const float sd = r0 * w.dx[0] + r1 * w.dx[1] + r2 * w.dx[2] + r3 * w.dx[3];
    const float wyz = w.wy[b] * w.wz[c];
    s.v = fmaf(sv, wyz, s.v);
    s.gx = fmaf(sd, wyz, s.gx);
    s.gy = fmaf(sv, w.dy[b] * w.wz[c], s.gy);
    s.gz = fmaf(sv, w.wy[b] * w.dz[c], s.gz);
}
__device__ __forceinline__ void spline_weights(float tx, float ty, float tz, SplineW &w) {
    bspline_weights(tx, w.wx, w.dx);
    bspline_weights(ty, w.wy, w.dy);
    bspline_weights(tz, w.wz, w.dz);
}
__device__ __forceinline__ void spline_result(const FieldParams &F, const SplineSum &s, float &n, float3 &g) {
    n = F.spline_base + s.v;
    g = f3(s.gx * F.xres[0], s.gy * F.xres[1], s.gz * F.xres[2]);
}

// The sixteen tap rows of one grid cell, kept in registers while a march stays in it. An ER step
// is a tenth of a cell or less on the usual grids (0.01 mm steps on 64 to 96 nodes over 10 mm), so
// a march reads its taps once per cell instead of once per step.
struct SplineCell {
    int x, y, z;
    float4 q[16];
    __device__ __forceinline__ void clear() {                      // no cell
        x = y = z = INT_MIN;
#pragma unroll
        for (int i = 0; i < 16; ++i) q[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
};

// The tap rows of cell (x, y, z), sixteen independent 16-byte loads: a cell of the grid or the one next
// to it on any side (a step that overshoots a face is evaluated there before it is taken back).
__device__ __forceinline__ bool spline_on_quads(const FieldParams &F, int x, int y, int z) {
    return (F.coeff4 != nullptr) & (unsigned(x + 1) < unsigned(F.N[0] + 2)) & (unsigned(y + 1) < unsigned(F.N[1] + 2)) &
           (unsigned(z + 1) < unsigned(F.N[2] + 2));
}
__device__ __forceinline__ void spline_rows(const FieldParams &F, int x, int y, int z, float4 q[16]) {
    int iy[4], iz[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        iy[a] = spline_wrap(y - 1 + a, F.N[1]) * F.qrow;
        iz[a] = spline_wrap(z - 1 + a, F.N[2]) * F.N[1] * F.qrow;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int b = 0; b < 4; ++b) q[4 * c + b] = __ldg(F.coeff4 + (iz[c] + iy[b] + x));
}

// taps read one by one: a point off the grid in x, or a plan without quads. Returns (grad n, n).
static __device__ __noinline__ float4 spline_taps(const FieldParams &F, float3 p) {
    const float tx = (p.x - F.xmin[0]) * F.xres[0], ty = (p.y - F.xmin[1]) * F.xres[1], tz = (p.z - F.xmin[2]) * F.xres[2];
    SplineW w;
    spline_weights(tx, ty, tz, w);
    const int bx = int(floorf(tx)) - 1, by = int(floorf(ty)) - 1, bz = int(floorf(tz)) - 1;
    const int N0 = F.N[0], N1 = F.N[1], N2 = F.N[2];
    int ix[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) ix[a] = spline_wrap(bx + a, N0);
    SplineSum s = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float *row = F.coeff + spline_wrap(bz + c, N2) * N0 * N1 + spline_wrap(by + b, N1) * N0;
            spline_row(w, b, c, __ldg(row + ix[0]), __ldg(row + ix[1]), __ldg(row + ix[2]), __ldg(row + ix[3]), s);
        }
    float n;
    float3 g;
    spline_result(F, s, n, g);
    return make_float4(g.x, g.y, g.z, n);
}

__device__ __forceinline__ bool spline_in_gap(const FieldParams &F, float3 p) { return p.x > F.egap || p.x < F.sgap; }

// n and grad n with the taps of the march's current cell kept in C. A straight line but for the reload:
// a point off the grid is redone with the taps one by one at the end.
__device__ __forceinline__ void spline_field_cell(const FieldParams &F, SplineCell &C, float3 p, float &n, float3 &g) {
    float fx, fy, fz;
    const int x = spline_cell_of((p.x - F.xmin[0]) * F.xres[0], fx), y = spline_cell_of((p.y - F.xmin[1]) * F.xres[1], fy),
              z = spline_cell_of((p.z - F.xmin[2]) * F.xres[2], fz);
    const bool on = spline_on_quads(F, x, y, z);
    if (on & ((x != C.x) | (y != C.y) | (z != C.z))) {
        spline_rows(F, x, y, z, C.q);
        C.x = x; C.y = y; C.z = z;
    }
    SplineW w;
    bspline_weights_f(fx, w.wx, w.dx);
    bspline_weights_f(fy, w.wy, w.dy);
    bspline_weights_f(fz, w.wz, w.dz);
    SplineSum s = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float4 q = C.q[4 * c + b];
            spline_row(w, b, c, q.x, q.y, q.z, q.w, s);
        }
    spline_result(F, s, n, g);
    if (!on) {
        const float4 r = spline_taps(F, p);
        n = r.w;
        g = f3(r.x, r.y, r.z);
    }
}

__device__ __forceinline__ void spline_field(const FieldParams &F, const float4 *brick, float3 p, float &n, float3 &g) {
    if (spline_in_gap(F, p)) {
        n = F.n_o;
        g = f3(0.0f, 0.0f, 0.0f);
        return;
    }
    if (brick == nullptr) {
        SplineCell C;
        C.clear();
        spline_field_cell(F, C, p, n, g);
        return;
    }
    const float tx = (p.x - F.xmin[0]) * F.xres[0], ty = (p.y - F.xmin[1]) * F.xres[1], tz = (p.z - F.xmin[2]) * F.xres[2];
    SplineW w;
    spline_weights(tx, ty, tz, w);
    const int bx = int(floorf(tx)) - 1, by = int(floorf(ty)) - 1, bz = int(floorf(tz)) - 1;
    // the staged brick holds every tap when floor(t) lies in its cells on all three axes (and on
    // the grid)
    const int4 h = *reinterpret_cast<const int4 *>(brick);
    const int ox = bx + 1 - h.x, oy = by + 1 - h.y, oz = bz + 1 - h.z;
    SplineSum s = {0.0f, 0.0f, 0.0f, 0.0f};
    if (h.w != 0 && unsigned(ox) < unsigned(kSplineBrick) && unsigned(oy) < unsigned(kSplineBrick) &&
        unsigned(oz) < unsigned(kSplineBrick) && unsigned(bx + 1) < unsigned(F.N[0]) && unsigned(by + 1) < unsigned(F.N[1]) &&
        unsigned(bz + 1) < unsigned(F.N[2])) {
        const float4 *bq = brick + 1 + (oz * kSplineBrickRows + oy) * kSplineBrick + ox;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const float4 q = bq[(c * kSplineBrickRows + b) * kSplineBrick];
                spline_row(w, b, c, q.x, q.y, q.z, q.w, s);
            }
    } else if (spline_on_quads(F, bx + 1, by + 1, bz + 1)) {
        float4 q[16];
        spline_rows(F, bx + 1, by + 1, bz + 1, q);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int b = 0; b < 4; ++b) spline_row(w, b, c, q[4 * c + b].x, q[4 * c + b].y, q[4 * c + b].z, q[4 * c + b].w, s);
    } else {
        const float4 r = spline_taps(F, p);
        n = r.w;
        g = f3(r.x, r.y, r.z);
        return;
    }
    spline_result(F, s, n, g);
}

// Bessel mode m in 0..2 chosen at run time, one branch-free path for all orders (lanes of a warp
// may hold photons of different instances and orders): cos/sin(m phi) by selects from
// (z + iy)/r, J_m' = (m/kr) J_m - J_{m+1}; beyond the table the order-specific formulas.
__device__ __forceinline__ void bessel_field_rt_any(const FieldParams &F, const float4 *tab, float3 p, float s, float &n, float3 &g) {
    const int M = F.mode;
    const float A = F.amp * s;
    float y = p.y, z = p.z;
    const float r2 = fmaf(y, y, z * z);
    float rs = rsqrt_fast(r2);                 // +inf at r2 = 0
    float r = r2 > 0.0f ? r2 * rs : 0.0f;
    float cm = 1.0f, sm = 0.0f;
    if (r2 > 0.0f) {
        const float c = z * rs, sn = y * rs;
        cm = M == 0 ? 1.0f : (M == 1 ? c : fmaf(c, c, -sn * sn));
        sm = M == 0 ? 0.0f : (M == 1 ? sn : 2.0f * c * sn);
    }
    float jm, jm1;
    const float t = F.kb * r;
    if (t < float(F.bint)) {
        const float tb = __fadd_rd(t, 8388608.0f);
        const int i = __float_as_int(tb) - 0x4B000000;
        const float f = t - (tb - 8388608.0f);
        const float4 a = tab[2 * i], b = tab[2 * i + 1];
        jm = fmaf(fmaf(fmaf(a.w, f, a.z), f, a.y), f, a.x);
        jm1 = fmaf(fmaf(fmaf(b.w, f, b.z), f, b.y), f, b.x);
    } else if (M == 0) {
        bessel_pair<0>(F.k_r * r, jm, jm1);
    } else if (M == 1) {
        bessel_pair<1>(F.k_r * r, jm, jm1);
    } else {
        bessel_pair<2>(F.k_r * r, jm, jm1);
    }
    n = fmaf(A * jm, cm, F.n_o);
    if (!(r >= kEps)) {                        // the gradient's near-axis substitution (scene.cpp:229-234)
        y = kEps; z = kEps; r = kEps; rs = 1.0f / kEps;
        if (M == 0) bessel_pair_table<0>(tab, F.bint, F.binv_h, F.k_r * kEps, jm, jm1);
        else if (M == 1) bessel_pair_table<1>(tab, F.bint, F.binv_h, F.k_r * kEps, jm, jm1);
        else bessel_pair_table<2>(tab, F.bint, F.binv_h, F.k_r * kEps, jm, jm1);
    }
    const float fm = float(M);
    const float djm = fmaf(fm * F.inv_k * rs, jm, -jm1);
    const float a1 = A * djm * F.k_r * rs * cm;
    const float a2 = A * jm * fm * sm * rs * rs;
    g = f3(0.0f, fmaf(a1, y, -a2 * z), fmaf(a1, z, a2 * y));
}
static __device__ __noinline__ float4 bessel_field_rt_rare(const FieldParams &F, const float4 *tab, float3 p, float s) {
    float n;
    float3 g;
    bessel_field_rt_any(F, tab, p, s, n, g);
    return make_float4(g.x, g.y, g.z, n);
}
__device__ __forceinline__ void bessel_rt_result(const FieldParams &F, int M, float A, float y, float z, float rs, float jm,
                                                 float jm1, float &n, float3 &g) {
    const float c = z * rs, sn = y * rs;
    const float cm = M == 0 ? 1.0f : (M == 1 ? c : fmaf(c, c, -sn * sn));
    const float sm = M == 0 ? 0.0f : (M == 1 ? sn : 2.0f * c * sn);
    n = fmaf(A * jm, cm, F.n_o);
    const float fm = float(M);
    const float djm = fmaf(fm * F.inv_k * rs, jm, -jm1);
    const float a1 = A * djm * F.k_r * rs * cm;
    const float a2 = A * jm * fm * sm * rs * rs;
    g = f3(0.0f, fmaf(a1, y, -a2 * z), fmaf(a1, z, a2 * y));
}
// in one straight line, as bessel_field_ng
template <class TAB>
__device__ __forceinline__ void bessel_field_rt_ng(const FieldParams &F, const TAB &tab, float3 p, float s, float &n, float3 &g) {
    const int M = F.mode;
    const float A = F.amp * s;
    const float y = p.y, z = p.z;
    const float r2 = fmaxf(fmaf(y, y, z * z), 1e-20f);
    const float rs = rsqrt_fast(r2);
    const float r = r2 * rs, t = F.kb * r;
    float jm, jm1;
    bessel_pair_clamped(F, tab, t, jm, jm1);
    bessel_rt_result(F, M, A, y, z, rs, jm, jm1, n, g);
    if (!((r >= kEps) & (t < F.bend))) {
        const float4 q = bessel_field_rt_rare(F, tab_plain(F, tab), p, s);
        n = q.w;
        g = f3(q.x, q.y, q.z);
    }
}

// Bessel mode m >= 3 (scene.cpp:206-257 take any integer order through jn(mode, .)): J_m and J_m+1
// from the per-plan table, which the host sizes to cover the whole box (k r <= 128, checked when the
// plan is made; a point beyond it reads the table's last interval); cos(m phi), sin(m phi) as
// ((z + i y)/r)^m by m - 1 complex products.
template <class TAB>
__device__ __forceinline__ void bessel_field_n_ng(const FieldParams &F, const TAB &tab, float3 p, float s, float &n, float3 &g) {
    const int M = F.mode;
    const float A = F.amp * s;
    float y = p.y, z = p.z;
    const float r2 = fmaf(y, y, z * z);
    float rs = rsqrt_fast(r2);                 // +inf at r2 = 0
    float r = r2 > 0.0f ? r2 * rs : 0.0f;
    float cm = 1.0f, sm = 0.0f;
    if (r2 > 0.0f) {
        const float c = z * rs, sn = y * rs;
        cm = c; sm = sn;
        for (int k = 1; k < M; ++k) {
            const float t = fmaf(cm, c, -sm * sn);
            sm = fmaf(cm, sn, sm * c);
            cm = t;
        }
    }
    auto lookup = [&](float x, float &jm, float &jm1) {
        float t = fminf(x * F.binv_h, float(F.bint) - 1.0f / 64.0f);
        const float tb = __fadd_rd(t, 8388608.0f);
        const int i = __float_as_int(tb) - 0x4B000000;
        const float f = t - (tb - 8388608.0f);
        float4 a, b;
        tab_load(tab, unsigned(i), a, b);
        jm = fmaf(fmaf(fmaf(a.w, f, a.z), f, a.y), f, a.x);
        jm1 = fmaf(fmaf(fmaf(b.w, f, b.z), f, b.y), f, b.x);
    };
    float jm, jm1;
    lookup(F.k_r * r, jm, jm1);
    n = fmaf(A * jm, cm, F.n_o);
    if (!(r >= kEps)) {                        // the gradient's near-axis substitution (scene.cpp:229-234)
        y = kEps; z = kEps; r = kEps; rs = 1.0f / kEps;
        lookup(F.k_r * kEps, jm, jm1);
    }
    const float fm = float(M);
    const float djm = fmaf(fm * F.inv_k * rs, jm, -jm1);
    const float a1 = A * djm * F.k_r * rs * cm;
    const float a2 = A * jm * fm * sm * rs * rs;
    g = f3(0.0f, fmaf(a1, y, -a2 * z), fmaf(a1, z, a2 * y));
}
// The whole warp on one spline photon. The sixteen tap rows of an evaluation are independent up to
// their sums, which run in a fixed order. When a warp has one photon left, its 32 lanes march it
// together (march.cuh spline_warp_march): every lane carries the whole march state and takes one
// row's dot product (lanes 0-15 with the value weights, 16-31 with the derivative weights), the
// products go through shared memory, and each of four lanes (all lanes, four by four) adds the
// sixteen rows of one sum in spline_row's order. One lane alone issues about 470 instructions a step,
// more than the instruction cache holds close, and took 535 ns.
struct SplineWarp {
    float s[2][16];            // row sums with the value (0) and derivative (1) weights
    float w[3][16];            // their factors: wy wz, dy wz, wy dz
};
struct SplineWarpCell {
    SplineWarp *buf;           // two, used in turn, so that one __syncwarp a step orders writes and reads
    int turn, lane;
    int x, y, z;
    float4 r;                  // this lane's row
};

// weight and derivative weight of tap `a` alone: the expressions of bspline_weights_f with g for f where
// that tap's are written in g (0.5 g g g is 0.5 (g g g): halving is exact)
__device__ __forceinline__ void bspline_tap(float f, int a, float &w, float &dw) {
    const bool low = (a & 1) == (a >> 1);             // taps 0 and 3: the outer ones
    const bool neg = a == 0 || a == 2;                // in g = 1 - f
    const float u = neg ? 1.0f - f : f;
    const float u2 = u * u, u3 = u2 * u;
    w = low ? u3 * (1.0f / 6.0f) : (2.0f / 3.0f) - u2 + 0.5f * u3;
    const float d = low ? 0.5f * u2 : (1.5f * u - 2.0f) * u;
    dw = neg ? -d : d;
}

// The evaluation above; every lane of the warp calls it with the same p.
__device__ __forceinline__ void spline_field_cell(const FieldParams &F, SplineWarpCell &C, float3 p, float &n, float3 &g) {
    float fx, fy, fz;
    const int x = spline_cell_of((p.x - F.xmin[0]) * F.xres[0], fx), y = spline_cell_of((p.y - F.xmin[1]) * F.xres[1], fy),
              z = spline_cell_of((p.z - F.xmin[2]) * F.xres[2], fz);
    if (spline_on_quads(F, x, y, z)) {
        const int row = C.lane & 15, b = row & 3, c = row >> 2, half = C.lane >> 4, q = C.lane & 3;
        if ((x != C.x) | (y != C.y) | (z != C.z)) {
            C.r = __ldg(F.coeff4 + ((spline_wrap(z - 1 + c, F.N[2]) * F.N[1] + spline_wrap(y - 1 + b, F.N[1])) * F.qrow + x));
            C.x = x; C.y = y; C.z = z;
        }
        SplineWarp &B = C.buf[C.turn];
        C.turn ^= 1;
        float wy, dy, wz, dz, wx[4], dx[4];
        bspline_tap(fy, b, wy, dy);
        bspline_tap(fz, c, wz, dz);
        bspline_weights_f(fx, wx, dx);
        B.w[half ? 2 : 0][row] = wy * (half ? dz : wz);
        B.w[1][row] = dy * wz;
        if (half) { wx[0] = dx[0]; wx[1] = dx[1]; wx[2] = dx[2]; wx[3] = dx[3]; }
        B.s[half][row] = C.r.x * wx[0] + C.r.y * wx[1] + C.r.z * wx[2] + C.r.w * wx[3];
        __syncwarp();
        const float4 *sp = reinterpret_cast<const float4 *>(B.s[q == 1 ? 1 : 0]);
        const float4 *wp = reinterpret_cast<const float4 *>(B.w[q < 2 ? 0 : q - 1]);
        float sum = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float4 u = sp[e], v = wp[e];
            sum = fmaf(u.x, v.x, sum);
            sum = fmaf(u.y, v.y, sum);
            sum = fmaf(u.z, v.z, sum);
            sum = fmaf(u.w, v.w, sum);
        }
        SplineSum T;
        T.v = __shfl_sync(0xffffffffu, sum, 0);
        T.gx = __shfl_sync(0xffffffffu, sum, 1);
        T.gy = __shfl_sync(0xffffffffu, sum, 2);
        T.gz = __shfl_sync(0xffffffffu, sum, 3);
        spline_result(F, T, n, g);
    } else {
        const float4 e = spline_taps(F, p);
        n = e.w;
        g = f3(e.x, e.y, e.z);
    }
}

// Field<FK>: the field of one kind. tab is the Bessel table (shared memory in the march kernel) or
// the staged spline brick, unused by the other kinds.
//   eval(F, tab, p, s, n, g)          n and grad n at p
//   eval_c(F, tab, C, p, s, n, g)     the same, with what the march carries from step to step in C
//   eval_in(F, tab, C, p, s, n, g)    the same for a p known to lie in the field (not in a gap)
// All three give the same bits at the same point.
struct NoCache {
    __device__ __forceinline__ void clear() {}
};
template <int FK> struct Field;
#define SMP_FIELD(FK, IN, ALL)                                                                                      \
    template <> struct Field<FK> {                                                                                  \
        using Cache = NoCache;                                                                                      \
        template <class TAB> static __device__ __forceinline__ void eval(const FieldParams &F, const TAB &tab, float3 p, float s, float &n, float3 &g) { ALL; } \
        template <class TAB> static __device__ __forceinline__ void eval_c(const FieldParams &F, const TAB &tab, Cache &, float3 p, float s, float &n, float3 &g) { ALL; } \
        template <class TAB> static __device__ __forceinline__ void eval_in(const FieldParams &F, const TAB &tab, Cache &, float3 p, float s, float &n, float3 &g) { IN; } \
    };
SMP_FIELD(FK_BESSEL0, bessel_field_ng<0>(F, tab, p, s, n, g), bessel_field<0>(F, tab, p, s, n, g))
SMP_FIELD(FK_BESSEL1, bessel_field_ng<1>(F, tab, p, s, n, g), bessel_field<1>(F, tab, p, s, n, g))
SMP_FIELD(FK_BESSEL2, bessel_field_ng<2>(F, tab, p, s, n, g), bessel_field<2>(F, tab, p, s, n, g))
SMP_FIELD(FK_BESSELN, bessel_field_n_ng(F, tab, p, s, n, g), bessel_field_n_ng(F, tab, p, in_gap(F, p) ? 0.0f : s, n, g))
// batched sweep: the instance's Bessel field
SMP_FIELD(FK_BATCH, bessel_field_rt_ng(F, tab, p, s, n, g), bessel_field_rt_ng(F, tab, p, in_gap(F, p) ? 0.0f : s, n, g))
SMP_FIELD(FK_PLANEWAVE, wave_field_ng(F, p, s, n, g), wave_field(F, p, s, n, g))
SMP_FIELD(FK_SOURCES, sources_field(F, p, n, g), sources_field(F, p, n, g))
#undef SMP_FIELD
// The field at a start point, for the discrete logic between marches: the spline's sixteen rows are
// kept out of its registers by a call.
template <int FK>
__device__ __forceinline__ void field_at(const FieldParams &F, const float4 *tab, float3 p, float s, float &n, float3 &g) {
    Field<FK>::eval(F, tab, p, s, n, g);
}
template <> struct Field<FK_SPLINE> {
    using Cache = SplineCell;
    // inlined only where a step of the brick kernel needs it; the discrete logic calls it
    static __device__ __forceinline__ void eval(const FieldParams &F, const float4 *brick, float3 p, float, float &n, float3 &g) {
        spline_field(F, brick, p, n, g);
    }
    static __device__ __noinline__ float4 eval_call(const FieldParams &F, float3 p) {
        float n;
        float3 g;
        spline_field(F, nullptr, p, n, g);
        return make_float4(g.x, g.y, g.z, n);
    }
    // CA: a SplineCell, or the whole warp's cell (SplineWarpCell)
    template <class CA>
    static __device__ __forceinline__ void eval_c(const FieldParams &F, const float4 *, CA &C, float3 p, float, float &n, float3 &g) {
        if (spline_in_gap(F, p)) {
            n = F.n_o;
            g = f3(0.0f, 0.0f, 0.0f);
            return;
        }
        spline_field_cell(F, C, p, n, g);
    }
    template <class CA>
    static __device__ __forceinline__ void eval_in(const FieldParams &F, const float4 *, CA &C, float3 p, float, float &n, float3 &g) {
        spline_field_cell(F, C, p, n, g);
    }
};

template <>
__device__ __forceinline__ void field_at<FK_SPLINE>(const FieldParams &F, const float4 *, float3 p, float, float &n, float3 &g) {
    const float4 r = Field<FK_SPLINE>::eval_call(F, p);
    n = r.w;
    g = f3(r.x, r.y, r.z);
}

}  // namespace smp
