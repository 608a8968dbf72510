// march.cuh -- the persistent photon-march kernel for sm_100a.
//
// One lane owns one photon at a time and runs the reference's per-photon algorithm
// (renderer/src/photon.cpp:302-335: genRay, scaling draw, directTracing, scatter with a sensor
// connection at every vertex) as a state machine. The expensive part -- traceTillBlock, the
// kick-drift-kick ER march with 10x refinement at faces and at the sampled distance
// (scene.cpp:385-425, :323-330) -- is one "step" that every marching lane of the warp executes
// together. When a lane's march ends it runs the discrete logic that follows (face normal,
// Fresnel BSDF, splat, Henyey-Greenstein scattering, roulette) until its next march starts; when
// its photon ends it takes a new photon index from a global counter (one atomic per warp), so
// warps stay full until the work runs out. Grid = resident CTAs over all SMs.
//
// Discrete decisions follow the reference CPU build exactly; the tests compare every photon's
// splats and end state with the CPU restatement on injected uniform streams.
#pragma once
#include <cooperative_groups.h>

#include <climits>
#include <type_traits>

#include "dev_field.cuh"
#include "kparams.h"

namespace smp {

namespace cg = cooperative_groups;

static constexpr unsigned kFull = 0xffffffffu;

// Resident 128-thread blocks per SM the march kernel is compiled for (register budget 65536 /
// (128 * blocks)).
#ifndef SMP_MIN_BLOCKS
#define SMP_MIN_BLOCKS 4
#endif
// The spline's lane loops hold the 64 taps of a cell in registers: two blocks.
constexpr int lane_blocks(int fk) { return fk == FK_SPLINE ? 2 : SMP_MIN_BLOCKS; }

enum LaneState : int { ST_FETCH = 0, ST_EVENT = 1, ST_MARCH = 2, ST_DONE = 3, ST_HOOK = 4 };
enum Event : int {
    EV_NEW = 0,          // photon fetched: genRay, scaling, direct or scatter
    EV_MARCH_END = 1,    // a traceTillBlock call finished
    EV_SCATTER = 2,      // Renderer::scatter entry (photon.cpp:97)
    EV_VERTEX = 3,       // head of the scatter loop (photon.cpp:113)
    EV_SCATTER_ONCE = 4, // Renderer::scatterOnce (photon.cpp:20)
    EV_FINISH = 5
};
enum Ctx : int { CTX_DIRECT = 0, CTX_CONNECT = 1, CTX_MOVE_FIRST = 2, CTX_MOVE_VERTEX = 3 };

struct Lane {
    // photon
    long long idx;
    float3 pos, dir;          // scatter()'s pos/dir (photon.cpp:98)
    float s;                  // temporal scaling (Bessel) / phase tau (plane waves)
    double total;             // running optical path length
    float totalDist;          // first sampled distance (photon.cpp:112)
    int depth, nspl, draws, steps, end;
    // uniforms
    unsigned r0, r1, r2, r3, rblk;
    int rhave;
    long long spos, send;
    // current march (traceTillBlock) and its caller (movePhoton / movePhotonTillSensor)
    float3 mp, md, mg;        // position, optical direction v, grad n at mp
    float mn;                 // n at mp
    double mtot;              // optical length accumulated by this march (FP64 form)
    float mtotf;              // the same in the FP32 form
    float dist_acc, dlimit, cur, hh;   // hh = cur / 2
    double cur_d;             // cur in double for the FP64 accumulator
    int stop;                 // step count at which traceTillBlock's loop count runs out (<= step cap)
    int prec, ctx, first;
    float large, d2s, rem, sampled;
    const float4 *tab;        // Bessel table in this block's shared memory
    const Inst *inst;         // batched sweep: the photon's instance
};

// Per-photon medium, weight, film and seed: the instance's in a batched sweep (n_inst is uniform
// over the grid, so these are uniform branches), else the plan's.
__device__ __forceinline__ float med_g(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->g : P.g; }
__device__ __forceinline__ float med_albedo(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->albedo : P.albedo; }
__device__ __forceinline__ float med_sigma_t(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->sigma_t : P.sigma_t; }
__device__ __forceinline__ float med_mfp(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->mfp : P.mfp; }
__device__ __forceinline__ float med_weight(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->weight : P.weight; }
__device__ __forceinline__ float med_large(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->large_dist : P.large_dist; }
__device__ __forceinline__ void *med_film(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->film : P.film; }
__device__ __forceinline__ unsigned long long med_seed(const Lane &L, const KParams &P) { return P.n_inst ? L.inst->seed : P.seed; }
// the field the photon marches through
template <int FK, class S>
__device__ __forceinline__ const FieldParams &field_of(const S &L, const KParams &P) {
    return FK == FK_BATCH ? L.inst->field : P.field;
}

// ---- uniforms -----------------------------------------------------------------------------
__device__ __forceinline__ void philox_block(unsigned &c0, unsigned &c1, unsigned &c2, unsigned &c3,
                                             unsigned k0, unsigned k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        unsigned hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        unsigned hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        c0 = hi1 ^ c1 ^ k0;
        c1 = lo1;
        c2 = hi0 ^ c3 ^ k1;
        c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

// one Philox block, kept out of line: draw() is called from many places in the event code
static __device__ __noinline__ uint4 philox_refill(unsigned blk, unsigned ph_lo, unsigned ph_hi, unsigned k0, unsigned k1) {
    unsigned c0 = blk, c1 = 0u, c2 = ph_lo, c3 = ph_hi;
    philox_block(c0, c1, c2, c3, k0, k1);
    return make_uint4(c0, c1, c2, c3);
}

__device__ __forceinline__ float draw(Lane &L, const KParams &P) {
    ++L.draws;
    if (P.rng == SMP_RNG_STREAM) {
        if (L.spos < L.send) return __ldg(P.stream + (L.spos++));
        L.end = SMP_END_STREAM;
        return 0.5f;
    }
    if (L.rhave == 0) {
        const unsigned long long seed = med_seed(L, P);
        uint4 b = philox_refill(L.rblk++, unsigned(L.idx), unsigned(L.idx >> 32), unsigned(seed), unsigned(seed >> 32));
        L.r0 = b.x; L.r1 = b.y; L.r2 = b.z; L.r3 = b.w;
        L.rhave = 4;
    }
    unsigned x = L.r0;
    L.r0 = L.r1; L.r1 = L.r2; L.r2 = L.r3;
    --L.rhave;
    return float(x >> 8) * (1.0f / 16777216.0f);
}

// ---- small pieces of the scene -------------------------------------------------------------
__device__ __forceinline__ int steps_for(float dlimit, float h0) {
    // (long)(dist/h + 1) as the reference's x86-64 build converts it (scene.cpp:391): out-of-range
    // values become INT64_MIN (no steps). Counts above 2^31 - 1 are clamped: the per-photon step
    // cap (<= 2e9) ends the photon first.
    float v = dlimit / h0 + 1.0f;
    if (!(v >= -9.2233720e18f && v < 9.2233720e18f)) return 0;
    if (v >= 2147483647.0f) return 2147483647;
    return int(v);
}


// nearest face of the medium box (scene.cpp:655-676 / :736-757)
__device__ __forceinline__ float3 face_normal(const KParams &P, float3 p) {
    float best = 3.40282347e+38f, dirv = 0.0f;
    int chosen = 3;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float pi = comp(p, i);
        float d = fabsf(P.L[i] - pi);
        if (d < best) { best = d; chosen = i; dirv = -1.0f; }
        d = fabsf(P.R[i] - pi);
        if (d < best) { best = d; chosen = i; dirv = 1.0f; }
    }
    return f3(chosen == 0 ? dirv : 0.0f, chosen == 1 ? dirv : 0.0f, chosen == 2 ? dirv : 0.0f);
}

// util.h:42-57
__device__ __forceinline__ float fresnel(float cosI, float cosT, float eta) {
    if (fabsf(eta - 1.0f) < kEps * fmaxf(1.0f, fabsf(eta))) return 0.0f;
    float Rs = (cosI - eta * cosT) / (cosI + eta * cosT);
    float Rp = (cosT - eta * cosI) / (cosT + eta * cosI);
    return 0.5f * (Rs * Rs + Rp * Rp);
}

// SmoothDielectric::sample (bsdf.cpp:26-58, util.h:64-88)
__device__ __forceinline__ float3 bsdf_sample(Lane &L, const KParams &P, float3 in, float3 n) {
    if (fabsf(P.ior1 - P.ior2) < kEps) return in;
    float eta = (dot3(in, n) < -kEps) ? P.ior2 / P.ior1 : P.ior1 / P.ior2;
    float an = dot3(in, n);
    float3 q = mul(n, an);
    float3 pp = divs(sub(in, q), eta);
    float3 refl = add(mul(n, -2.0f * an), in);
    if (len3(pp) > 1.0f) return refl;                       // total internal reflection
    q = normalized(q);
    float t = 1.0f - dot3(pp, pp);
    float3 outT = add(pp, mul(q, t > 0.0f ? sqrtf(t) : 0.0f));
    float cosI = fabsf(dot3(n, in)), cosT = fabsf(dot3(n, outT));
    float F = fresnel(cosI, cosT, eta);
    return (draw(L, P) < F) ? refl : outT;
}

// thin lens deflection (lens.cpp:70-97); returns the path-length change in add_len
__device__ __forceinline__ bool lens_deflect(float sqap, float focal, float3 pos, float3 &dir, float &add_len) {
    float sq = pos.y * pos.y + pos.z * pos.z;
    if (sq > sqap) return false;
    float invd = -1.0f / dir.x;
    dir = f3(-focal, dir.y * invd * focal - pos.y, dir.z * invd * focal - pos.z);
    add_len = focal * invd - len3(dir);
    dir = normalized(dir);
    return true;
}

__device__ __forceinline__ void acc_total(double &t, float v, bool fp64) {
    t = fp64 ? t + double(v) : double(float(t) + v);
}

// Camera::propagate_till_sensor (camera.cpp:54-75): the distance goes into the caller's local
// distanceToSensor, which the caller then adds to its path length.
__device__ __forceinline__ bool propagate_till_sensor(const KParams &P, float3 &pos, float3 &dir, float &dts) {
    if (P.cam_lens_active) {
        float a = 0.0f;
        if (!lens_deflect(P.cam_lens_sqap, P.cam_lens_focal, pos, dir, a)) return false;
        dts += a;
    }
    float dist = (P.cam_origin[0] - pos.x) / dir.x;
    pos = add(pos, mul(dir, dist));
    dts += dist;
    return true;
}

// Film cell of a splat at sensor point p with path length pl (scene.cpp:782-829) on a film X
// pixels wide: the bilinear base pixel (ix, iy), its fractions (fx, fy) and the bin iz; false when
// pl is outside the binned range.
__device__ __forceinline__ bool splat_bin(const KParams &P, int X, float3 p, double pl, int depth,
                                          int &ix, int &iy, int &iz, float &fx, float &fy) {
    float x = dot3(ld3(P.cam_h), p) - P.cam_origin[1];
    float y = dot3(ld3(P.cam_v), p) - P.cam_origin[2];
    bool nobin = (P.pl_min == -1.0f) && (P.pl_max == -1.0f);
    bool inrange = P.fp64 ? (pl > double(P.pl_min) && pl < double(P.pl_max))
                          : (float(pl) > P.pl_min && float(pl) < P.pl_max);
    if (!(nobin || inrange)) return false;
    x = (x / P.cam_plane[0] + 0.5f) * float(X);
    y = (y / P.cam_plane[1] + 0.5f) * float(P.Y);
    float flx = floorf(x), fly = floorf(y);
    ix = int(flx); iy = int(fly);
    if (P.bounce) iz = depth;
    else if (nobin) iz = 0;
    else if (P.fp64) iz = int(floor((pl - double(P.pl_min)) / (double(P.pl_max) - double(P.pl_min)) * double(P.Z)));
    else iz = int(floorf(((float(pl) - P.pl_min) / (P.pl_max - P.pl_min)) * float(P.Z)));
    fx = x - flx; fy = y - fly;
    return true;
}

// Scene::addEnergyToImage (scene.cpp:782-829) with bilinear sharing (USE_PIXEL_SHARING): the four taps
// of base pixel (ix, iy) in bin iz, each with Image3::addEnergy's bounds check (image.h:320-324,
// scene.h:305-312). Warp-aggregated: the lanes that splat together and share a base pixel share all four
// taps, so one match groups them, the group's first lane sums the others' values (in double for the
// FP64 film) and issues the atomics. A narrow beam's direct light lands on a handful of pixels, where
// one atomic per lane would serialise on the same address. Most groups are a single lane, which then
// goes straight to its atomics; a match and a tree reduction per tap took twice the instructions.
template <class T>
__device__ __forceinline__ void add_tap(const KParams &P, T *film, int x, int y, int z, T v) {
    if (x >= 0 && x < P.X && y >= 0 && y < P.Y && z >= 0 && z < P.Z) atomicAdd(film + (size_t(z) * P.Y + y) * P.X + x, v);
}
template <class T>
__device__ __forceinline__ void add_taps_t(const KParams &P, T *film, int ix, int iy, int iz, float v0, float v1, float v2,
                                           float v3) {
    // a base pixel none of whose taps can lie on the film
    if (ix < -1 || ix >= P.X || iy < -1 || iy >= P.Y || iz < 0 || iz >= P.Z) return;
    const unsigned act = __activemask();
    const unsigned lane = threadIdx.x & 31u;
    unsigned same = __match_any_sync(act, ((unsigned long long)iz * unsigned(P.Y + 1) + unsigned(iy + 1)) * unsigned(P.X + 1) + unsigned(ix + 1));
    if (P.n_inst) same &= __match_any_sync(act, reinterpret_cast<unsigned long long>(film));     // a sweep's films
    T s0 = T(v0), s1 = T(v1), s2 = T(v2), s3 = T(v3);
    const bool first = (same & ((1u << lane) - 1u)) == 0u;
    unsigned rest = first ? same & (same - 1u) : 0u;      // the first lane collects the others
    while (__any_sync(act, rest != 0u)) {
        const int src = rest ? __ffs(rest) - 1 : int(lane);
        const float a = __shfl_sync(act, v0, src), b = __shfl_sync(act, v1, src), c = __shfl_sync(act, v2, src),
                    d = __shfl_sync(act, v3, src);
        if (rest) {
            s0 += T(a); s1 += T(b); s2 += T(c); s3 += T(d);
            rest &= rest - 1u;
        }
    }
    if (!first) return;
    add_tap(P, film, ix, iy, iz, s0);
    add_tap(P, film, ix + 1, iy, iz, s1);
    add_tap(P, film, ix, iy + 1, iz, s2);
    add_tap(P, film, ix + 1, iy + 1, iz, s3);
}
__device__ __forceinline__ void add_taps(const KParams &P, void *film, int ix, int iy, int iz, float v0, float v1, float v2,
                                         float v3) {
    if (P.fp64) add_taps_t(P, static_cast<double *>(film), ix, iy, iz, v0, v1, v2, v3);
    else add_taps_t(P, static_cast<float *>(film), ix, iy, iz, v0, v1, v2, v3);
}

__device__ __forceinline__ void splat(Lane &L, const KParams &P, float3 p, double pl, int depth, float val) {
    if (P.records) {
        smp_photon_record *rec = P.records + (L.idx - P.first_photon);
        if (L.nspl < SMP_TRACE_MAX_SPLATS) {
            smp_splat_record &sr = rec->splats[L.nspl];
            sr.p[0] = p.x; sr.p[1] = p.y; sr.p[2] = p.z;
            sr.depth = depth;
            sr.pathlength = pl;
            sr.value = double(val);
        }
    }
    ++L.nspl;
    int ix, iy, iz;
    float fx, fy;
    if (!splat_bin(P, P.X, p, pl, depth, ix, iy, iz, fx, fy)) return;
    add_taps(P, med_film(L, P), ix, iy, iz, val * (1.0f - fx) * (1.0f - fy), val * fx * (1.0f - fy),
             val * (1.0f - fx) * fy, val * fx * fy);
}

// Henyey-Greenstein (phase.cpp:17-21, :40-76; util.h:17-27)
__device__ __forceinline__ float hg_f(float g, float3 in, float3 out) {
    float c = dot3(in, out);
    float b = 1.0f + g * g - 2.0f * g * c;
    return (1.0f / (4.0f * 3.14159265358979f)) * (1.0f - g * g) / (b * sqrtf(b));
}
__device__ __forceinline__ float3 hg_sample(Lane &L, const KParams &P, float3 in) {
    float sx = draw(L, P);
    float sy = draw(L, P);
    float g = med_g(L, P), cosT;
    if (fabsf(g) < kEps) cosT = 1.0f - 2.0f * sx;
    else {
        float sq = (1.0f - g * g) / (1.0f - g + 2.0f * g * sx);
        cosT = (1.0f + g * g - sq * sq) / (2.0f * g);
    }
    float sinT = sqrtf(fmaxf(0.0f, 1.0f - cosT * cosT));
    float phi = 6.28318548202514648f * sy;
    float sP, cP;
    sincos_near(phi, sP, cP);
    float3 ax, ay;
    if (fabsf(in.x) > fabsf(in.y)) {
        float inv = 1.0f / sqrtf(in.x * in.x + in.z * in.z);
        ay = f3(in.z * inv, 0.0f, -in.x * inv);
    } else {
        float inv = 1.0f / sqrtf(in.y * in.y + in.z * in.z);
        ay = f3(0.0f, in.z * inv, -in.y * inv);
    }
    ax = cross3(ay, in);
    return add(add(mul(ax, sinT * cP), mul(ay, sinT * sP)), mul(in, cosT));
}

// sampleRandomDirection (scene.cpp:26-39, warp.cpp:22-34): first draw -> azimuth, second -> z,
// the order the reference's GCC build evaluates Vec2f(sampler(), sampler()).
__device__ __forceinline__ float3 random_direction(Lane &L, const KParams &P) {
    float uy = draw(L, P);
    float ux = draw(L, P);
    float tmp = sqrtf(1.0f - ux * ux);
    float sP, cP;
    sincos_near(6.28318548202514648f * uy, sP, cP);
    return f3(-ux, cP * tmp, sP * tmp);
}

__device__ __forceinline__ bool roulette(Lane &L, const KParams &P) {
    const float albedo = med_albedo(L, P);
    return (albedo > 0.0f) && ((albedo >= 1.0f) || (draw(L, P) < albedo));
}

// area_textured_source::sample_ray (scene.cpp:107-137) + DiscreteDistribution::sample (pmf.h:109-121)
__device__ __forceinline__ bool gen_ray(Lane &L, const KParams &P, float3 &pos, float3 &dir, double &total) {
    float u = draw(L, P);
    int lo = 0, hi = P.n_tex + 1;                 // lower_bound over n_tex + 1 cdf entries
    if (P.cdf_guide) {
        // u's bucket of the guide table narrows the search to a few entries; the CDF is monotone
        // (the host builds no guide otherwise), so the lower bound found is the same
        const int G = 1 << P.guide_bits;
        const int b = min(int(u * float(G)), G);
        lo = __ldg(P.cdf_guide + b);
        hi = __ldg(P.cdf_guide + b + 1);
    }
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (__ldg(P.cdf + mid) < u) lo = mid + 1; else hi = mid;
    }
    int idx = min(P.n_tex - 1, max(0, lo - 1));
    while (idx < P.n_tex && __ldg(P.cdf + idx + 1) - __ldg(P.cdf + idx) == 0.0f) ++idx;
    if (idx > P.n_tex - 1) idx = P.n_tex - 1;
    int py = idx / P.tex_x;
    int px = idx - py * P.tex_x;
    pos = ld3(P.src_origin);
    float uy = draw(L, P);
    pos.y += -P.plane[0] / 2.0f + float(px) * P.pixsize[0] + uy * P.pixsize[0];
    float uz = draw(L, P);
    pos.z += -P.plane[1] / 2.0f + float(py) * P.pixsize[1] + uz * P.pixsize[1];
    float z = draw(L, P) * (1.0f - P.ct) + P.ct;
    float zt = sqrtf(1.0f - z * z);
    float phi = draw(L, P) * 2.0f * 3.14159265358979f;
    float sP, cP;
    sincos_near(phi, sP, cP);
    dir = f3(-z, zt * cP, zt * sP);
    // Lens::propagate_till_lens (lens.cpp:20-33)
    float dist = -(pos.x - P.src_lens_origin[0]) / dir.x;
    pos = add(pos, mul(dir, dist));
    acc_total(total, dist, P.fp64);
    if (P.src_lens_active) {
        float a = 0.0f;
        if (!lens_deflect(P.src_lens_sqap, P.src_lens_focal, pos, dir, a)) return false;
        acc_total(total, a, P.fp64);
    }
    return true;
}

// ---- the traceTillBlock step ----------------------------------------------------------------
// the photon's ER step and refinement steps: its instance's in a batched sweep, else the plan's
template <int FK, class S>
__device__ __forceinline__ float step_h0(const S &L, const KParams &P) { return FK == FK_BATCH ? L.inst->h0 : P.h0; }
template <int FK, class S>
__device__ __forceinline__ const float *step_tab(const S &L, const KParams &P) {
    return FK == FK_BATCH ? L.inst->cur_tab : P.cur_tab;
}

template <int FK>
__device__ __forceinline__ void begin_march(Lane &L, const KParams &P, float dlimit, bool eval) {
    if (eval) field_at<FK>(field_of<FK>(L, P), L.tab, L.mp, L.s, L.mn, L.mg);
    const float h0 = step_h0<FK>(L, P);
    L.dist_acc = 0.0f;
    L.dlimit = dlimit;
    L.cur = h0;
    L.hh = 0.5f * h0;
    L.cur_d = double(h0);
    L.prec = P.precision;
    L.stop = int(min((long long)L.steps + (long long)steps_for(dlimit, h0), (long long)P.step_cap));
    L.mtotf = float(L.mtot);
}
// a march with no steps ends at once (traceTillBlock's maxsteps <= 0)
__device__ __forceinline__ bool march_has_steps(const Lane &L) { return L.stop > L.steps; }

// One iteration of the traceTillBlock loop (scene.cpp:395-419): kick, drift, one fused field
// evaluation, kick, then the loop's tests. Returns true when the march has ended (loop count or
// refinement exhausted, or the photon aborted). S is a Lane or any state with the same march
// members.
//
// The tests are arranged for the common case, an accepted step with steps to go: the box test
// (thresholds box_lo/box_hi, exact) and the distance test (dist_acc + cur <= dlimit) are one chain
// of predicate comparisons, and the loop count and the step cap share one counter (`stop` is the
// loop's end clamped to the cap; the cap is told apart on the rare path).
//
// C carries what the field keeps from step to step (Field<FK>::Cache), or is a NoCache: the field is
// then evaluated through L.tab alone (the staged spline brick).
template <int FK, int FP = -1, class S, class CA>
__device__ __forceinline__ bool march_step(S &L, const KParams &P, CA &C) {
    const bool f64 = FP < 0 ? P.fp64 != 0 : FP != 0;     // FP: the path-length form, if fixed at compile time
    const float3 d = f3(fmaf(L.hh, L.mg.x, L.md.x), fmaf(L.hh, L.mg.y, L.md.y), fmaf(L.hh, L.mg.z, L.md.z));
    const float hinv = L.cur * rcp_fast(L.mn);
    const float3 p = f3(fmaf(d.x, hinv, L.mp.x), fmaf(d.y, hinv, L.mp.y), fmaf(d.z, hinv, L.mp.z));
    float n2;
    float3 g2;
    if constexpr (std::is_same<CA, NoCache>::value) Field<FK>::eval(field_of<FK>(L, P), L.tab, p, L.s, n2, g2);
    else Field<FK>::eval_c(field_of<FK>(L, P), L.tab, C, p, L.s, n2, g2);
    const float3 d2 = f3(fmaf(L.hh, g2.x, d.x), fmaf(L.hh, g2.y, d.y), fmaf(L.hh, g2.z, d.z));
    ++L.steps;
    const float sacc = L.dist_acc + L.cur;
    // p - L > -eps and R - p > -eps per axis (as thresholds) and dist + h <= dlimit, as one chain of
    // predicate comparisons; a NaN coordinate fails it, as it fails the reference's test
    const bool ok = (p.x >= P.box_lo[0]) & (p.x <= P.box_hi[0]) & (p.y >= P.box_lo[1]) & (p.y <= P.box_hi[1]) &
                    (p.z >= P.box_lo[2]) & (p.z <= P.box_hi[2]) & (sacc <= L.dlimit);
    if (ok && L.steps < L.stop) {
        L.mp = p; L.md = d2; L.mn = n2; L.mg = g2;
        L.dist_acc = sacc;
        if (f64) L.mtot = fma(L.cur_d, double(n2), L.mtot);
        else L.mtotf = fmaf(L.cur, n2, L.mtotf);
        return false;
    }
    // A non-finite position fails the box test, so refinement ends the march within
    // `precision` steps; run_events checks finiteness when the march ends.
    if (L.steps >= P.step_cap) { L.end = SMP_END_STEP_CAP; return true; }
    if (ok) {                                     // accepted, and the loop count is exhausted
        L.mp = p; L.md = d2; L.mn = n2; L.mg = g2;
        L.dist_acc = sacc;
        if (f64) L.mtot = fma(L.cur_d, double(n2), L.mtot);
        else L.mtotf = fmaf(L.cur, n2, L.mtotf);
        return true;
    }
    if (--L.prec < 0) {                           // refinement exhausted: keep the failed step
        L.mp = p; L.md = d2; L.mn = n2; L.mg = g2;
        return true;
    }
    L.cur = step_tab<FK>(L, P)[P.precision - L.prec];   // restore (mp, md unchanged) and refine: cur / 10
    L.hh = 0.5f * L.cur;
    L.cur_d = double(L.cur);
    L.stop = min(L.steps + 10, P.step_cap);       // maxsteps = 11 from i = 0: ten more steps
    return false;
}

// ---- untested windows -------------------------------------------------------------------------
// A step's tests (seven comparisons in a chain, the loop count, the branch they feed) come after its
// position, and the next step waits for their branch: one photon alone in its warp took 440 cycles a
// step, three times the arithmetic's own chain. Far from a face and from the sampled distance none
// of them can fail, so a lane that marches alone, or with few others, runs windows: the number of
// steps that provably pass every test is worked out once, and those steps run without them. The
// steps' arithmetic is march_step's own, so the photon is the same bit for bit.
//
// safe_steps: a lower bound on the steps, at most `cap`, that pass every test of march_step from
// here (<= 0: none known). A step moves a coordinate by at most h |d_a| / n, where n >= n_low and the
// momentum component d_a changes by at most h grad_bound a step; 3 % and 3e-7 a step cover the
// rounding of the momentum, the reciprocal and this bound itself, win_round the position's. The path
// distance gains h a step, and the rounding of its sum. The x range is the field's, inside the gaps.
template <int FK, class S>
__device__ __forceinline__ int safe_steps(const S &L, const KParams &P, int cap) {
    const FieldParams &F = field_of<FK>(L, P);
    const float h = L.cur;
    if (!(F.n_low > 0.0f) || !(h >= P.win_hmin)) return 0;
    const float kick = fmaf(F.grad_bound, h, 3e-7f) * float(cap + 1);
    const float q = __fdividef(1.03f * h, F.n_low);
    const float mx = fminf(L.mp.x - fmaxf(P.box_lo[0], F.sgap), fminf(P.box_hi[0], F.egap) - L.mp.x);
    const float my = fminf(L.mp.y - P.box_lo[1], P.box_hi[1] - L.mp.y);
    const float mz = fminf(L.mp.z - P.box_lo[2], P.box_hi[2] - L.mp.z);
    const float kx = __fdividef(mx, fmaf(q, fabsf(L.md.x) + kick, P.win_round));
    const float ky = __fdividef(my, fmaf(q, fabsf(L.md.y) + kick, P.win_round));
    const float kz = __fdividef(mz, fmaf(q, fabsf(L.md.z) + kick, P.win_round));
    const float left = L.dlimit - L.dist_acc, kd = __fdividef(left, fmaf(1.03f, h, 1.2e-7f * L.dlimit));
    const float k = 0.999f * fminf(fminf(kx, ky), fminf(kz, kd));
    // Room for a step, and a state that is finite: a minimum drops an operand that is not a number, a sum
    // keeps it (kd alone may be inf / inf, for a distance limit of inf). A step from any other state moves
    // nowhere, and march_step's tests end its march.
    if (!((k >= 1.0f) & ((kx + ky) + kz >= 1.0f) & (left > 0.0f) & (L.mn >= F.n_low))) return 0;
    return min(int(fminf(k, float(cap))), L.stop - L.steps - 1);
}

// The field along a window. begin(p, v, h/n) starts (or restarts) it at a point, eval(p) gives n and
// grad n at the next point and false where it could not (the caller then takes the field from
// Field<FK>::eval_in). The same bits either way.
template <int FK, class CA> struct WindowField {
    CA &C;
    const FieldParams &F;
    const float4 *tab;
    float s;
    __device__ __forceinline__ void begin(float3, float3, float) {}
    __device__ __forceinline__ bool eval(float3 p, float &n, float3 &g) {
        Field<FK>::eval_in(F, tab, C, p, s, n, g);
        return true;
    }
};
// Bessel modes 0-2 (RT: by the batched sweep's order-general formulas). The table entry a step needs
// is known one step ahead all but always: the table coordinate t moves by nearly the same amount
// each step. So the entry of the interval t + dt falls in is loaded while the step before it is still
// under way, which takes the index, the address and the load off the chain of dependent
// instructions; a point in another interval (or off the table, or on the axis) fails f's test.
template <int M, bool RT> struct WindowBessel {
    const FieldParams &F;
    const float4 *tab;
    float s;
    float t, fi;
    float4 a, b;
    __device__ __forceinline__ void load(float tp) {
        const float big = 8388608.0f;
        const float tb = fminf(__fadd_rd(fmaxf(tp, 0.0f), big), big + (F.bend - 1.0f));
        const unsigned i = unsigned(__float_as_int(tb) - 0x4B000000);
        fi = tb - big;
        a = tab[2 * i];
        b = tab[2 * i + 1];
    }
    __device__ __forceinline__ void begin(float3 p, float3 v, float hinv) {
        const float r2 = fmaf(p.y, p.y, p.z * p.z), rs = rsqrt_fast(r2);
        t = F.kb * (r2 * rs);
        load(fmaf(F.kb * rs * hinv, fmaf(p.y, v.y, p.z * v.z), t));
    }
    __device__ __forceinline__ bool eval(float3 p, float &n, float3 &g) {
        const float y = p.y, z = p.z;
        const float r2 = fmaf(y, y, z * z);
        const float rs = rsqrt_fast(r2);
        const float r = r2 * rs, tn = F.kb * r;
        const float f = tn - fi;
        const bool ok = (r >= kEps) & (f >= 0.0f) & (f < 1.0f);
        const float jm = fmaf(fmaf(fmaf(a.w, f, a.z), f, a.y), f, a.x);
        const float jm1 = fmaf(fmaf(fmaf(b.w, f, b.z), f, b.y), f, b.x);
        load(tn + (tn - t));
        t = tn;
        if (RT) bessel_rt_result(F, M, F.amp * s, y, z, rs, jm, jm1, n, g);
        else bessel_result<M>(F, F.amp * s, y, z, rs, jm, jm1, n, g);
        return ok;
    }
};

// `k` steps of march_step (a multiple of four) that safe_steps has shown to be accepted, in blocks of
// four without a branch (one for the spline, whose unrolled step does not fit the instruction cache
// four times: 633 against 535 ns a step); a block in which the field's prediction failed runs again
// from its start.
template <int FK, int FP, class S, class CA, class WF>
__device__ __forceinline__ void window_steps(S &L, const KParams &P, int k, CA &C, WF W) {
    const FieldParams &F = field_of<FK>(L, P);
    const float h = L.cur, hh = L.hh, s = L.s;
    const double hd = L.cur_d;
    float3 p = L.mp, v = L.md, g = L.mg;
    float n = L.mn, acc = L.dist_acc, totf = L.mtotf;
    double tot = L.mtot;
    W.begin(p, v, h * rcp_fast(n));
    constexpr int B = FK == FK_SPLINE ? 1 : 4;
#pragma unroll 1
    for (int i = 0; i < k; i += B) {
        const float3 p0 = p, v0 = v, g0 = g;
        const float n0 = n, acc0 = acc, totf0 = totf;
        const double tot0 = tot;
        bool ok = true;
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const float3 d = f3(fmaf(hh, g.x, v.x), fmaf(hh, g.y, v.y), fmaf(hh, g.z, v.z));
            const float hinv = h * rcp_fast(n);
            p = f3(fmaf(d.x, hinv, p.x), fmaf(d.y, hinv, p.y), fmaf(d.z, hinv, p.z));
            ok &= W.eval(p, n, g);
            v = f3(fmaf(hh, g.x, d.x), fmaf(hh, g.y, d.y), fmaf(hh, g.z, d.z));
            acc = acc + h;
            if (FP) tot = fma(hd, double(n), tot);
            else totf = fmaf(h, n, totf);
        }
        if (!ok) {
            p = p0; v = v0; g = g0; n = n0; acc = acc0; totf = totf0; tot = tot0;
#pragma unroll 1
            for (int j = 0; j < B; ++j) {
                const float3 d = f3(fmaf(hh, g.x, v.x), fmaf(hh, g.y, v.y), fmaf(hh, g.z, v.z));
                const float hinv = h * rcp_fast(n);
                p = f3(fmaf(d.x, hinv, p.x), fmaf(d.y, hinv, p.y), fmaf(d.z, hinv, p.z));
                Field<FK>::eval_in(F, L.tab, C, p, s, n, g);
                v = f3(fmaf(hh, g.x, d.x), fmaf(hh, g.y, d.y), fmaf(hh, g.z, d.z));
                acc = acc + h;
                if (FP) tot = fma(hd, double(n), tot);
                else totf = fmaf(h, n, totf);
            }
            W.begin(p, v, h * rcp_fast(n));
        }
    }
    L.mp = p; L.md = v; L.mg = g; L.mn = n;
    L.dist_acc = acc; L.mtotf = totf; L.mtot = tot;
    L.steps += k;
}

template <int FK, int FP, class S, class CA>
__device__ __forceinline__ void march_window_fp(S &L, const KParams &P, int k, CA &C) {
    const FieldParams &F = field_of<FK>(L, P);
    if constexpr (FK <= FK_BESSEL2) {
        window_steps<FK, FP>(L, P, k, C, WindowBessel<FK, false>{F, L.tab, L.s});
    } else if constexpr (FK == FK_BATCH) {
        if (F.mode == 0) window_steps<FK, FP>(L, P, k, C, WindowBessel<0, true>{F, L.tab, L.s});
        else if (F.mode == 1) window_steps<FK, FP>(L, P, k, C, WindowBessel<1, true>{F, L.tab, L.s});
        else window_steps<FK, FP>(L, P, k, C, WindowBessel<2, true>{F, L.tab, L.s});
    } else {
        window_steps<FK, FP>(L, P, k, C, WindowField<FK, CA>{C, F, L.tab, L.s});
    }
}
template <int FK, class S, class CA>
__device__ __forceinline__ void march_window(S &L, const KParams &P, int k, CA &C) {
    if (P.fp64) march_window_fp<FK, 1>(L, P, k, C);
    else march_window_fp<FK, 0>(L, P, k, C);
}

// ---- a lone spline photon on the whole warp ------------------------------------------------------
// Marches the photon of lane `src`, the warp's last, to the end of its march with the whole warp
// (SplineWarpCell): the lane's march state in every lane, the same windows and steps in all of them,
// the result back to the owner. Returns the accepted steps. All 32 lanes call it.
__device__ __forceinline__ int spline_warp_march(Lane &L, const KParams &P, int src, SplineWarp *buf, int lane) {
    struct {
        float3 mp, md, mg;
        float mn, cur, hh, dist_acc, dlimit, mtotf, s;
        double mtot, cur_d;
        int steps, stop, prec, end;
        const float4 *tab;
        const Inst *inst;
    } M;
    auto from = [&](float x) { return __shfl_sync(kFull, x, src); };
    auto fromi = [&](int x) { return __shfl_sync(kFull, x, src); };
    M.mp = f3(from(L.mp.x), from(L.mp.y), from(L.mp.z));
    M.md = f3(from(L.md.x), from(L.md.y), from(L.md.z));
    M.mg = f3(from(L.mg.x), from(L.mg.y), from(L.mg.z));
    M.mn = from(L.mn); M.cur = from(L.cur); M.hh = from(L.hh);
    M.dist_acc = from(L.dist_acc); M.dlimit = from(L.dlimit); M.mtotf = from(L.mtotf);
    M.mtot = __shfl_sync(kFull, L.mtot, src);
    M.cur_d = __shfl_sync(kFull, L.cur_d, src);
    M.steps = fromi(L.steps); M.stop = fromi(L.stop); M.prec = fromi(L.prec); M.end = fromi(L.end);
    M.s = 0.0f;
    M.tab = nullptr;
    M.inst = nullptr;
    SplineWarpCell C;
    C.buf = buf; C.turn = 0; C.lane = lane;
    C.x = C.y = C.z = INT_MIN;
    C.r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncwarp();
    int accepted = 0;
    for (bool end = false; !end;) {
        const int w = safe_steps<FK_SPLINE>(M, P, 1024);
        if (w >= 4) {
            march_window<FK_SPLINE>(M, P, w, C);
            accepted += w;
            continue;
        }
#pragma unroll 1
        for (int t = 0; t < 8 && !end; ++t) {
            const float3 q = M.mp;
            end = march_step<FK_SPLINE>(M, P, C);
            accepted += (q.x != M.mp.x || q.y != M.mp.y || q.z != M.mp.z) ? 1 : 0;
        }
    }
    __syncwarp();
    if (lane == src) {
        L.mp = M.mp; L.md = M.md; L.mg = M.mg; L.mn = M.mn;
        L.cur = M.cur; L.hh = M.hh; L.cur_d = M.cur_d;
        L.dist_acc = M.dist_acc; L.mtotf = M.mtotf; L.mtot = M.mtot;
        L.steps = M.steps; L.stop = M.stop; L.prec = M.prec; L.end = M.end;
    }
    return accepted;
}

// ---- discrete logic between marches ---------------------------------------------------------
// Observation points for path replay (adjoint.cuh). The render kernels use NoHook, for which every
// hook call below is compiled out.
struct NoHook {
    static constexpr bool on = false;
    __device__ bool at(Lane &, int) { return false; }
    __device__ void splatted(const Lane &, float3, double, int, float) {}
    __device__ void photon_begin(const Lane &) {}
    __device__ void photon_end(const Lane &) {}
    __device__ void march_begin() {}
    __device__ void accepted(int) {}
};

// Runs the lane's events until it starts a march (returns ST_MARCH) or its photon ends
// (returns ST_FETCH). With a hook, h->at(L, ev) is asked at the entry of EV_SCATTER and
// EV_SCATTER_ONCE and at EV_VERTEX once the depth test has passed; true stops here with ST_HOOK
// (the lane state is that of the event's entry). h->splatted sees every splat.
template <int FK, class H = NoHook>
__device__ __forceinline__ int run_events(Lane &L, const KParams &P, int ev, H *h = nullptr) {
    for (;;) {
        float dlimit = 0.0f;                                    // the march the event starts,
        bool go = false, at_start = false;                      // if it does, and whether its field is still unknown
        if (ev == EV_MARCH_END) {
            if (!P.fp64) L.mtot = double(L.mtotf);
            if (L.end == 0 && !isfinite((L.mp.x + L.mp.y) + (L.mp.z + L.md.x) + (L.md.y + L.md.z) + L.mn))
                L.end = SMP_END_NAN;
        }
        if (ev != EV_FINISH && L.end != 0) {                    // aborted (cap, NaN, stream)
            if (ev == EV_MARCH_END) {
                if (L.ctx == CTX_MOVE_FIRST || L.ctx == CTX_MOVE_VERTEX) { L.pos = L.mp; L.dir = L.md; L.total = L.mtot; }
                else if (L.ctx == CTX_DIRECT) L.total = L.mtot;
            }
            ev = EV_FINISH;
        }
        switch (ev) {
        case EV_NEW: {
            L.total = 0.0;
            L.depth = 0; L.nspl = 0; L.draws = 0; L.steps = 0; L.end = 0;
            L.rblk = 0; L.rhave = 0;
            if (P.rng == SMP_RNG_STREAM) {
                long long k = L.idx - P.first_photon;
                L.spos = P.offsets[k];
                L.send = P.offsets[k + 1];
            }
            if (FK == FK_BATCH) {
                // sweep photon index -> (instance, the instance's photon index)
                int lo = 0, hi = P.n_inst;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (P.inst_first[mid] <= L.idx) lo = mid; else hi = mid;
                }
                L.inst = P.insts + lo;
                L.idx -= P.inst_first[lo];
                L.tab = L.inst->field.btab;
            }
            if (!gen_ray(L, P, L.pos, L.dir, L.total)) { L.end = SMP_END_GENRAY_FAIL; ev = EV_FINISH; break; }
            float u = draw(L, P);
            const FieldParams &F = field_of<FK>(L, P);
            if (FK == FK_PLANEWAVE) L.s = fmaf(F.phi_range, u, F.phi_min);
            else if (FK == FK_SOURCES) L.s = 0.0f;
            else {
                float sn, cs;
                sincos_red(F.phi_min + F.phi_range * u, sn, cs);
                L.s = fmaxf(fminf(sn, F.max_scaling), -F.max_scaling);
            }
            L.mp = L.pos;
            field_at<FK>(F, L.tab, L.mp, L.s, L.mn, L.mg);
            L.dir = mul(L.dir, L.mn);                     // photon.cpp:329
            if (P.use_direct) {
                L.ctx = CTX_DIRECT;
                L.md = L.dir;
                L.mtot = L.total;
                L.first = 1;
                L.large = med_large(L, P);
                dlimit = L.large;
                go = true;
            } else {
                ev = EV_SCATTER;
            }
            break;
        }
        case EV_MARCH_END: {
            // movePhotonTillSensor (scene.cpp:622-703) for the direct march and connections, movePhoton
            // (scene.cpp:706-780) for moves; both meet a face here
            const float disy = L.dist_acc;
            const bool sensor = L.ctx == CTX_DIRECT || L.ctx == CTX_CONNECT;
            bool face, hit = false;
            if (sensor) {
                if (L.first) { L.d2s = disy; L.first = 0; } else { L.d2s += disy; }
                L.large -= disy;
                face = !(L.large < 0.0f);
            } else {
                L.rem -= disy;
                face = L.rem > kEps;
            }
            if (face) {
                const float3 n = face_normal(P, L.mp);
                if (sensor && fabsf(P.cam_dir[0] - n.x) < kEps && fabsf(P.cam_dir[1] - n.y) < kEps &&
                    fabsf(P.cam_dir[2] - n.z) < kEps) {
                    hit = true;
                } else {
                    const float mag = sensor ? 1.0f : len3(L.md);
                    const float3 d1 = bsdf_sample(L, P, sensor ? L.md : divs(L.md, mag), n);
                    if (dot3(d1, n) < 0.0f) {                   // reflected: the march goes on
                        L.md = sensor ? d1 : mul(d1, mag);
                        dlimit = sensor ? L.large : L.rem;
                        go = true;
                        break;
                    }
                }
            }
            if (sensor) {
                // directTracing (photon.cpp:41-87: its path length is the photon's own) and
                // addEnergyInParticle (scene.cpp:866-946: its path length is a copy)
                const bool connect = L.ctx == CTX_CONNECT;
                double tot = L.mtot;
                if (!connect) L.total = tot;
                if (hit) {
                    const float3 dsen = normalized(L.md);
                    const float ior = L.mn;
                    float3 refr = dsen;
                    float fw = 1.0f;
                    if (ior > 1.0f) {
                        refr.x = refr.x / ior;
                        refr = normalized(refr);
                        fw = (1.0f - fresnel(dsen.x, refr.x, 1.0f / ior)) / ior / ior;
                    }
                    const float3 out = refr;                    // before the sensor lens
                    float3 p1 = L.mp;
                    float dts = 0.0f;
                    if (propagate_till_sensor(P, p1, refr, dts)) {
                        acc_total(tot, dts, P.fp64);
                        if (!connect) L.total = tot;
                        float val = med_weight(L, P);
                        if (connect) val = val * 6.28318548202514648f;
                        val = val * expf(-med_sigma_t(L, P) * L.d2s);
                        if (connect) {
                            const float fore = dot3(out, ld3(P.cam_dir)) / dot3(dsen, ld3(P.cam_dir));
                            val = val * hg_f(med_g(L, P), divs(L.dir, len3(L.dir)), dsen) * fore;
                        }
                        val = val * fw;
                        splat(L, P, p1, tot, L.depth, val);     // depth 0: direct
                        if (H::on) h->splatted(L, p1, tot, L.depth, val);
                    }
                }
                ev = connect ? EV_SCATTER_ONCE : EV_SCATTER;
            } else {
                const bool ok = !face;                          // else refracted out
                L.total = L.mtot;
                L.pos = L.mp;
                L.dir = L.md;
                if (!ok) { L.end = SMP_END_ESCAPED; ev = EV_FINISH; break; }
                if (L.ctx == CTX_MOVE_FIRST) { L.depth = 1; L.totalDist = L.sampled; }
                else ++L.depth;
                ev = EV_VERTEX;
            }
            break;
        }
        case EV_VERTEX: {
            if (!((P.max_depth < 0 || L.depth <= P.max_depth) &&
                  (P.max_pathlength < 0.0f || L.totalDist <= P.max_pathlength))) {
                L.end = SMP_END_MAX_DEPTH; ev = EV_FINISH; break;
            }
            if (H::on && h->at(L, EV_VERTEX)) return ST_HOOK;
            if (P.use_angular && !(double(L.pos.x - P.cam_origin[0]) < 1e-4)) {
                float3 dts = random_direction(L, P);
                // mp == pos and (mn, mg) are the field at pos: the move march ended there
                L.md = mul(dts, L.mn);
                L.ctx = CTX_CONNECT;
                L.mtot = L.total;
                L.first = 1;
                L.large = med_large(L, P);
                dlimit = L.large;
                go = true;
                break;
            }
            ev = EV_SCATTER_ONCE;
            break;
        }
        case EV_SCATTER:
        case EV_SCATTER_ONCE: {
            const bool once = ev == EV_SCATTER_ONCE;            // at a vertex: a new direction
            if (H::on && h->at(L, ev)) return ST_HOOK;
            if (!roulette(L, P)) { L.end = once ? SMP_END_ABSORBED : SMP_END_NO_SCATTER; ev = EV_FINISH; break; }
            if (once) {
                const float mag = len3(L.dir);
                const float3 d1 = hg_sample(L, P, divs(L.dir, mag));
                L.dir = mul(d1, mag);
            }
            const float dist = -med_mfp(L, P) * logf(draw(L, P));
            L.ctx = once ? CTX_MOVE_VERTEX : CTX_MOVE_FIRST;
            if (!once) L.sampled = dist;
            L.rem = dist;
            L.mp = L.pos;
            L.md = L.dir;
            L.mtot = L.total;
            dlimit = dist;
            go = true;
            at_start = true;
            break;
        }
        default: {   // EV_FINISH
            if (P.records) {
                smp_photon_record *rec = P.records + (L.idx - P.first_photon);
                rec->photon = L.idx;
                rec->end = L.end;
                rec->draws = L.draws;
                rec->depth = L.depth;
                rec->n_splats = L.nspl;
                rec->pos[0] = L.pos.x; rec->pos[1] = L.pos.y; rec->pos[2] = L.pos.z;
                rec->dir[0] = L.dir.x; rec->dir[1] = L.dir.y; rec->dir[2] = L.dir.z;
                rec->total_optical = L.total;
                rec->er_steps = L.steps;
            }
            return ST_FETCH;
        }
        }
        // one march start for every event: the lanes of a warp meet here, and the code is there once
        if (go) {
            begin_march<FK>(L, P, dlimit, at_start);
            if (march_has_steps(L)) return ST_MARCH;
            ev = EV_MARCH_END;
        }
    }
}

struct LaneStats {
    unsigned long long steps = 0, splats = 0, photons = 0, cap = 0, nan = 0, stream = 0;
};

template <int FK>
__device__ __forceinline__ void finish_photon_stats(const Lane &L, LaneStats &S) {
    S.steps += (unsigned long long)L.steps;
    S.splats += (unsigned long long)L.nspl;
    S.photons += 1;
    if (L.end == SMP_END_STEP_CAP) S.cap += 1;
    if (L.end == SMP_END_NAN) S.nan += 1;
    if (L.end == SMP_END_STREAM) S.stream += 1;
}

// ---- shared-memory staging with the Tensor Memory Accelerator ---------------------------------
// One elected thread issues a 1-D bulk copy (cp.async.bulk, no multicast) of `bytes` (a multiple of
// 16, both addresses 16-byte aligned) into this block's shared memory and the block waits on an
// mbarrier. Every wait is bounded: on timeout the block records the failure, waits (bounded) once
// more so no copy is left writing into its shared memory, and reports false.
__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity, int limit) {
    for (int it = 0; it < limit; ++it) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
static __device__ __noinline__ bool stage_to_shared(void *dst, const void *src, unsigned bytes, unsigned long long *err) {
    __shared__ __align__(8) unsigned long long bar;
    const unsigned b = smem_u32(&bar);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(b)
            : "memory");
    }
    bool ok = mbar_wait_bounded(b, 0, 1 << 22);
    if (!ok) {
        mbar_wait_bounded(b, 0, 1 << 22);
        if (threadIdx.x == 0) atomicAdd(err, 1ull);
    }
    __syncthreads();
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

// The lane loop of the persistent kernel: event phase (lanes whose march ended, or that need a
// photon, run their discrete logic together until every live lane marches again; photons come
// from the global counter, one atomic per warp) alternating with the march phase (an untested window or
// eight ER steps per vote, two for point sources, until event_batch lanes, scaled by the live lanes, wait for events). A lane enters with
// `st` = ST_FETCH (no photon) or ST_MARCH (a photon loaded mid-march). All 32 lanes call it.
// A hook (adjoint.cuh's checkpointing trace) also sees each photon's start and end; the render
// kernels use NoHook.
template <int FK, class H = NoHook>
__device__ __forceinline__ void lane_loop(Lane &L, int st, const KParams &P, LaneStats &S, int lane, H *h = nullptr) {
    __shared__ __align__(16) SplineWarp s_warp[FK == FK_SPLINE ? 8 : 1];      // 128-thread blocks
    int pending_ev = EV_NEW;
    for (;;) {
        for (;;) {
            unsigned need = __ballot_sync(kFull, st == ST_FETCH);
            if (need) {
                int leader = __ffs(need) - 1;
                unsigned long long base = 0;
                if (lane == leader) base = atomicAdd(P.counters + CNT_NEXT_PHOTON, (unsigned long long)__popc(need));
                base = __shfl_sync(kFull, base, leader);
                if (st == ST_FETCH) {
                    unsigned long long k = base + __popc(need & ((1u << lane) - 1u)) + (unsigned long long)P.fetch_from;
                    if (k < (unsigned long long)P.n_photons) {
                        L.idx = P.first_photon + (long long)k;
                        L.end = 0;                       // the previous photon's end code
                        st = ST_EVENT;
                        pending_ev = EV_NEW;
                        if (H::on) h->photon_begin(L);
                    } else {
                        st = ST_DONE;
                    }
                }
            }
            if (st == ST_EVENT) {
                st = run_events<FK, H>(L, P, pending_ev, h);
                if (st == ST_FETCH) {
                    finish_photon_stats<FK>(L, S);
                    if (H::on) h->photon_end(L);
                }
                if (H::on && st == ST_MARCH) h->march_begin();
            }
            if (!__any_sync(kFull, st == ST_FETCH)) break;
        }
        const unsigned alive = __ballot_sync(kFull, st != ST_DONE);
        if (alive == 0) break;
        const int thr = max(1, (P.event_batch * __popc(alive) + 16) >> 5);
        // a lane alone in its warp takes long windows; lanes together take short ones, so that none
        // waits long for another's
        const int wcap = (alive & (alive - 1u)) == 0u ? 1024 : 32;
        typename Field<FK>::Cache C;
        C.clear();
        for (;;) {
            if constexpr (FK == FK_SPLINE) {
                if ((alive & (alive - 1u)) == 0u) {
                    const int n = spline_warp_march(L, P, __ffs(alive) - 1, s_warp + 2 * (threadIdx.x >> 5), lane);
                    if (st == ST_MARCH) {
                        if (H::on) h->accepted(n);
                        st = ST_EVENT;
                        pending_ev = EV_MARCH_END;
                    }
                    break;
                }
            }
            if (st == ST_MARCH) {
                bool end = false;
                if constexpr (FK == FK_SOURCES) {
                    // two steps in a straight line (no windows, and no hook: the adjoint has no sources). As a
                    // loop of one step, like the other kinds', the sums in it took half as long again: 8
                    // photons of 2,000 sources 42.6 ms against 28 on the persistent kernel, 150,000 437
                    // against 368 in one launch.
                    end = march_step<FK>(L, P, C) || march_step<FK>(L, P, C);
                } else if (const int w = safe_steps<FK>(L, P, wcap); w >= 4) {
                    march_window<FK>(L, P, w & ~3, C);
                    if (H::on) h->accepted(w & ~3);
                } else {
#pragma unroll 1
                    for (int t = 0; t < 8 && !end; ++t) {
                        const float3 q = L.mp;
                        end = march_step<FK>(L, P, C);
                        if (H::on && (q.x != L.mp.x || q.y != L.mp.y || q.z != L.mp.z)) h->accepted(1);
                    }
                }
                if (end) {
                    st = ST_EVENT;
                    pending_ev = EV_MARCH_END;
                }
            }
            const unsigned waiting = __ballot_sync(kFull, st == ST_EVENT);
            if (__popc(waiting) >= thr || !__any_sync(kFull, st == ST_MARCH)) break;
        }
    }
}

// warp-reduces the statistics, one atomic per warp per counter
__device__ __forceinline__ void flush_stats(LaneStats &S, const KParams &P, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        S.steps += __shfl_down_sync(kFull, S.steps, o);
        S.splats += __shfl_down_sync(kFull, S.splats, o);
        S.photons += __shfl_down_sync(kFull, S.photons, o);
        S.cap += __shfl_down_sync(kFull, S.cap, o);
        S.nan += __shfl_down_sync(kFull, S.nan, o);
        S.stream += __shfl_down_sync(kFull, S.stream, o);
    }
    if (lane == 0 && S.photons) {
        atomicAdd(P.counters + CNT_STEPS, S.steps);
        atomicAdd(P.counters + CNT_SPLATS, S.splats);
        atomicAdd(P.counters + CNT_PHOTONS, S.photons);
        if (S.cap) atomicAdd(P.counters + CNT_STEP_CAP, S.cap);
        if (S.nan) atomicAdd(P.counters + CNT_NAN, S.nan);
        if (S.stream) atomicAdd(P.counters + CNT_STREAM, S.stream);
    }
}

template <int FK>
__global__ void __launch_bounds__(128, lane_blocks(FK)) march_kernel(const __grid_constant__ KParams P) {
    extern __shared__ __align__(16) float4 smem_tab[];
    const int lane = threadIdx.x & 31;
    Lane L;
    L.end = 0;
    L.idx = 0;
    L.tab = P.field.btab;
    if (FK <= FK_BESSELN && P.field.btab != nullptr) {
        if (!stage_to_shared(smem_tab, P.field.btab, unsigned(P.field.bnodes) * 16u, P.counters + CNT_STAGE_TIMEOUT))
            return;                                  // whole block: other blocks take the photons
        L.tab = smem_tab;
    }
    LaneStats S;
    lane_loop<FK>(L, ST_FETCH, P, S, lane);
    flush_stats(S, P, lane);
}

// n(p) alone of the point-source field at host-given points, bit for bit sources_field's sum. Its sum
// runs over the arcs' rows: a source's x depends on its row and (y, z) on its place in the row, so a
// point's squared distance in (y, z) to each of the row's nt places is worked out once (in shared memory,
// four to a 16-byte load, a column of its own per thread) and a term is one FMA, the reciprocal square
// root, the phase and one cosine: 15 instructions instead of the 33 with the gradient, and two
// conversion-pipe operations instead of three, which bound it (16 cycles a term and scheduler).
static constexpr int kValuesBlock = 128;
static __global__ void __launch_bounds__(kValuesBlock)
sources_values_kernel(const __grid_constant__ FieldParams F, int nt, long long n, const double *pts, double *n_out) {
    extern __shared__ __align__(16) float4 s_yz[];            // [(nt + 3) / 4][kValuesBlock]
    const long long k = (long long)blockIdx.x * kValuesBlock + threadIdx.x;
    const bool on = k < n;
    const float3 p = on ? f3(float(pts[3 * k]), float(pts[3 * k + 1]), float(pts[3 * k + 2])) : f3(0.0f, 0.0f, 0.0f);
    if (!on) return;                                          // no barrier below: a column is its thread's own
    if (p.x > F.egap || p.x < F.sgap) {
        n_out[k] = F.n_o;
        return;
    }
    float4 *col = s_yz + threadIdx.x;
    float *colf = reinterpret_cast<float *>(col);
    const int nz = F.nsources / nt, full = nt >> 2;
    float rif = 0.0f;
    const float pi = 3.14159265358979f;
    for (int c = 1; c <= F.n_coeff; ++c) {
        const float fc = float(c);
        const float sf = ((c & 1) ? 4.0f : -4.0f) / (fc * pi * fc * pi * float(F.nsources));
        float trif = 0.0f;
        for (int arc = 0; arc < 2; ++arc) {
            if (!(arc == 0 ? F.active1 : F.active2)) continue;
            const float ph = arc == 0 ? F.phase1 : F.phase2;
            const float4 *cen = F.centers + arc * F.nsources;
            for (int i = 0; i < nt; ++i) {
                const float4 q = __ldg(cen + i);
                const float dy = p.y - q.y, dz = p.z - q.z;
                colf[(i >> 2) * (4 * kValuesBlock) + (i & 3)] = fmaf(dy, dy, dz * dz);
            }
            auto term = [&](float dx, float yz) {
                const float rr2 = fmaf(dx, dx, yz);
                const float ir = rsqrt_fast(rr2);             // rsqrtf's value for every normal rr2
                const float r = rr2 * ir;
                const float krc = F.k_r * r * fc;
                float sn, cs;
                sincos_near(krc + ph, sn, cs);
                trif = fmaf(cs, ir, trif);
            };
            for (int j = 0; j < nz; ++j) {
                const float dx = p.x - __ldg(&cen[size_t(j) * nt].x);
#pragma unroll 2
                for (int i = 0; i < full; ++i) {
                    const float4 t = col[i * kValuesBlock];
                    term(dx, t.x); term(dx, t.y); term(dx, t.z); term(dx, t.w);
                }
                for (int i = full << 2; i < nt; ++i) term(dx, colf[(i >> 2) * (4 * kValuesBlock) + (i & 3)]);
            }
        }
        rif = fmaf(trif, sf, rif);
    }
    n_out[k] = fmaf(F.n_scaling, rif, F.n_o);
}

// n(p), grad n(p) at host-given points with the march's own field code
template <int FK>
__global__ void field_probe_kernel(const __grid_constant__ FieldParams F, float s, long long n,
                                   const double *pts, double *n_out, double *g_out) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 p = f3(float(pts[3 * i]), float(pts[3 * i + 1]), float(pts[3 * i + 2]));
    float nn;
    float3 g;
    Field<FK>::eval(F, F.btab, p, s, nn, g);
    n_out[i] = nn;
    g_out[3 * i] = g.x; g_out[3 * i + 1] = g.y; g_out[3 * i + 2] = g.z;
}

}  // namespace smp
