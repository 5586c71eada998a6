// The served Kerr march, one or two rays per lane.
//
// F2 holds two FP32 values in a register pair and computes with the packed
// f32x2 instructions of sm_100 (add, mul and fma of two floats, each rounded
// as its scalar instruction rounds). The scalar step (lanes.cuh) is bound by
// instruction issue: 89 % of the issue slots busy, the FMA pipe 64 %, 425
// instructions per ray step. A packed instruction does the work of two in
// one issue slot and two cycles of the FMA pipe (measured: 2.06 cycles a
// warp for fma, add and mul), so with two rays in a lane the arithmetic
// takes half the issue slots. Min, max, selects, reciprocals and square
// roots have no packed form and run once per ray. A ray step then issues 249
// instructions, the azimuth's sine and cosine and the path taken only near
// the slab. What bounds it now is the FMA pipe, on which a packed instruction
// takes two cycles, and latency: 16 warps per SM (128 registers) keep the
// pipe 71 % and the issue slots 62 % busy; 20 warps (96 registers, spilled)
// were slower, as was the RK4 loop rolled. Measured on a 1920x1080 4096-step
// Kerr still in one wave: 6.55 -> 5.54 ms, of which 5.85 before the rays went
// through the image in tiles; on the mixed served stream 79.5 -> 95 G
// ray-steps/s. (Hamilton's equations in
// 32 operations instead of 40 and the RK4 sum in its final weights reached
// 5.35 ms and 103 G, but round differently, and a ray's last bit decides
// which cell of the starfield it meets.)
//
// Schwarzschild rays stay one to a lane (lanes.cuh): they take 58 steps
// rather than 230 and gather in 60 % of them, which pairs do not speed up,
// and two to a lane they ran 1.35 times slower.
//
// Everything here is a template over R: F2 (two neighbouring pixels per
// lane) or float (one ray per lane). Radius, polar angle, their momenta and
// the gauges advance operation by operation as k_step's compiled code rounds
// them (lanes.cuh): every multiply-add is written out as the fused or the
// separate operation it is there, so steps, outcomes and drifts are the image
// march's bit for bit (tested), and a ray's values do not depend on the ray
// it shares a lane with. The azimuth, which enters none of these, is not: the
// compiler contracts its rate differently from kernel to kernel, and a
// sample's place and path come from a series of their own (kerr_step);
// colours differ in the last bits.
#pragma once

#include "lanes.cuh"

namespace gg {

// ------------------------------------------------------------- arithmetic

template <typename R> struct Rays;
template <> struct Rays<float> {
    static constexpr int N = 1;
};
template <> struct Rays<F2> {
    static constexpr int N = 2;
};

// One value for every ray of a lane.
template <typename R> __device__ __forceinline__ R all(float x);
template <> __device__ __forceinline__ float all<float>(float x) { return x; }
template <> __device__ __forceinline__ F2 all<F2>(float x) { return f2(x, x); }

// Ray j's value, and a lane's from its rays'.
__device__ __forceinline__ float part(float a, int) { return a; }
__device__ __forceinline__ float part(F2 a, int j) {
    const float2 p = parts(a);
    return j == 0 ? p.x : p.y;
}
template <typename R> __device__ __forceinline__ R join(const float* x);
template <> __device__ __forceinline__ float join<float>(const float* x) { return x[0]; }
template <> __device__ __forceinline__ F2 join<F2>(const float* x) { return f2(x[0], x[1]); }

__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float neg(float a) { return -a; }
__device__ __forceinline__ F2 neg(F2 a) {
    const float2 p = parts(a);
    return f2(-p.x, -p.y);
}
template <typename R> __device__ __forceinline__ R sub(R a, R b) { return add(a, neg(b)); }
// a b where a plain addition follows. The assembler would contract a packed
// product and the addition into one fma; a packed fma with an addend of -0
// that it does not know rounds the product and adds nothing to it.
__device__ __forceinline__ float product(float a, float b, float) { return __fmul_rn(a, b); }
__device__ __forceinline__ F2 product(F2 a, F2 b, float minus_zero) { return mad(a, b, f2(minus_zero, minus_zero)); }

// A number of the lane's type, from the double it is closest to.
template <typename R> __device__ __forceinline__ R num(double x) { return all<R>((float)x); }

// A scalar function of each ray's value.
template <typename Fn> __device__ __forceinline__ float each(float a, Fn f) { return f(a); }
template <typename Fn> __device__ __forceinline__ F2 each(F2 a, Fn f) {
    const float2 p = parts(a);
    return f2(f(p.x), f(p.y));
}
__device__ __forceinline__ F2 rcp(F2 a) {
    return each(a, [](float x) { return rcp(x); });
}
__device__ __forceinline__ F2 asqrt(F2 a) {
    return each(a, [](float x) { return asqrt(x); });
}
template <typename R> __device__ __forceinline__ R clamp(R a, float lo, float hi) {
    return each(a, [=](float x) { return fminf(fmaxf(x, lo), hi); });
}
template <typename R> __device__ __forceinline__ R magnitude(R a) {
    return each(a, [](float x) { return fabsf(x); });
}
__device__ __forceinline__ float lesser(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ F2 lesser(F2 a, F2 b) {
    const float2 p = parts(a), q = parts(b);
    return f2(fminf(p.x, q.x), fminf(p.y, q.y));
}
// The largest magnitude, and the smallest value, among a lane's rays.
__device__ __forceinline__ float largest(float a) { return fabsf(a); }
__device__ __forceinline__ float largest(F2 a) {
    const float2 p = parts(a);
    return fmaxf(fabsf(p.x), fabsf(p.y));
}
__device__ __forceinline__ float smallest(float a) { return a; }
__device__ __forceinline__ float smallest(F2 a) {
    const float2 p = parts(a);
    return fminf(p.x, p.y);
}

// fast_sincos of every ray's angle, bit for bit up to |x| = 2^22 pi/2 (only a
// state that blew up is beyond). k = rint(x 2/pi) comes from adding 1.5 2^23
// to the rounded product, whose sum holds k in its low bits: no conversion
// instructions. (Fused, near ties k is the other neighbour: of 635,000 rays
// one ended with another drift.)
template <typename R> __device__ __forceinline__ void sincos_of(R x, float minus_zero, R* s_out, R* c_out) {
    constexpr int N = Rays<R>::N;
    const R kk = add(product(x, all<R>(0.636619772367581f), minus_zero), all<R>(12582912.0f));
    const R k = add(kk, all<R>(-12582912.0f));
    R r = mad(k, all<R>(-1.57079601287841796875f), x);
    r = mad(k, all<R>(-3.13916478650481e-07f), r);
    const R r2 = mul(r, r);
    R ps = mad(r2, num<R>(1.0 / 362880.0), num<R>(-1.0 / 5040.0));
    ps = mad(r2, ps, num<R>(1.0 / 120.0));
    ps = mad(r2, ps, num<R>(-1.0 / 6.0));
    const R sr = mad(mul(r, r2), ps, r);
    R pc = mad(r2, num<R>(-1.0 / 3628800.0), num<R>(1.0 / 40320.0));
    pc = mad(r2, pc, num<R>(-1.0 / 720.0));
    pc = mad(r2, pc, num<R>(1.0 / 24.0));
    pc = mad(r2, pc, num<R>(-0.5));
    const R cr = mad(r2, pc, num<R>(1.0));
    float s[N], c[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t b = __float_as_uint(part(kk, j));
        const bool swap = (b & 1u) != 0u;
        s[j] = __uint_as_float(__float_as_uint(swap ? part(cr, j) : part(sr, j)) ^ ((b << 30) & 0x80000000u));
        c[j] = __uint_as_float(__float_as_uint(swap ? part(sr, j) : part(cr, j)) ^ (((b + 1u) << 30) & 0x80000000u));
    }
    *s_out = join<R>(s);
    *c_out = join<R>(c);
}

template <typename R> struct SinCos {
    R s, c;
};

// rotate's other cases: the long series, and beyond 0.35 the angle afresh.
template <typename R> __device__ __forceinline__ SinCos<R> rotate_more(R st0, R ct0, R delta, R angle) {
    constexpr int N = Rays<R>::N;
    const R d2 = mul(delta, delta), d3 = mul(delta, d2);
    const R ss = mad(d3, num<R>(-1.0 / 6.0), delta);
    const R cs = mad(d2, mad(d2, num<R>(1.0 / 24.0), num<R>(-0.5)), num<R>(1.0));
    R ps = mad(d2, num<R>(-1.0 / 5040.0), num<R>(1.0 / 120.0));
    ps = mad(d2, ps, num<R>(-1.0 / 6.0));
    const R sl = mad(d3, ps, delta);
    R pc = mad(d2, num<R>(1.0 / 40320.0), num<R>(-1.0 / 720.0));
    pc = mad(d2, pc, num<R>(1.0 / 24.0));
    pc = mad(d2, pc, num<R>(-0.5));
    const R cl = mad(d2, pc, num<R>(1.0));
    float s[N], c[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const bool is_short = fabsf(part(delta, j)) <= 0.02f;
        s[j] = is_short ? part(ss, j) : part(sl, j);
        c[j] = is_short ? part(cs, j) : part(cl, j);
    }
    const R sd = join<R>(s), cd = join<R>(c);
    SinCos<R> o{mad(st0, cd, mul(ct0, sd)), mad(ct0, cd, neg(mul(st0, sd)))};
    if (largest(delta) <= 0.35f) return o;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        s[j] = part(o.s, j);
        c[j] = part(o.c, j);
        if (!(fabsf(part(delta, j)) <= 0.35f)) fast_sincos(part(angle, j), &s[j], &c[j]);
    }
    return SinCos<R>{join<R>(s), join<R>(c)};
}
// Out of line for pairs, as are the other rare cases of a step: the loop's
// instructions then stay closer to the instruction cache (2 % on the served
// stream). In line for one ray to a lane: there it is the last few rays, which
// pass close to the hole and so come here often, that a wave waits for.
__noinline__ __device__ SinCos<F2> rotate_pair(F2 st0, F2 ct0, F2 delta, F2 angle) {
    return rotate_more(st0, ct0, delta, angle);
}
__device__ __forceinline__ SinCos<F2> rotate_far(F2 st0, F2 ct0, F2 delta, F2 angle) {
    return rotate_pair(st0, ct0, delta, angle);
}
__device__ __forceinline__ SinCos<float> rotate_far(float st0, float ct0, float delta, float angle) {
    return rotate_more(st0, ct0, delta, angle);
}

// sin and cos of angles delta beyond those whose sine and cosine are (st0,
// ct0), ray by ray as sincos_shift takes them: its short series for |delta|
// <= 0.02, the usual size of a stage's offset, its long one to 0.35, and
// afresh from at() beyond.
template <typename R, typename At>
__device__ __forceinline__ void rotate(R st0, R ct0, R delta, At at, R* st, R* ct) {
    if (largest(delta) <= 0.02f) {
        const R d2 = mul(delta, delta);
        const R sd = mad(mul(delta, d2), num<R>(-1.0 / 6.0), delta);
        const R cd = mad(d2, mad(d2, num<R>(1.0 / 24.0), num<R>(-0.5)), num<R>(1.0));
        *st = mad(st0, cd, mul(ct0, sd));
        *ct = mad(ct0, cd, neg(mul(st0, sd)));
    } else {
        const SinCos<R> f = rotate_far(st0, ct0, delta, at());
        *st = f.s;
        *ct = f.c;
    }
}

// x += k w, compensated (comp_add): the increment is rounded before the error
// word joins it.
template <typename R, typename View> __device__ __forceinline__ void settle(R& x, R& e, R k, R w, const View& u) {
    const R b = add(product(k, w, u.minus_zero), e);
    const R t = add(x, b);
    e = sub(b, sub(t, x));
    x = t;
}

// 2 (1 - cos d), the squared chord of an arc d at radius one: for |d| <=
// 0.35 as d^2 (1 - d^2/12 + d^4/360 - d^6/20160), the next term below 4e-11.
template <typename R> __device__ __forceinline__ R chord_series(R d) {
    const R d2 = mul(d, d);
    const R p = mad(d2, mad(d2, num<R>(-1.0 / 20160.0), num<R>(1.0 / 360.0)), num<R>(-1.0 / 12.0));
    return mul(d2, mad(d2, p, num<R>(1.0)));
}
template <typename R> __noinline__ __device__ R chord_squared_far(R d) {
    return each(d, [](float x) {
        if (fabsf(x) <= 0.35f) return chord_series(x);
        float s, c;
        fast_sincos(x, &s, &c);
        return fmaf(-2.0f, c, 2.0f);
    });
}
template <typename R> __device__ __forceinline__ R chord_squared(R d) {
    return largest(d) <= 0.35f ? chord_series(d) : chord_squared_far(d);
}

// ------------------------------------------------------------- shading

// What a gather reads of a request. A warp on one request keeps them in
// shared memory: read where a sample is taken, they hold no registers in the
// steps outside the slab.
struct GatherWords {
    cudaTextureObject_t emission, velocity;
    float half_extent, opacity;
    uint32_t redshift, pad;
};

// The request as the steps of a warp that marches one request see it.
struct WarpView {
    float factor, escape, minus_zero;
    bool gas;
    const volatile GatherWords* words;
    __device__ __forceinline__ GatherView gather() const {
        return GatherView{words->emission, words->velocity, words->half_extent, words->opacity, words->redshift};
    }
};

// The same for a lane whose request differs from its neighbours'.
struct LaneView {
    float factor, escape, minus_zero;
    bool gas;
    const MarchUniforms* u;
    cudaTextureObject_t emission, velocity;
    __device__ __forceinline__ GatherView gather() const { return gather_view(*u, emission, velocity); }
};

// What a lane keeps of each of its rays besides the state. The served
// targets hold no depth, so no depth weights are kept.
template <int N> struct Shade {
    float longest[N];  // the step length's limit; 0 once the ray has ended, which holds it where it is
    float min_r[N];
    float3 color[N];
    float transmittance[N];
    uint32_t end[N];   // steps taken | outcome << 30, once it has ended
    uint32_t samples;  // of all the lane's rays
};

__device__ __forceinline__ uint32_t end_word(uint32_t steps, uint32_t outcome) { return steps | (outcome << 30); }
__device__ __forceinline__ uint32_t end_steps(uint32_t w) { return w & 0x3fffffffu; }
__device__ __forceinline__ uint32_t end_outcome(uint32_t w) { return w >> 30; }
static_assert(STEP_CAP_STILL < (1u << 30) && RayExhausted < 4, "the step count and outcome share a word");

template <int N> __device__ __forceinline__ void begin_shade(Shade<N>& sh, int j, float min_r, float longest) {
    sh.longest[j] = longest;
    sh.min_r[j] = min_r;
    sh.color[j] = make_float3(0.0f, 0.0f, 0.0f);
    sh.transmittance[j] = 1.0f;
    sh.end[j] = 0u;
}

template <int N> __device__ __forceinline__ bool alive(const Shade<N>& sh, int j) { return sh.longest[j] > 0.0f; }
template <int N> __device__ __forceinline__ bool any_alive(const Shade<N>& sh) {
    return fmaxf(sh.longest[0], sh.longest[N - 1]) > 0.0f;
}

// One in-slab sample into ray j's colour: gather_sample_with<true>, with
// every multiply-add written out so that each copy of it (one or two rays to
// a lane) rounds alike.
template <int N, typename Direction>
__device__ __forceinline__ void gather_ray(Shade<N>& sh, int j, const GatherView& gv, float3 at, float lapse, float path,
                                           Direction direction) {
    if (!(sh.transmittance[j] > 0.004f)) return;
    sh.samples += 1u;
    const float3 c = volume_coordinates(at, gv.half_extent);
    const float4 e = tex3D<float4>(gv.emission, c.x, c.y, c.z);
    if (!(e.w > 0.0f)) return;
    float g3 = 1.0f;
    if (gv.redshift != 0u) {
        const float4 v = tex3D<float4>(gv.velocity, c.x, c.y, c.z);
        const float speed2 = fmaf(v.z, v.z, fmaf(v.y, v.y, __fmul_rn(v.x, v.x)));
        const float magnitude = asqrt(speed2);
        const float t = rcp(__fadd_rn(__expf(__fmul_rn(fminf(magnitude, 8.0f), 2.0f / GAS_SPEED_CEILING)), 1.0f));
        const float beta = __fmul_rn(GAS_SPEED_CEILING, fmaf(-2.0f, t, 1.0f));
        const float scale = magnitude > 0.0f ? __fmul_rn(beta, rcp(magnitude)) : 0.0f;
        const float gravity = asqrt(fmaxf(lapse, 0.0f));
        const float3 d = direction();
        const float along = fmaf(d.z, v.z, fmaf(d.y, v.y, __fmul_rn(d.x, v.x)));
        const float g = __fmul_rn(__fmul_rn(gravity, asqrt(fmaf(-beta, beta, 1.0f))), rcp(fmaf(along, scale, 1.0f)));
        const float bulk = fminf(__fmul_rn(e.w, 1.0f / BEAMING_DENSITY_FLOOR), 1.0f);
        const float gr3 = __fmul_rn(__fmul_rn(gravity, gravity), gravity);
        g3 = fmaf(fmaf(__fmul_rn(g, g), g, -gr3), bulk, gr3);
    }
    const float alpha = __fsub_rn(1.0f, __expf(__fmul_rn(__fmul_rn(-gv.opacity, e.w), path)));
    const float k = __fmul_rn(__fmul_rn(sh.transmittance[j], g3), path);
    sh.color[j].x = fmaf(e.x, k, sh.color[j].x);
    sh.color[j].y = fmaf(e.y, k, sh.color[j].y);
    sh.color[j].z = fmaf(e.z, k, sh.color[j].z);
    sh.transmittance[j] = __fmul_rn(sh.transmittance[j], __fsub_rn(1.0f, alpha));
}

// --------------------------------------------------------------------- Kerr

template <typename R> struct KerrRays {
    static constexpr int N = Rays<R>::N;
    R r, th, ph, pr, pt;       // state
    R er, eth, eph, epr, ept;  // its error words
    R st, ct;                  // sin and cos of th
    R E, L, aE, aL, L2, a2E2, two_aEL, carter0;
    float gauge[N];  // max over the steps' gauges; a captured ray's drift, final
    float a, a2, capture;
    Shade<N> sh;
};

// A ray's drift and its pixel are out of line, compiled once for every kernel
// and R, so that they round alike; the launch stays inline (out of line it
// cost the served stream 3 %).
__device__ __forceinline__ KLane<float> kerr_launched(const MarchUniforms& u, uint2 pixel) {
    KLane<float> l;
    k_init(l, to_f3(u.cameraPosition), camera_direction(u, pixel.x, pixel.y), u);
    return l;
}
__noinline__ __device__ float kerr_drift(const KLane<float>& l) { return k_drift(l); }
__noinline__ __device__ PixelResult kerr_pixel(const KLane<float>& l, const MarchUniforms& u, const float4* blackbody) {
    return k_finish(l, u, blackbody);
}

// The photon's direction at a sample (k_direction).
__device__ __forceinline__ float3 kerr_heading(const KLane<float>& l, float sp, float cp) {
    const KConst<float>& k = l.k;
    const float r = l.s.r, st = l.st, ct = l.ct;
    const float delta = mad(r, add(r, -2.0f), k.a2);
    const float inv_sigma = rcp(mad(k.a2, mul(ct, ct), mul(r, r)));
    float inv_sin2, inv_sc;
    k_sin_inverses(st, &inv_sin2, &inv_sc);
    const float p = mad(mad(r, r, k.a2), k.E, -k.aL);
    const float rdot = mul(mul(delta, l.s.pr), inv_sigma);
    const float r_thdot = mul(mul(r, l.s.pt), inv_sigma);
    const float phdot = mul(add(mad(k.a, mul(p, rcp(delta)), mul(k.L, inv_sin2)), -k.aE), inv_sigma);
    const float r_st_phdot = mul(mul(r, st), phdot);
    const float in_plane = mad(rdot, st, mul(r_thdot, ct));  // along (cp, sp, 0)
    const float x = mad(in_plane, cp, -mul(r_st_phdot, sp)), y = mad(in_plane, sp, mul(r_st_phdot, cp));
    const float z = mad(rdot, ct, -mul(r_thdot, st));
    const float len2 = mad(z, z, mad(y, y, mul(x, x)));
    if (!(len2 > 0.0f)) return make_float3(mul(st, cp), mul(st, sp), ct);
    const float w = rsqrtT(len2);
    return make_float3(mul(x, w), mul(y, w), mul(z, w));
}

// The lane's rays from launched scalar lanes (k_init).
template <typename R>
__device__ __forceinline__ void kerr_load(KerrRays<R>& p, const KLane<float>* l, const float* longest) {
    constexpr int N = Rays<R>::N;
    float v[15][N];
    p.sh.samples = 0u;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const KLane<float>& q = l[j];
        const float w[15] = {q.s.r, q.s.th, q.s.ph, q.s.pr, q.s.pt, q.st, q.ct, q.k.E, q.k.L, q.k.aE, q.k.aL, q.carter0,
                         q.k.L2, q.k.a2E2, q.k.two_aEL};
#pragma unroll
        for (int i = 0; i < 15; ++i) v[i][j] = w[i];
        begin_shade(p.sh, j, q.min_r, longest[j]);
        p.gauge[j] = 0.0f;
    }
    p.r = join<R>(v[0]);
    p.th = join<R>(v[1]);
    p.ph = join<R>(v[2]);
    p.pr = join<R>(v[3]);
    p.pt = join<R>(v[4]);
    p.st = join<R>(v[5]);
    p.ct = join<R>(v[6]);
    p.E = join<R>(v[7]);
    p.L = join<R>(v[8]);
    p.aE = join<R>(v[9]);
    p.aL = join<R>(v[10]);
    p.carter0 = join<R>(v[11]);
    p.L2 = join<R>(v[12]);
    p.a2E2 = join<R>(v[13]);
    p.two_aEL = join<R>(v[14]);
    p.er = p.eth = p.eph = p.epr = p.ept = num<R>(0.0);
    p.a = l[0].k.a;
    p.a2 = l[0].k.a2;
    p.capture = l[0].capture;
}

// Ray j as the scalar lane that k_drift, k_direction and k_finish read.
template <typename R> __device__ __forceinline__ KLane<float> kerr_lane(const KerrRays<R>& p, int j) {
    KLane<float> l;
    l.s = KState<float>{part(p.r, j), part(p.th, j), part(p.ph, j), part(p.pr, j), part(p.pt, j)};
    l.k.a = p.a;
    l.k.a2 = p.a2;
    l.k.E = part(p.E, j);
    l.k.L = part(p.L, j);
    l.k.aE = part(p.aE, j);
    l.k.aL = part(p.aL, j);
    l.k.L2 = part(p.L2, j);
    l.k.a2E2 = part(p.a2E2, j);
    l.k.two_aEL = part(p.two_aEL, j);
    l.k.four_E = mul(4.0f, l.k.E);
    l.st = part(p.st, j);
    l.ct = part(p.ct, j);
    l.carter0 = part(p.carter0, j);
    l.scale = fmaxf(fabsf(l.carter0), mul(l.k.E, l.k.E));
    l.gauge = p.gauge[j];
    l.steps = end_steps(p.sh.end[j]);
    return l;
}

template <typename R> struct KerrSlope {
    R r, th, ph, pr, pt;
    R F, inv_sigma, inv_sin2, r2, ct2;  // 2 Sigma H, 1/Sigma, 1/sin^2, r^2, cos^2
};

// k_sin_inverses for every ray.
template <typename R> __device__ __forceinline__ void sin_inverses(R st, R* inv_sin2, R* inv_sc) {
    constexpr int N = Rays<R>::N;
    float i[N], c[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        i[j] = rcp(fmaxf(fabsf(part(st, j)), 1e-4f));
        c[j] = part(st, j) > 0.0f ? i[j] : 1e4f;
    }
    const R inv = join<R>(i);
    *inv_sin2 = mul(inv, inv);
    *inv_sc = join<R>(c);
}

// k_derivative's Sigma times Hamilton's equations (Kerr.h:63-90), operation
// by operation as the scalar step's compiled code rounds them.
template <typename R>
__device__ __forceinline__ KerrSlope<R> kerr_slope(const KerrRays<R>& k, R r, R pr, R pt, R st, R ct, float minus_zero) {
    KerrSlope<R> o;
    const R a2 = all<R>(k.a2);
    o.r2 = product(r, r, minus_zero);
    o.ct2 = mul(ct, ct);
    const R delta = mad(r, add(r, num<R>(-2.0)), a2);
    o.inv_sigma = rcp(mad(a2, o.ct2, o.r2));
    const R inv_delta = rcp(delta);
    const R sin2 = each(mul(st, st), [](float x) { return fmaxf(x, 1e-8f); });
    R inv_sin2, inv_sc;
    sin_inverses(st, &inv_sin2, &inv_sc);
    const R ra = add(o.r2, a2);
    const R p = mad(ra, k.E, neg(k.aL));
    o.inv_sin2 = inv_sin2;
    const R g = mad(k.a2E2, sin2, mad(k.L2, inv_sin2, neg(k.two_aEL)));
    const R pr2 = mul(pr, pr);
    const R pp = mul(p, p);
    const R p2d = product(pp, inv_delta, minus_zero);
    o.F = mad(delta, pr2, mad(pt, pt, sub(g, p2d)));
    const R two_h = mul(o.F, o.inv_sigma);
    // f_r / 2: k_derivative's f_r with every term halved, which rounds alike.
    const R m1 = add(r, num<R>(-1.0));
    const R half_fr = mad(m1, pr2, mul(inv_delta, mad(p2d, m1, mul(mul(mul(num<R>(-2.0), k.E), r), p))));
    o.r = mul(delta, pr);
    o.th = pt;
    o.ph = mad(all<R>(-k.a), k.E, mad(all<R>(k.a), mul(p, inv_delta), mul(k.L, inv_sin2)));
    o.pr = mad(r, two_h, neg(half_fr));
    o.pt = mul(neg(ct), mad(mul(a2, st), two_h, mad(k.a2E2, st, mul(mul(neg(k.L2), inv_sin2), inv_sc))));
    return o;
}

// Whether ray j's state is five finite numbers.
template <typename R> __device__ __forceinline__ bool finite_state(const KerrRays<R>& p, int j) {
    const float sum = part(p.r, j) + part(p.th, j) + part(p.ph, j) + part(p.pr, j) + part(p.pt, j);
    return fabsf(sum) < INFINITY;
}

// One step of every ray of the lane (march.metal:140-173), after `step`
// others. Rays that ended stay where they are: their step length is zero.
template <typename R, typename View>
__device__ __forceinline__ void kerr_step(KerrRays<R>& p, const View& u, uint32_t step) {
    constexpr int N = Rays<R>::N;
    Shade<N>& sh = p.sh;
    // kerrStepLength (Kerr.h:177-186)
    R h;
    {
        const R above = add(p.r, all<R>(KERR_CAPTURE_MARGIN - p.capture));
        const R pole = clamp(mul(num<R>(1.0 / 0.08), p.st), 0.05f, 1.0f);
        const R want = mul(lesser(mul(all<R>(u.factor), p.r), mul(num<R>(0.2), above)), pole);
        float hj[N];
#pragma unroll
        for (int j = 0; j < N; ++j) hj[j] = fminf(fmaxf(part(want, j), 0.002f), sh.longest[j]);
        h = join<R>(hj);
    }
    const R hh = mul(num<R>(0.5), h), w = mul(h, num<R>(1.0 / 6.0));
    const R r0 = p.r, ph0 = p.ph, st0 = p.st, ct0 = p.ct;
    R br, bth, bph, bpr, bpt;
    R xr = p.r, xpr = p.pr, xpt = p.pt, st = p.st, ct = p.ct;
#pragma unroll
    for (int stage = 0; stage < 4; ++stage) {
        const KerrSlope<R> d = kerr_slope(p, xr, xpr, xpt, st, ct, u.minus_zero);
        if (stage == 0) {
            // The gauge of the state the step starts from (k_gauge); the
            // launch state has none.
            const R carter = mad(d.ct2, mad(p.L2, d.inv_sin2, neg(p.a2E2)), mul(xpt, xpt));
            const R off = sub(carter, p.carter0), null = mul(d.F, rcp(d.r2));
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const float most = fmaxf(p.gauge[j], fmaxf(fabsf(part(off, j)), fabsf(part(null, j))));
                p.gauge[j] = step > 0u && alive(sh, j) ? most : p.gauge[j];
            }
        }
        if (stage == 0) {
            br = mul(d.r, d.inv_sigma);
            bth = mul(d.th, d.inv_sigma);
            bph = mul(d.ph, d.inv_sigma);
            bpr = mul(d.pr, d.inv_sigma);
            bpt = mul(d.pt, d.inv_sigma);
        } else {
            const R k = stage == 3 ? d.inv_sigma : mul(num<R>(2.0), d.inv_sigma);
            br = mad(d.r, k, br);
            bth = mad(d.th, k, bth);
            bph = mad(d.ph, k, bph);
            bpr = mad(d.pr, k, bpr);
            bpt = mad(d.pt, k, bpt);
        }
        if (stage == 3) break;
        const R wx = mul(stage < 2 ? hh : h, d.inv_sigma);
        xr = mad(d.r, wx, p.r);
        xpr = mad(d.pr, wx, p.pr);
        xpt = mad(d.pt, wx, p.pt);
        rotate(st0, ct0, mul(d.th, wx), [&] { return mad(d.th, wx, p.th); }, &st, &ct);
    }
    settle(p.r, p.er, br, w, u);
    settle(p.th, p.eth, bth, w, u);
    settle(p.ph, p.eph, bph, w, u);
    settle(p.pr, p.epr, bpr, w, u);
    settle(p.pt, p.ept, bpt, w, u);
    sincos_of(p.th, u.minus_zero, &p.st, &p.ct);
    // The azimuth enters only a sample's position: its sine and cosine, and
    // the path since the previous state (the chord between the two in
    // cylinder coordinates, in which nothing cancels), are taken only near
    // the slab.
    const R z = mul(p.r, p.ct);
    if (smallest(magnitude(z)) < DISK_SLAB_HALF_HEIGHT && u.gas) {
        R sp, cp;
        sincos_of(p.ph, u.minus_zero, &sp, &cp);
        const R rho = mul(asqrt(mad(p.r, p.r, all<R>(p.a2))), p.st);
        const R axial0 = asqrt(mad(r0, r0, all<R>(p.a2))), rho0 = mul(axial0, st0);
        const R out = mad(neg(axial0), st0, rho), up = mad(neg(r0), ct0, z);
        const R path = asqrt(mad(out, out, mad(mul(rho, rho0), chord_squared(sub(p.ph, ph0)), mul(up, up))));
        const R px = mul(rho, cp), py = mul(rho, sp);
        const GatherView gv = u.gather();
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float r = part(p.r, j);
            const float3 at = make_float3(part(px, j), part(py, j), part(z, j));
            if (alive(sh, j) && r > p.capture && in_slab(at, gv.half_extent)) {
                const float ctj = part(p.ct, j);
                const float lapse = fmaf(-2.0f * r, rcp(fmaf(p.a2, ctj * ctj, r * r)), 1.0f);
                gather_ray(sh, j, gv, at, fmaxf(lapse, 0.0f), part(path, j), [&] {
                    return kerr_heading(kerr_lane(p, j), part(sp, j), part(cp, j));
                });
            }
        }
    }
    bool ended = false;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const float r = part(p.r, j);
        sh.min_r[j] = fminf(sh.min_r[j], r);
        ended = ended || (alive(sh, j) && !(r > p.capture && r < u.escape));
    }
    if (ended) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float r = part(p.r, j);
            if (!alive(sh, j) || (r > p.capture && r < u.escape)) continue;
            // A last step beside the horizon can leave a state that is no
            // number and would stay so to the step cap: it ends as one that
            // got there, with a drift over any budget and a radius inside any
            // limit, so that it is re-integrated in FP64 (needs_fp64).
            const bool in = r <= p.capture;
            sh.end[j] = end_word(step + 1u, in ? RayCaptured : r >= u.escape ? RayEscaped : RayExhausted);
            sh.longest[j] = 0.0f;
            if (!in && !finite_state(p, j)) {
                p.gauge[j] = INFINITY;
                sh.min_r[j] = 0.0f;
            }
            if (in) p.gauge[j] = kerr_drift(kerr_lane(p, j));  // now: held inside the horizon, it need not stay finite
            // A step of length zero adds the error words: without them it moves nothing.
            R* words[5] = {&p.er, &p.eth, &p.eph, &p.epr, &p.ept};
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                float e[N];
#pragma unroll
                for (int m = 0; m < N; ++m) e[m] = m == j ? 0.0f : part(*words[i], m);
                *words[i] = join<R>(e);
            }
        }
    }
}

// The rays still under way at the step cap.
template <typename R> __device__ __forceinline__ void kerr_exhaust(KerrRays<R>& p, uint32_t cap) {
#pragma unroll
    for (int j = 0; j < Rays<R>::N; ++j)
        if (alive(p.sh, j)) {
            p.sh.end[j] = end_word(cap, RayExhausted);
            p.sh.longest[j] = 0.0f;
        }
}

// A finished ray's pixel (k_finish).
template <typename R>
__device__ __forceinline__ PixelResult kerr_finish(const KerrRays<R>& p, int j, const MarchUniforms& u,
                                                   const float4* blackbody) {
    KLane<float> l = kerr_lane(p, j);
    l.color = p.sh.color[j];
    l.transmittance = p.sh.transmittance[j];
    l.travelled = l.weighted_depth = l.depth_weight = 0.0f;
    l.samples = j == 0 ? p.sh.samples : 0u;
    l.outcome = end_outcome(p.sh.end[j]);
    l.min_r = p.sh.min_r[j];
    // A state that is no number gives no direction to look up a star in:
    // written as it is (where the FP64 list is full), its ray finds none.
    if (!finite_state(p, j)) l.outcome = RayCaptured;
    PixelResult r = kerr_pixel(l, u, blackbody);
    r.outcome = end_outcome(p.sh.end[j]);
    if (r.outcome == RayCaptured) r.drift = p.gauge[j];
    return r;
}

}  // namespace gg
