// Primary and shadow ray traversal over the device-resident hash DAG, and
// point queries.
//
// Reference: Tracer::trace_paths (tracer.cu:145-252) with
// compute_intersection_mask (:19-136) and next_child (:7-17);
// intersect_ray_node_out_of_order (:453-543) and trace_shadows (:589-697)
// with ray_box_intersection (:574-587); DAGUtils::get_value
// (dag_utils.h:138-172).  Camera rays as get_trace_params builds them
// (dag_tracer.cu:71-113).
//
// Arithmetic: this file is compiled with -fmad=false, so every float/double
// expression is rounded operation by operation in source order; FMA = 1
// places explicit fused multiply-adds where the reference's default nvcc
// build contracts a product into the following add.
#include <map>
#include <mutex>
#include <string>
#include <tuple>

#include <algorithm>
#include <cmath>

#include "hd_ctx.h"

namespace hd {

HD_D float fmax_r(float a, float b) { return a > b ? a : b; } // constexpr_max (cuda_math.h:13)
HD_D float fmin_r(float a, float b) { return a < b ? a : b; }

// The camera read where it is used, with loads the compiler may neither
// merge with other reads of it nor move: the camera is then dead during a
// walk instead of held (and spilled) across it.  Generic addressing (the
// camera may be a kernel parameter's copy or global memory), default
// caching.
HD_D double reload_f64(const double* p)
{
    double r;
    asm volatile("ld.f64 %0, [%1];" : "=d"(r) : "l"(p));
    return r;
}
HD_D hd_camera reload_camera(const hd_camera* c)
{
    hd_camera r;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        r.position[a] = reload_f64(c->position + a);
        r.ray_min[a] = reload_f64(c->ray_min + a);
        r.ray_ddx[a] = reload_f64(c->ray_ddx + a);
        r.ray_ddy[a] = reload_f64(c->ray_ddy + a);
    }
    return r;
}

// ray_min + px * ddx + py * ddy - position and its squared length, double
template <int FMA>
HD_D double camera_vec(const hd_camera& cam, double px, double py, double v[3])
{
#pragma unroll
    for (int a = 0; a < 3; a++) {
        double t;
        if (FMA) {
            t = __fma_rn(px, cam.ray_ddx[a], cam.ray_min[a]);
            t = __fma_rn(py, cam.ray_ddy[a], t);
        } else {
            t = cam.ray_min[a] + px * cam.ray_ddx[a];
            t = t + py * cam.ray_ddy[a];
        }
        v[a] = t - cam.position[a];
    }
    return FMA ? __fma_rn(v[2], v[2], __fma_rn(v[1], v[1], v[0] * v[0])) : (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2];
}

// normalize(ray_min + px * ddx + py * ddy - position), double
template <int FMA>
HD_D void camera_dir(const hd_camera& cam, double px, double py, double out[3])
{
    double v[3];
    const double dot = camera_vec<FMA>(cam, px, py, v);
    const double inv = 1.0 / sqrt(dot);
    out[0] = inv * v[0];
    out[1] = inv * v[1];
    out[2] = inv * v[2];
}

// Exact double of a 32-bit unsigned integer, built from its bits.
HD_D double u32_to_double(uint32_t u)
{
    if (u == 0)
        return 0.0;
    const uint32_t e = 31 - __clz(u);
    const uint64_t frac = (uint64_t(u) << (52 - e)) & ((1ull << 52) - 1);
    return __longlong_as_double((long long)((uint64_t(1023 + e) << 52) | frac));
}

// v rounded to the nearest float, from its bits.  False when v lies halfway
// between two floats or outside [2^-125, 2^126].
HD_D bool round_to_float(double v, float& out)
{
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    const uint32_t sign = uint32_t(b >> 32) & 0x80000000u;
    const uint64_t mag = b & 0x7FFFFFFFFFFFFFFFull;
    if (mag == 0) {
        out = __uint_as_float(sign);
        return true;
    }
    const int32_t e = int32_t(mag >> 52) - 1023 + 127;
    if (e < 2 || e > 253)
        return false;
    const uint32_t rem = uint32_t(mag) & ((1u << 29) - 1), mid = 1u << 28;
    if (rem == mid)
        return false;
    out = __uint_as_float(sign | ((uint32_t(e) << 23) + (uint32_t(mag >> 29) & 0x7FFFFFu) + (rem > mid ? 1u : 0u)));
    return true;
}

// ---- float(normalize(v)) on the FP32 pipe ------------------------------------
// The reference normalises the camera ray in double: dot = |v|^2, 1 / sqrt(dot)
// and the products, each rounded (relative error below 2^-50.8 against the
// exact v / |v| of its own double v), then rounds each component to float.
// The GB300 runs double operations at 2 per SM cycle against 128 for float,
// and every primary ray pays for this normalisation, so it is done here in
// float-float arithmetic (pairs hi + lo of floats) from the same double v:
//  * v = hi + lo: hi keeps v's 24 leading significant bits, lo the other 29
//    rounded to float (2^-47 |v|);
//  * |v|^2 = S + Slo: the squares of the hi parts summed exactly (TwoSum),
//    their fused-multiply-add remainders and the 2 hi lo terms added in float
//    (2^-45 |v|^2);
//  * y = 1 / |v| = r0 + corr: an rsqrtf seed refined by one float
//    Newton-Raphson step (2^-22.9 even for a seed 64 ulps off), then one
//    Newton-Raphson step in float-float, r0 + r0 (1 - |v|^2 r0^2) / 2, whose
//    residual is formed with fused multiply-adds (1.5 e^2 plus roundings,
//    below 2^-44.5);
//  * each component y v = P + L, P = r0 hi and its exact remainder, plus the
//    small cross terms (2^-45.5).
// The sum P + L lies within 2^-44 (measured on 10^8 vectors: 2^-44.3) of the
// exact component, and so within 2^-43.9 of the reference's double; when
// P + L is more than 2^-40 |P + L| from every float rounding midpoint both
// round to the same float.  False (about one ray in ten thousand, and for
// components outside [2^-40, 2^40) or results below 2^-63) sends the ray to
// the exact double path.

// v = hi + lo within 2^-47 |v|; false for a nonzero |v| outside [2^-40, 2^40).
HD_D bool split_f64(double v, float& hi, float& lo)
{
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    const uint32_t sign = uint32_t(b >> 32) & 0x80000000u;
    const uint64_t mag = b & 0x7FFFFFFFFFFFFFFFull;
    if (mag == 0) {
        hi = __uint_as_float(sign);
        lo = 0.0f;
        return true;
    }
    const int32_t e = int32_t(mag >> 52) - 1023;
    if (e < -40 || e >= 40)
        return false;
    hi = __uint_as_float(sign | (uint32_t(e + 127) << 23) | (uint32_t(mag >> 29) & 0x7FFFFFu));
    const float scale = __uint_as_float(sign | (uint32_t(e - 52 + 127) << 23)); // exact power of two
    lo = __fmul_rn(__uint2float_rn(uint32_t(mag) & ((1u << 29) - 1u)), scale);
    return true;
}

// s + t = a + b exactly (Knuth's TwoSum)
HD_D void two_sum(float a, float b, float& s, float& t)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    t = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// The float nearest to P + L (|L| well below |P|), when that sum lies more
// than 2^-40 |P + L| from the rounding midpoints either side of it (and the
// result's magnitude is in [2^-63, 2^64)).
HD_D bool round_pair(float P, float L, float& out)
{
    const float R = __fadd_rn(P, L);
    const float r = __fsub_rn(L, __fsub_rn(R, P)); // P + L - R exactly (Fast2Sum, |P| >= |L|)
    const uint32_t rb = __float_as_uint(R);
    const uint32_t ex = (rb >> 23) & 0xFFu;
    if (ex < 64 || ex > 190)
        return false;
    const float half_up = __uint_as_float((ex - 24) << 23);                            // ulp(R) / 2
    const float half_down = (rb & 0x7FFFFFu) ? half_up : __uint_as_float((ex - 25) << 23); // below a power of two
    const float margin = __uint_as_float((ex - 39) << 23);                              // >= 2^-40 |R|
    const float s = (rb >> 31) ? -r : r; // the remainder, positive away from zero
    if (!(__fsub_rn(half_up, s) > margin && __fadd_rn(half_down, s) > margin))
        return false;
    out = R;
    return true;
}

HD_D bool dir_from_vec(const double v[3], F3& d)
{
    float h[3], l[3];
    if (!(split_f64(v[0], h[0], l[0]) && split_f64(v[1], h[1], l[1]) && split_f64(v[2], h[2], l[2])))
        return false;
    const float p0 = __fmul_rn(h[0], h[0]), p1 = __fmul_rn(h[1], h[1]), p2 = __fmul_rn(h[2], h[2]);
    const float e = __fadd_rn(__fadd_rn(__fmaf_rn(h[0], h[0], -p0), __fmaf_rn(h[1], h[1], -p1)),
                              __fmaf_rn(h[2], h[2], -p2));
    const float c = __fadd_rn(__fadd_rn(__fmul_rn(__fadd_rn(h[0], h[0]), l[0]), __fmul_rn(__fadd_rn(h[1], h[1]), l[1])),
                              __fmul_rn(__fadd_rn(h[2], h[2]), l[2]));
    float s1, t1, S, t2;
    two_sum(p0, p1, s1, t1);
    two_sum(s1, p2, S, t2);
    const float Slo = __fadd_rn(__fadd_rn(__fadd_rn(t1, t2), e), c);
    if (!(S >= 0x1p-80f))
        return false;
    // the seed, refined once in float
    const float x0 = __fadd_rn(S, Slo);
    const float q0 = rsqrtf(x0);
    const float xq = __fmul_rn(x0, q0);
    const float r0 = __fmaf_rn(__fmul_rn(q0, __fmaf_rn(-xq, q0, 1.0f)), 0.5f, q0);
    // float-float step: hh = 1 - (S + Slo) r0^2, with S r0 = A + Al exactly
    const float A = __fmul_rn(S, r0);
    const float Al = __fmaf_rn(S, r0, -A);
    const float hh = __fsub_rn(__fmaf_rn(-A, r0, 1.0f), __fmaf_rn(Al, r0, __fmul_rn(__fmul_rn(Slo, r0), r0)));
    const float corr = __fmul_rn(__fmul_rn(r0, hh), 0.5f);
    float out[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (h[a] == 0.0f) { // a zero component keeps its sign, as inv * v does
            out[a] = h[a];
            continue;
        }
        const float P = __fmul_rn(r0, h[a]);
        const float Pl = __fmaf_rn(r0, h[a], -P);
        const float L =
            __fadd_rn(Pl, __fadd_rn(__fmul_rn(r0, l[a]), __fadd_rn(__fmul_rn(corr, h[a]), __fmul_rn(corr, l[a]))));
        if (!round_pair(P, L, out[a]))
            return false;
    }
    d = F3{out[0], out[1], out[2]};
    return true;
}

// float(normalize(...)) of camera_dir without double-precision arithmetic
// past the ray's vector (dir_from_vec).
template <int FMA>
HD_D bool camera_dir_float(const hd_camera& cam, uint32_t x, uint32_t y, F3& d)
{
    double v[3];
    camera_vec<FMA>(reload_camera(&cam), u32_to_double(x), u32_to_double(y), v);
    return dir_from_vec(v, d);
}

// ---- per-view camera tables -------------------------------------------------
// Of ray_min + px * ddx + py * ddy - position, the part that depends on the
// column alone, ray_min + px * ddx (rounded as camera_vec rounds it), is the
// same for every row, and with every operation rounded on its own (FMA = 0)
// py * ddy is the same for every column: tables of both per view leave a
// pixel two additions (or one fused multiply-add and a subtraction) per axis
// instead of four or five operations on the GB300's narrow FP64 pipe.  Per
// view: W column entries, then H row entries, 3 doubles each
// (camera_table_words).

// Entry k of a view's tables.  A second table holds the same parts relative
// to the camera as floats (x, y, z, 0), for misses_root.
template <int FMA>
HD_D void camera_table_entry(const hd_camera& cam, uint32_t W, uint32_t H, uint32_t k, double* tables)
{
    double* out = tables + 3ull * k;
    float4 f;
    float* fa = &f.x;
    f.w = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (k < W) {
            const double px = u32_to_double(k);
            out[a] = FMA ? __fma_rn(px, cam.ray_ddx[a], cam.ray_min[a]) : cam.ray_min[a] + px * cam.ray_ddx[a];
            fa[a] = float(out[a] - cam.position[a]);
        } else {
            out[a] = u32_to_double(k - W) * cam.ray_ddy[a];
            fa[a] = float(out[a]);
        }
    }
    camera_float_table(tables, W, H)[k] = f;
}

template <int FMA>
__global__ void k_camera_tables(const hd_camera* __restrict__ cams, uint32_t n_views, uint32_t W, uint32_t H,
                                double* __restrict__ tables)
{
    const uint64_t per = uint64_t(W) + H;
    HD_GRID_STRIDE(i, per * n_views)
    {
        const uint32_t v = uint32_t(i / per), k = uint32_t(i % per);
        camera_table_entry<FMA>(cams[v], W, H, k, tables + camera_table_words(W, H) * v);
    }
}

// True when the ray of pixel (x, y) surely leaves the root's cube [0, 2^D]^3
// aside, so that the walk would end at the root (tmin >= tmax there).  In
// float, along the ray's vector v instead of its direction (which scales all
// distances alike): v is the sum of two table entries, each within 2^-24 of
// its part, so a component at least 2^-8 of their magnitudes (and 2^-30 of the
// position's, whose subtraction rounds in double) is within 2^-14
// of the walk's (a smaller one decides nothing); the root's distances here
// and in the walk's own float arithmetic then differ by less than 2^-13
// (|tmid| + slab), and the interval ends are widened by twice that.
// Rays that miss the cube are common in views from outside; in whole tiles
// of them (k_trace_views votes) their set-up and root test, some 400
// instructions a warp, give way to these 50: 4 views of 1080p at 2^13, 606 ->
// 581 us of primary rays.
HD_D bool misses_root(const float4& c, const float4& r, const F3& o, float half)
{
    float tmin = 0.0f, tmax = __uint_as_float(0x7f7fffffu);
    bool sure = true;
    auto axis = [&](float cv, float rv, float ov) {
        const float v = cv + rv;
        sure &= fabsf(v) > __fmaf_rn(0x1p-30f, fabsf(ov), 0x1p-8f * (fabsf(cv) + fabsf(rv))) && fabsf(ov) < 0x1p24f &&
                fabsf(v) > 0x1p-100f && fabsf(v) < 0x1p100f;
        const float inv = __fdividef(1.0f, v);
        const float tmid = (half - ov) * inv, slab = half * fabsf(inv);
        const float m = 0x1p-12f * (fabsf(tmid) + slab);
        tmin = fmaxf(tmin, (tmid - slab) - m);
        tmax = fminf(tmax, (tmid + slab) + m);
    };
    axis(c.x, r.x, o.x);
    axis(c.y, r.y, o.y);
    axis(c.z, r.z, o.z);
    return sure && tmin > tmax;
}

// camera_vec of pixel (x, y) from its view's tables: the same doubles.
template <int FMA>
HD_D double camera_vec_tab(const hd_camera* cam, const double* __restrict__ tab, uint32_t W, uint32_t x, uint32_t y,
                           double v[3])
{
    const double* col = tab + 3ull * x;
    const double* row = tab + 3ull * (uint64_t(W) + y);
    const double py = u32_to_double(y);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double t = FMA ? __fma_rn(py, reload_f64(cam->ray_ddy + a), col[a]) : col[a] + row[a];
        v[a] = t - reload_f64(cam->position + a);
    }
    return FMA ? __fma_rn(v[2], v[2], __fma_rn(v[1], v[1], v[0] * v[0])) : (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2];
}

// The exact path of camera_dir_float, out of line: it runs for about one ray
// in ten thousand, and inlined its double-precision temporaries would
// raise the register pressure of every ray.
template <int FMA>
__device__ __noinline__ F3 camera_dir_exact(const hd_camera* cam, uint32_t x, uint32_t y)
{
    double dd[3];
    camera_dir<FMA>(*cam, double(x), double(y), dd);
    return {float(dd[0]), float(dd[1]), float(dd[2])};
}

// ---- the walk ------------------------------------------------------------------
// A node is held by lg = depth - level (its edge is 2^lg voxels) and the
// voxel coordinates (X, Y, Z) of its low corner.  The walk is bound by the
// instructions it issues (the many-view launch issued on 65 % of its cycles)
// as much as by its loads, so its steps are kept short:
//  * a node's centre as a float comes from its bits (X | half | exponent of
//    2^23, less 2^23: exact, as coordinates stay below 2^20) instead of a
//    conversion, which runs on a quarter-rate pipe;
//  * `pending` has bit lg set when the stack holds unvisited children of the
//    current path's node of that size: a finished node goes straight to the
//    nearest one instead of popping level by level, and nothing is pushed for
//    a node without further children;
//  * the next child is picked as a single-bit mask by three tests, and
//    serves as it is for the child pointer's offset and the corner;
//  * rays whose values cannot become infinite or NaN (safe_inv, safe_origin:
//    all but those along an axis plane) take minima and maxima with one
//    instruction each.
// Kernel times at 2^13 with longer steps before and these (and misses_root,
// split_walks): 16 views of 1080p, primary rays 2294 -> 1857 us (1984 -> 1751
// M warp instructions), shadow rays 953 -> 839 us; one view of 1080p, 255 ->
// 223 us and 217 -> 113 us.

// A ray whose slab distances stay finite: |1/d| and the distance of any node
// to the origin bounded, hence no product overflows and no NaN arises.
HD_D bool safe_inv(const F3& inv) { return fabsf(inv.x) < 0x1p100f && fabsf(inv.y) < 0x1p100f && fabsf(inv.z) < 0x1p100f; }
HD_D bool safe_origin(const F3& o) { return fabsf(o.x) < 0x1p24f && fabsf(o.y) < 0x1p24f && fabsf(o.z) < 0x1p24f; }

// compute_intersection_mask: children crossed by the ray of the node of edge
// 2^lg at (X, Y, Z), as an 8-bit mask.  SAFE: the ray is a safe one; its
// minima and maxima then do not depend on how NaNs compare (the reference's
// a > b ? a : b), nor does any comparison on the sign of a zero.
template <int FMA, bool SAFE>
HD_D uint32_t crossed_children(uint32_t lg, uint32_t X, uint32_t Y, uint32_t Z, bool is_root, const F3& o, const F3& d,
                               const F3& inv)
{
    const uint32_t bits = 0x4B000000u | (1u << (lg - 1)); // 2^23 + half
    const float radius = __uint_as_float((126u + lg) << 23);
    const F3 crr = {(__uint_as_float(X | bits) - 0x1p23f) - o.x, (__uint_as_float(Y | bits) - 0x1p23f) - o.y,
                    (__uint_as_float(Z | bits) - 0x1p23f) - o.z};
    const F3 tmid = {crr.x * inv.x, crr.y * inv.y, crr.z * inv.z};
    const F3 slab = {radius * fabsf(inv.x), radius * fabsf(inv.y), radius * fabsf(inv.z)};
    F3 pmin, pmax;
    if (FMA) {
        pmin = {__fmaf_rn(crr.x, inv.x, -slab.x), __fmaf_rn(crr.y, inv.y, -slab.y), __fmaf_rn(crr.z, inv.z, -slab.z)};
        pmax = {__fmaf_rn(crr.x, inv.x, slab.x), __fmaf_rn(crr.y, inv.y, slab.y), __fmaf_rn(crr.z, inv.z, slab.z)};
    } else {
        pmin = {tmid.x - slab.x, tmid.y - slab.y, tmid.z - slab.z};
        pmax = {tmid.x + slab.x, tmid.y + slab.y, tmid.z + slab.z};
    }
    const float tmin = SAFE ? fmaxf(fmaxf(pmin.x, pmin.y), fmaxf(pmin.z, 0.0f))
                            : fmax_r(fmax_r(pmin.x, fmax_r(pmin.y, pmin.z)), 0.0f);
    const float tmax = SAFE ? fminf(pmax.x, fminf(pmax.y, pmax.z)) : fmin_r(pmax.x, fmin_r(pmax.y, pmax.z));
    if (is_root && tmin >= tmax)
        return 0;
    uint32_t result;
    {
        const float s = 0.5f * (tmin + tmax);
        const uint32_t first = ((s * d.x) >= crr.x ? 4u : 0u) + ((s * d.y) >= crr.y ? 2u : 0u) +
                               ((s * d.z) >= crr.z ? 1u : 0u);
        result = 1u << first;
    }
    const float eps = 1e-4f;
    const F3 lo = {crr.x - eps, crr.y - eps, crr.z - eps}, hi = {crr.x + eps, crr.y + eps, crr.z + eps};
    // children on either side of a plane within eps of the crossing point:
    // with tests on both sides, both halves (0xFF), one or (unsafe rays) none
    auto side = [](float v, float l, float h, uint32_t up, uint32_t down) {
        return (v >= l ? up : 0u) | (v <= h ? down : 0u);
    };
    if (tmin <= tmid.x && tmid.x <= tmax)
        result |= side(tmid.x * d.y, lo.y, hi.y, 0xCC, 0x33) & side(tmid.x * d.z, lo.z, hi.z, 0xAA, 0x55);
    if (tmin <= tmid.y && tmid.y <= tmax)
        result |= side(tmid.y * d.x, lo.x, hi.x, 0xF0, 0x0F) & side(tmid.y * d.z, lo.z, hi.z, 0xAA, 0x55);
    if (tmin <= tmid.z && tmid.z <= tmax)
        result |= side(tmid.z * d.x, lo.x, hi.x, 0xF0, 0x0F) & side(tmid.z * d.y, lo.y, hi.y, 0xCC, 0x33);
    return result;
}

HD_D uint32_t first_child_mask(uint32_t low, uint32_t high) // Leaf::get_first_child_mask (base_dag.h:16-52)
{
    const uint32_t a = __vcmpne4(low, 0u) & 0x08040201u;
    const uint32_t b = __vcmpne4(high, 0u) & 0x08040201u;
    return ((a * 0x01010101u) >> 24) | (((b * 0x01010101u) >> 24) << 4);
}

// The child order of a ray (rayChildOrder and next_child, tracer.cu:7-17,
// :161-164): child ^ octant, 0..7, i.e. per axis the half the ray enters
// first.  Each member: the children in that half.
struct ChildOrder {
    uint32_t x, y, z;
};
HD_HD ChildOrder child_order(const F3& d)
{
    return {d.x < 0.f ? 0xF0u : 0x0Fu, d.y < 0.f ? 0xCCu : 0x33u, d.z < 0.f ? 0xAAu : 0x55u};
}
// The first child of a nonempty mask in that order, as a single-bit mask.
HD_D uint32_t next_child(const ChildOrder& c, uint32_t m)
{
    uint32_t h = m & c.x;
    m = h ? h : m;
    h = m & c.y;
    m = h ? h : m;
    h = m & c.z;
    return h ? h : m;
}

// The walk's stack: for a node of edge 2^lg, lg >= 2 (row lg - 2; the children
// of a smaller one are voxels, and the first ends the walk), its physical pool
// offset and its child mask | visit mask << 8.
struct LocalStack {
    struct {
        uint32_t index, masks;
    } e[HD_MAX_DEPTH];
    HD_D void set(uint32_t row, uint32_t index, uint32_t masks) { e[row] = {index, masks}; }
    HD_D uint32_t index(uint32_t row) const { return e[row].index; }
    HD_D uint32_t masks(uint32_t row) const { return e[row].masks; }
};
// The same stack in the kernel's dynamic shared memory: row r of thread k
// at [r * blockDim.x + k], node indices and 16-bit masks in two arrays (6
// bytes a row).  Addresses come from the thread index and the array
// itself, so a walk holds no pointer registers for its stack.
extern __shared__ uint32_t hd_walk_stack[];
struct SharedStack {
    uint32_t msk_words; // start of the mask array: blockDim.x * (depth - 1) words
    HD_D void set(uint32_t row, uint32_t index, uint32_t masks) const
    {
        const uint32_t k = row * blockDim.x + threadIdx.x;
        hd_walk_stack[k] = index;
        reinterpret_cast<uint16_t*>(hd_walk_stack + msk_words)[k] = uint16_t(masks);
    }
    HD_D uint32_t index(uint32_t row) const { return index_of(row, threadIdx.x); }
    HD_D uint32_t masks(uint32_t row) const { return masks_of(row, threadIdx.x); }
    // another thread's entry
    HD_D uint32_t index_of(uint32_t row, uint32_t thread) const { return hd_walk_stack[row * blockDim.x + thread]; }
    HD_D uint32_t masks_of(uint32_t row, uint32_t thread) const
    {
        return reinterpret_cast<const uint16_t*>(hd_walk_stack + msk_words)[row * blockDim.x + thread];
    }
};
// Shared bytes of a SharedStack for `threads` threads and depth D.
HD_HD uint32_t shared_stack_bytes(uint32_t threads, uint32_t D) { return threads * (D - 1) * 6; }
HD_D SharedStack shared_stack(uint32_t D) { return SharedStack{blockDim.x * (D - 1)}; }

// The stack walk shared by the primary ray (nearest hit, children in the
// ray's octant order) and the shadow ray (any hit), as a state machine:
// start() enters the root, each step() goes to one child and returns 0 (going
// on), 1 (reached a voxel, at X, Y, Z) or 2 (left the root).  The reference's
// shadow walk takes children highest first; whether a ray hits anything does
// not depend on the order (the walk visits every crossed child until a voxel
// is reached), so shadow walks take the front-to-back order too and meet the
// nearest occluders first.
template <int FMA, bool SAFE>
struct Walker {
    uint32_t lg, X, Y, Z, index, child_mask, visit, pending, leaf_lo, leaf_hi;

    // node, its children's mask: the root's
    HD_D void start(const Table& t, uint32_t node, uint32_t children, const F3& o, const F3& d, const F3& inv)
    {
        lg = t.g.depth;
        X = Y = Z = 0;
        pending = 0;
        leaf_lo = leaf_hi = 0;
        index = node;
        child_mask = children;
        visit = child_mask & crossed_children<FMA, SAFE>(lg, 0, 0, 0, true, o, d, inv);
    }

    template <typename Stack>
    HD_D uint32_t step(const Table& t, const F3& o, const F3& d, const F3& inv, const ChildOrder& order, Stack& stack,
                       uint32_t& descents, uint32_t& leaves)
    {
        if (!visit) {
            if (!pending)
                return 2;
            lg = __ffs(pending) - 1;
            pending &= pending - 1;
            index = stack.index(lg - 2);
            const uint32_t m = stack.masks(lg - 2);
            child_mask = m & 0xffu;
            visit = m >> 8;
            const uint32_t keep = ~0u << lg;
            X &= keep;
            Y &= keep;
            Z &= keep;
        }
        const uint32_t c = next_child(order, visit);
        const uint32_t half = 1u << (lg - 1);
        X |= (c & 0xF0u) ? half : 0u;
        Y |= (c & 0xCCu) ? half : 0u;
        Z |= (c & 0xAAu) ? half : 0u;
        if (lg == 1)
            return 1;
        visit ^= c;
        if (visit) {
            stack.set(lg - 2, index, child_mask | (visit << 8));
            pending |= 1u << lg;
        }
        lg--;
        // child c's pointer follows those of the children before it
        if (lg > 2) {
            index = t.phys(t.pool[index + popc32(child_mask & (c - 1)) + 1]);
            child_mask = t.pool[index] & 0xffu;
            descents++;
        } else if (lg == 2) {
            const uint32_t addr = t.phys(t.pool[index + popc32(child_mask & (c - 1)) + 1]);
            const uint2 lf = *(reinterpret_cast<const uint2*>(t.pool + addr));
            leaf_lo = lf.x;
            leaf_hi = lf.y;
            child_mask = first_child_mask(leaf_lo, leaf_hi);
            leaves++;
        } else {
            child_mask = ((c & 0xF0u) ? leaf_hi : leaf_lo) >> (((__ffs(c) - 1) & 3) * 8) & 0xffu;
        }
        visit = child_mask & crossed_children<FMA, SAFE>(lg, X, Y, Z, false, o, d, inv);
        return 0;
    }
};

// The walks differ in length by orders of magnitude, and at the end of a
// launch a warp would wait for its longest one.  Then its idle lanes take part
// in the walks that go on: lane by lane, a walk with pending children gives
// away the highest node of its stack (the unvisited children nearest the
// root, which come last in its order), and the taker walks them as a walk of
// its own.  Warp-wide; a taker's ray state is up to the caller: the lane each
// lane took from, its own when it took nothing.
template <int FMA, bool SAFE>
HD_D uint32_t split_walks(Walker<FMA, SAFE>& w, const SharedStack& stack, bool& active)
{
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    __syncwarp(); // the givers' stack entries and mask bytes are written (the votes below order no memory)
    const uint32_t idle = __ballot_sync(0xffffffffu, !active);
    const uint32_t givers = __ballot_sync(0xffffffffu, active && w.pending != 0);
    const uint32_t n = min(__popc(idle), __popc(givers));
    const bool takes = !active && uint32_t(__popc(idle & lt)) < n;
    const bool gives = ((givers >> lane) & 1u) && uint32_t(__popc(givers & lt)) < n;
    // the giver of this taker: the same rank among the givers
    const uint32_t src = takes ? __fns(givers, 0, __popc(idle & lt) + 1) : lane;
    const uint32_t top = w.pending ? 31u - __clz(w.pending) : 0u;
    const uint32_t lg = __shfl_sync(0xffffffffu, top, src);
    const uint32_t X = __shfl_sync(0xffffffffu, w.X, src), Y = __shfl_sync(0xffffffffu, w.Y, src),
                   Z = __shfl_sync(0xffffffffu, w.Z, src);
    const uint32_t lo = __shfl_sync(0xffffffffu, w.leaf_lo, src), hi = __shfl_sync(0xffffffffu, w.leaf_hi, src);
    if (takes) {
        const uint32_t thread = (threadIdx.x & ~31u) + src;
        w.lg = lg;
        w.index = stack.index_of(lg - 2, thread);
        const uint32_t m = stack.masks_of(lg - 2, thread);
        w.child_mask = m & 0xffu;
        w.visit = m >> 8;
        const uint32_t keep = ~0u << lg;
        w.X = X & keep;
        w.Y = Y & keep;
        w.Z = Z & keep;
        w.leaf_lo = lo;
        w.leaf_hi = hi;
        w.pending = 0;
        active = true;
    }
    if (gives)
        w.pending &= ~(1u << top);
    __syncwarp(); // the giver's entry was read before it writes its stack again
    return src;
}

template <int FMA, bool SAFE, typename Stack>
HD_D bool walk_steps(const Table& t, uint32_t root, const F3& o, const F3& d, const F3& inv, uint32_t* hit,
                     uint32_t& descents, uint32_t& leaves, Stack& stack)
{
    const ChildOrder order = child_order(d);
    Walker<FMA, SAFE> w;
    const uint32_t node = t.phys(root);
    w.start(t, node, t.pool[node] & 0xffu, o, d, inv);
    uint32_t r;
    do
        r = w.step(t, o, d, inv, order, stack, descents, leaves);
    while (!r);
    const bool h = r == 1;
    hit[0] = h ? w.X : 0;
    hit[1] = h ? w.Y : 0;
    hit[2] = h ? w.Z : 0;
    return h;
}

// The walk of a ray that is not a safe one (a direction along an axis plane,
// a camera far outside), out of line.
struct WalkResult {
    uint32_t x, y, z, hit, descents, leaves;
};
template <int FMA>
__device__ __noinline__ WalkResult walk_unsafe(const Table& t, uint32_t root, F3 o, F3 d, F3 inv)
{
    LocalStack stack;
    uint32_t hit[3];
    WalkResult r{};
    r.hit = walk_steps<FMA, false>(t, root, o, d, inv, hit, r.descents, r.leaves, stack);
    r.x = hit[0];
    r.y = hit[1];
    r.z = hit[2];
    return r;
}

template <int FMA, typename Stack = LocalStack>
HD_D bool walk(const Table& t, uint32_t root, const F3& o, const F3& d, const F3& inv, uint32_t* hit,
               uint32_t& descents, uint32_t& leaves, Stack stack = Stack{})
{
    if (safe_inv(inv) && safe_origin(o))
        return walk_steps<FMA, true>(t, root, o, d, inv, hit, descents, leaves, stack);
    const WalkResult r = walk_unsafe<FMA>(t, root, o, d, inv);
    hit[0] = r.x;
    hit[1] = r.y;
    hit[2] = r.z;
    descents += r.descents;
    leaves += r.leaves;
    return r.hit != 0;
}

// The reference takes float(1.0 / double(x)) (tracer.cu:160): the double
// quotient rounded again to float.  Rounding a quotient first to a p'-bit
// and then to a p-bit significand equals rounding it once to p bits when
// p' >= 2p + 2 (S. Figueroa, "When is double rounding innocuous?", SIGNUM
// Newsletter 30(3), 1995); double (53) and float (24) qualify.  So the
// correctly rounded float reciprocal (__frcp_rn) gives the same bits with no
// double-precision work, which the GB300's small FP64 pipe would otherwise
// spend on every ray.
HD_D F3 inverse_dir(const F3& d) { return {__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z)}; }

// 8x8 pixel tiles per 64-thread block; a warp covers 8x4 pixels.
// Traversal work counters (COUNT instances only): rays, interior descents,
// leaf fetches.
HD_D void add_counts(unsigned long long* counters, uint32_t rays, uint32_t descents, uint32_t leaves)
{
    atomicAdd(counters + 0, rays);
    atomicAdd(counters + 1, descents);
    atomicAdd(counters + 2, leaves);
}

// tab (TAB): the view's camera tables (k_camera_tables)
template <int FMA, bool COUNT, typename Stack = LocalStack, bool TAB = false>
HD_D uint4 primary_ray(const Table& t, uint32_t root, const hd_camera& cam, uint32_t W, uint32_t H, uint32_t x,
                       uint32_t y, uint4* __restrict__ out, unsigned long long* counters, Stack stack = Stack{},
                       const double* __restrict__ tab = nullptr)
{
    F3 d;
    bool fast;
    if (TAB) {
        double v[3];
        camera_vec_tab<FMA>(&cam, tab, W, x, y, v);
        fast = dir_from_vec(v, d);
    } else {
        fast = camera_dir_float<FMA>(cam, x, y, d);
    }
    if (!fast)
        d = camera_dir_exact<FMA>(&cam, x, y);
    const F3 inv = inverse_dir(d);
    F3 o;
    if (!(round_to_float(cam.position[0], o.x) && round_to_float(cam.position[1], o.y) &&
          round_to_float(cam.position[2], o.z)))
        o = {float(cam.position[0]), float(cam.position[1]), float(cam.position[2])};
    uint32_t hit[3], descents = 0, leaves = 0;
    walk<FMA, Stack>(t, root, o, d, inv, hit, descents, leaves, stack);
    const uint4 path = make_uint4(hit[0], hit[1], hit[2], 0);
    out[uint64_t(H - 1 - y) * W + x] = path;
    if (COUNT)
        add_counts(counters, 1, descents, leaves);
    return path;
}

template <int FMA, bool COUNT>
__global__ void __launch_bounds__(64) k_trace_primary(Table t, const uint32_t* __restrict__ d_root, hd_camera cam,
                                                      uint32_t W, uint32_t H, uint4* __restrict__ out,
                                                      unsigned long long* counters)
{
    const uint32_t x = blockIdx.x * 8 + (threadIdx.x & 7);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 3);
    if (x >= W || y >= H)
        return;
    primary_ray<FMA, COUNT>(t, *d_root, cam, W, H, x, y, out, counters);
}

// A shadow ray of the compacted list: the output pixel (view * W * H +
// pixel) and its origin.
struct ShadowRay {
    uint32_t idx;
    float ox, oy, oz;
};

// sun_direction(): the light normalised in float (tracer.cu:546-549)
template <int FMA>
HD_D F3 light_dir(F3 light)
{
    const float dot = FMA ? __fmaf_rn(light.z, light.z, __fmaf_rn(light.y, light.y, light.x * light.x))
                          : (light.x * light.x + light.y * light.y) + light.z * light.z;
    const float il = 1.0f / sqrtf(dot);
    return F3{il * light.x, il * light.y, il * light.z};
}

// Origin of the shadow ray of output pixel (x, row r) whose primary ray hit
// voxel p (tracer.cu:589-697 reduced to the hit test): the exact hit point on
// the hit voxel's box (ray_box_intersection, :574-587, in double) plus
// bias * light.
// Out of line: its double-precision temporaries stay out of the register
// allocation of the walk that precedes it.
template <int FMA>
__device__ __noinline__ F3 shadow_origin(const hd_camera& cam, uint32_t H, uint32_t x, uint32_t r, uint4 p, F3 dir,
                                      float bias)
{
    double cd[3];
    camera_dir<FMA>(cam, double(x), double(H - 1 - r), cd);
    const double bmin[3] = {double(float(p.x)), double(float(p.y)), double(float(p.z))};
    double real_min[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        // min(t0, t1) with t0 = (bmin - pos) / cd, t1 = (bmin + 1 - pos) / cd:
        // the numerators are ordered (bmin + 1 is exact, rounding is
        // monotonic), so for cd > 0 the minimum is t0 and for cd < 0 it is t1
        // (equal quotients give the same value either way); only cd = 0 needs
        // both.
        const double n0 = bmin[a] - cam.position[a];
        const double n1 = (bmin[a] + 1.0) - cam.position[a];
        if (cd[a] > 0.0) {
            real_min[a] = n0 / cd[a];
        } else if (cd[a] < 0.0) {
            real_min[a] = n1 / cd[a];
        } else {
            const double t0 = n0 / cd[a], t1 = n1 / cd[a];
            real_min[a] = t0 < t1 ? t0 : t1;
        }
    }
    const double maxmin = fmax(fmax(real_min[0], real_min[1]), real_min[2]);
    F3 start, o;
    if (FMA) {
        start = {float(__fma_rn(cd[0], maxmin, cam.position[0])), float(__fma_rn(cd[1], maxmin, cam.position[1])),
                 float(__fma_rn(cd[2], maxmin, cam.position[2]))};
        o = {__fmaf_rn(bias, dir.x, start.x), __fmaf_rn(bias, dir.y, start.y), __fmaf_rn(bias, dir.z, start.z)};
    } else {
        start = {float(cam.position[0] + cd[0] * maxmin), float(cam.position[1] + cd[1] * maxmin),
                 float(cam.position[2] + cd[2] * maxmin)};
        o = {start.x + bias * dir.x, start.y + bias * dir.y, start.z + bias * dir.z};
    }
    return o;
}

// Where view v's paths go when a launch splits its output (out_copied set):
// the views view_copied names (the last 8 - kCopiedFrom of every 8) to
// out_copied, packed in view order, the others to out.  The host-buffer
// entry point writes the first kind straight into host memory during the
// primary launch and copies the second during the shadow launch, so that
// both parts of the step move paths over the host link.
HD_D uint4* view_paths(uint4* out, uint4* out_copied, uint32_t v, uint64_t frame)
{
    if (out_copied && (v & 7) >= kCopiedFrom)
        return out_copied + (uint64_t(v >> 3) * (8 - kCopiedFrom) + (v & 7) - kCopiedFrom) * frame;
    return out + uint64_t(v) * frame;
}

// Several views in one launch, as persistent warps: each warp takes 8x4
// pixel tiles from a counter (view-major, then tile rows), so warps whose
// rays end early take more tiles and every resident warp stays busy to the
// end of the launch; the next tile is fetched before the current one is
// traced.  View v writes its paths at out + v * W * H (the single-view
// layout), or, with out_copied, the views view_paths sets aside there.  The
// shadow pass's set-up is fused in: a pixel whose primary ray
// hit appends its shadow ray (origin on the hit voxel, as shadow_origin) to
// the list, warp by warp; a miss gets mask 2 at once.  12 blocks an SM: with 16
// (32 registers) the walk spilled, 22 M local loads in 16 views.  The times do
// not tell 11 to 16 blocks apart: 8 views to the host took 2366 us with 16 and
// 2335 with 12, and boxes differ by 10 %.
template <int FMA>
__global__ void __launch_bounds__(128, 12)
    k_trace_views(__grid_constant__ const Table t, const uint32_t* __restrict__ d_root,
                  const hd_camera* __restrict__ cams, uint32_t W, uint32_t H, uint32_t n_views,
                  uint4* __restrict__ out, F3 light, float bias, uint8_t* __restrict__ mask,
                  ShadowRay* __restrict__ list, uint32_t* __restrict__ head, const double* __restrict__ tables,
                  uint4* __restrict__ out_copied)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t tx = (W + 7) / 8, ty = (H + 3) / 4;
    const uint32_t per_view = tx * ty, n_tiles = per_view * n_views;
    const SharedStack stack = shared_stack(t.g.depth);
    const uint32_t root = *d_root;
    const float half = __uint_as_float((126u + t.g.depth) << 23);
    uint32_t* next_tile = head + 1;
    uint32_t tile = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(next_tile, 1u) : 0u, 0);
    while (tile < n_tiles) {
        const uint32_t next = lane == 0 ? atomicAdd(next_tile, 1u) : 0u;
        const uint32_t v = tile / per_view, k = tile - v * per_view;
        const uint32_t x = (k % tx) * 8 + (lane & 7), y = (k / tx) * 4 + (lane >> 3);
        const bool in = x < W && y < H;
        uint4* const view_out = view_paths(out, out_copied, v, uint64_t(W) * H);
        const double* const tab = tables + camera_table_words(W, H) * v;
        bool may_hit = false;
        if (in) {
            const float4* ft = camera_float_table(tab, W, H);
            const double* pos = cams[v].position;
            may_hit = !misses_root(ft[x], ft[W + y], F3{float(pos[0]), float(pos[1]), float(pos[2])}, half);
        }
        bool hit = false;
        uint4 p = make_uint4(0, 0, 0, 0);
        if (__any_sync(0xffffffffu, may_hit)) {
            if (in) {
                p = primary_ray<FMA, false, SharedStack, true>(t, root, cams[v], W, H, x, y, view_out, nullptr, stack,
                                                               tab);
                hit = (p.x | p.y | p.z) != 0;
            }
        } else if (in) {
            view_out[uint64_t(H - 1 - y) * W + x] = p;
        }
        const uint64_t i = uint64_t(v) * W * H + uint64_t(H - 1 - y) * W + x;
        if (in && !hit)
            mask[i] = 2;
        const uint32_t b = __ballot_sync(0xffffffffu, hit);
        if (b) {
            const uint32_t base =
                __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(head, uint32_t(__popc(b))) : 0u, 0);
            if (hit) {
                const F3 o = shadow_origin<FMA>(cams[v], H, x, H - 1 - y, p, light_dir<FMA>(light), bias);
                list[base + __popc(b & ((1u << lane) - 1u))] = ShadowRay{uint32_t(i), o.x, o.y, o.z};
            }
        }
        tile = __shfl_sync(0xffffffffu, next, 0);
    }
}

// Shadow rays start only at hit pixels (a path of (0, 0, 0) is a miss,
// tracer.cu:644-648).  The hit pixels of each 8x8 tile are appended to the
// list, tile by tile, with their ray origins, so that
// the traversal kernel runs full warps of rays from neighbouring pixels and
// carries none of the double-precision set-up; misses get mask 2 here.  Rows
// are output rows (the layout of the paths image).  1080p at 2^13: 63 us, 42 of
// them the origins (a warp's double operation takes 16 cycles); blocks of 128 to
// 512 threads and persistent warps that read ahead took 60 to 73.
template <int FMA>
__global__ void __launch_bounds__(64) k_shadow_list(__grid_constant__ const hd_camera cam, uint32_t W, uint32_t H,
                                                    const uint4* __restrict__ paths, F3 light, float bias,
                                                    uint8_t* __restrict__ mask, ShadowRay* __restrict__ list,
                                                    uint32_t* __restrict__ count)
{
    __shared__ uint32_t warp_base[2];
    const uint32_t x = blockIdx.x * 8 + (threadIdx.x & 7);
    const uint32_t r = blockIdx.y * 8 + (threadIdx.x >> 3);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool in = x < W && r < H;
    const uint64_t i = uint64_t(r) * W + x;
    bool hit = false;
    uint4 p = make_uint4(0, 0, 0, 0);
    if (in) {
        p = paths[i];
        hit = (p.x | p.y | p.z) != 0;
        if (!hit)
            mask[i] = 2;
    }
    const uint32_t b = __ballot_sync(0xffffffffu, hit);
    if (lane == 0)
        warp_base[warp] = __popc(b);
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t n0 = warp_base[0], n1 = warp_base[1];
        const uint32_t base = (n0 + n1) ? atomicAdd(count, n0 + n1) : 0u;
        warp_base[0] = base;
        warp_base[1] = base + n0;
    }
    __syncthreads();
    if (hit) {
        const F3 o = shadow_origin<FMA>(cam, H, x, r, p, light_dir<FMA>(light), bias);
        list[warp_base[warp] + __popc(b & ((1u << lane) - 1u))] = ShadowRay{uint32_t(i), o.x, o.y, o.z};
    }
}

// The any-hit walk of every ray of the list toward the light
// (intersect_ray_node_out_of_order, tracer.cu:453-543) as persistent warps
// whose lanes refill independently: a lane whose ray has ended takes the next
// ray of the list as soon as kShadowRefill lanes of its warp are idle, so the
// warp does not wait for its longest walk (the walks differ by orders of
// magnitude).  When the list has run out, idle lanes walk parts of the rays
// that go on (split_walks); the mask byte starts at 0, and any part that hits
// sets it.  Each ray's result depends on that ray only.  Without the splitting
// a single frame ended with its longest rays, 11 lanes of a warp at work
// on average: 1080p at 2^13, 217 us against 113; 320x180 at 2^10, 59 against 43.
// Rays are taken from the list 32 at a time, one share ahead: an atomic per
// refill had its latency in every refill.  Sizes measured: refill at 4 idle
// lanes and 8 steps between refills are up to 1 % slower.
constexpr uint32_t kShadowRefill = 8;  // idle lanes that trigger a fetch
constexpr uint32_t kShadowSteps = 4;   // walk steps between fetches
constexpr uint32_t kShadowTake = 32;   // rays a warp takes from the list at a time

// The one direction of a pass's shadow rays, made on the host with the
// device's operations (light_dir, inverse_dir): kernel parameters, so that a
// walk holds no registers for it.
struct ShadowDir {
    F3 dir, inv;
    ChildOrder order;
};

static ShadowDir shadow_dir(const float light[3], int fma)
{
    // each operation rounded on its own (volatile: no contraction)
    volatile float xx = light[0] * light[0], yy = light[1] * light[1], zz = light[2] * light[2];
    volatile float xy = xx + yy;
    volatile float dot = xy + zz;
    if (fma)
        dot = std::fma(light[2], light[2], std::fma(light[1], light[1], float(xx)));
    volatile float root = std::sqrt(float(dot));
    volatile float il = 1.0f / root;
    volatile float x = il * light[0], y = il * light[1], z = il * light[2];
    volatile float ix = 1.0f / x, iy = 1.0f / y, iz = 1.0f / z;
    const F3 d{x, y, z};
    return {d, F3{ix, iy, iz}, child_order(d)};
}

template <int FMA, bool COUNT>
__global__ void __launch_bounds__(128) k_trace_shadow(__grid_constant__ const Table t,
                                                      const uint32_t* __restrict__ d_root,
                                                      __grid_constant__ const ShadowDir sd,
                                                      uint8_t* __restrict__ mask, const ShadowRay* __restrict__ list,
                                                      uint32_t* __restrict__ head, unsigned long long* counters)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = head[0];
    const uint32_t root_node = t.phys(*d_root), root_mask = t.pool[root_node] & 0xffu;
    SharedStack stack = shared_stack(t.g.depth);
    Walker<FMA, false> w;
    w.pending = 0;
    F3 o;
    uint32_t idx = 0, descents = 0, leaves = 0;
    bool active = false;
    // the warp's share of the list: rays [at, end), the next share on its way
    uint32_t at = 0, end = 0;
    uint32_t ahead = lane == 0 ? atomicAdd(head + 2, kShadowTake) : 0u;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !active);
        if (__popc(idle) >= kShadowRefill) {
            if (at == end) {
                at = __shfl_sync(0xffffffffu, ahead, 0);
                at = at < n ? at : n;
                end = n - at < kShadowTake ? n : at + kShadowTake;
                if (at < end && lane == 0)
                    ahead = atomicAdd(head + 2, kShadowTake);
            }
            if (!active) {
                const uint32_t j = at + __popc(idle & ((1u << lane) - 1u));
                if (j < end) {
                    const ShadowRay ray = list[j];
                    idx = ray.idx;
                    o = F3{ray.ox, ray.oy, ray.oz};
                    mask[idx] = 0;
                    w.start(t, root_node, root_mask, o, sd.dir, sd.inv);
                    active = true;
                }
            }
            at = min(end, at + uint32_t(__popc(idle)));
        }
        if (at == end && end == n && idle) {
            if (!__any_sync(0xffffffffu, active))
                break;
            if (!COUNT) {
                // no ray left: the idle lanes help (a ray's parts all write
                // its mask byte, which starts at 0, when they hit)
                const uint32_t src = split_walks(w, stack, active);
                o = F3{__shfl_sync(0xffffffffu, o.x, src), __shfl_sync(0xffffffffu, o.y, src),
                       __shfl_sync(0xffffffffu, o.z, src)};
                idx = __shfl_sync(0xffffffffu, idx, src);
            }
        }
        bool hit = false;
        for (uint32_t s = 0; s < kShadowSteps && active; s++) {
            const uint32_t r = w.step(t, o, sd.dir, sd.inv, sd.order, stack, descents, leaves);
            if (r) {
                hit = r == 1;
                active = false;
                if (COUNT) {
                    add_counts(counters, 1, descents, leaves);
                    descents = leaves = 0;
                }
            }
        }
        if (hit)
            mask[idx] = 1;
        if (!COUNT && at == end && end == n) {
            // the other parts of a ray that hit are over
            for (uint32_t m = __ballot_sync(0xffffffffu, hit); m; m &= m - 1)
                if (__shfl_sync(0xffffffffu, idx, __ffs(m) - 1) == idx)
                    active = false;
        }
    }
}

// Blocks of a persistent launch of `kernel` with `threads` threads: as many
// as stay resident on every SM with smem_bytes of dynamic shared memory
// (queried once per kernel and size).
static uint32_t resident_blocks(const void* kernel, int threads, uint32_t smem_bytes)
{
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, uint32_t>, uint32_t> known;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(kernel, threads, smem_bytes);
    auto it = known.find(key);
    if (it != known.end())
        return it->second;
    int dev = 0, sms = 0, per_sm = 0;
    HD_CUDA(cudaGetDevice(&dev));
    HD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    HD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem_bytes));
    const uint32_t n = uint32_t(std::max(1, sms * std::max(1, per_sm)));
    known[key] = n;
    return n;
}

void trace_primary(hd_ctx* c, const hd_camera& cam, uint32_t w, uint32_t h, uint32_t* d_paths,
                   unsigned long long* d_counters, cudaStream_t stream, const uint32_t* d_root)
{
    cudaStream_t st = stream ? stream : c->stream;
    const uint32_t* rt = d_root ? d_root : c->d_root;
    if ((h + 7) / 8 > kMaxGridRows)
        throw StatusError{HD_ERR_INVALID, "image height " + std::to_string(h) + " exceeds " +
                                              std::to_string(8 * kMaxGridRows) + " rows"};
    uint4* out = reinterpret_cast<uint4*>(d_paths);
    dim3 grid((w + 7) / 8, (h + 7) / 8);
    if (d_counters) {
        if (c->fp_mode)
            k_trace_primary<1, true><<<grid, 64, 0, st>>>(c->t, rt, cam, w, h, out, d_counters);
        else
            k_trace_primary<0, true><<<grid, 64, 0, st>>>(c->t, rt, cam, w, h, out, d_counters);
    } else {
        if (c->fp_mode)
            k_trace_primary<1, false><<<grid, 64, 0, st>>>(c->t, rt, cam, w, h, out, nullptr);
        else
            k_trace_primary<0, false><<<grid, 64, 0, st>>>(c->t, rt, cam, w, h, out, nullptr);
    }
    HD_LAUNCH_CHECK();
}

// The any-hit walks of a shadow-ray list (head: ray count, two work
// counters) over px pixels.
static void shadow_walks(hd_ctx* c, uint64_t px, const float light[3], uint8_t* d_mask,
                         unsigned long long* d_counters, cudaStream_t st, const uint32_t* rt, const ShadowRay* list,
                         uint32_t* head)
{
    const ShadowDir sd = shadow_dir(light, int(c->fp_mode));
    auto launch = [&](auto kernel) {
        const uint32_t smem = shared_stack_bytes(128, c->t.g.depth);
        const uint32_t blocks = uint32_t(
            std::min<uint64_t>((px + 127) / 128, resident_blocks(reinterpret_cast<const void*>(kernel), 128, smem)));
        kernel<<<blocks, 128, smem, st>>>(c->t, rt, sd, d_mask, list, head, d_counters);
    };
    if (d_counters)
        c->fp_mode ? launch(k_trace_shadow<1, true>) : launch(k_trace_shadow<0, true>);
    else
        c->fp_mode ? launch(k_trace_shadow<1, false>) : launch(k_trace_shadow<0, false>);
    HD_LAUNCH_CHECK();
}

// Shadow pass of one frame from its paths: the hit list with origins, then
// the any-hit walks.
static void shadow_pass(hd_ctx* c, const hd_camera& cam, uint32_t w, uint32_t h, const uint32_t* d_paths,
                        const float light[3], float bias, uint8_t* d_mask, unsigned long long* d_counters,
                        cudaStream_t st, const uint32_t* rt, uint32_t* d_list)
{
    const uint64_t px = uint64_t(w) * h;
    if ((h + 7) / 8 > kMaxGridRows)
        throw StatusError{HD_ERR_INVALID, "image height " + std::to_string(h) + " exceeds " +
                                              std::to_string(8 * kMaxGridRows) + " rows"};
    uint32_t* buf = d_list ? d_list : c->scratch.get<uint32_t>("shadow_list", shadow_list_words(px));
    ShadowRay* list = reinterpret_cast<ShadowRay*>(buf);
    uint32_t* head = buf + 4 * px;
    HD_CUDA(cudaMemsetAsync(head, 0, 16, st));
    dim3 tiles((w + 7) / 8, (h + 7) / 8);
    const uint4* p = reinterpret_cast<const uint4*>(d_paths);
    const F3 l = {light[0], light[1], light[2]};
    if (c->fp_mode)
        k_shadow_list<1><<<tiles, 64, 0, st>>>(cam, w, h, p, l, bias, d_mask, list, head);
    else
        k_shadow_list<0><<<tiles, 64, 0, st>>>(cam, w, h, p, l, bias, d_mask, list, head);
    HD_LAUNCH_CHECK();
    shadow_walks(c, px, light, d_mask, d_counters, st, rt, list, head);
}

void trace_shadow(hd_ctx* c, const hd_camera& cam, uint32_t w, uint32_t h, const uint32_t* d_paths,
                  const float light[3], float bias, uint8_t* d_mask, unsigned long long* d_counters,
                  cudaStream_t stream, const uint32_t* d_root, uint32_t* d_list)
{
    shadow_pass(c, cam, w, h, d_paths, light, bias, d_mask, d_counters, stream ? stream : c->stream,
                d_root ? d_root : c->d_root, d_list);
}

// n_views frames in three launches: the views' camera tables, primary rays
// of every view with the shadow-ray list, then the shadow rays of every hit
// pixel of every view.
void trace_views(hd_ctx* c, const hd_camera* d_cams, uint32_t n_views, uint32_t w, uint32_t h, uint32_t* d_paths,
                 const float light[3], float bias, uint8_t* d_mask, cudaStream_t stream, uint32_t* d_list,
                 cudaEvent_t mid, const uint32_t* d_root, double* d_tables, uint32_t* d_paths_copied)
{
    cudaStream_t st = stream ? stream : c->stream;
    const uint32_t* rt = d_root ? d_root : c->d_root;
    const uint64_t px = uint64_t(w) * h * n_views;
    if (px >= 0xFFFFFFFFull)
        throw StatusError{HD_ERR_INVALID, "views x width x height must stay below 2^32 pixels"};
    uint32_t* buf = d_list ? d_list : c->scratch.get<uint32_t>("shadow_list", shadow_list_words(px));
    ShadowRay* list = reinterpret_cast<ShadowRay*>(buf);
    uint32_t* head = buf + 4 * px;
    HD_CUDA(cudaMemsetAsync(head, 0, 16, st));
    uint4* out = reinterpret_cast<uint4*>(d_paths);
    const uint64_t tiles = uint64_t((w + 7) / 8) * ((h + 3) / 4);
    const F3 l = {light[0], light[1], light[2]};
    const uint64_t tab_words = camera_table_words(w, h) * n_views;
    double* tables = d_tables ? d_tables : c->scratch.get<double>("cam_tables", tab_words);
    const uint32_t tab_blocks = grid_for(uint64_t(w + h) * n_views, 256);
    auto launch = [&](auto tab_kernel, auto kernel) {
        tab_kernel<<<tab_blocks, 256, 0, st>>>(d_cams, n_views, w, h, tables);
        HD_LAUNCH_CHECK();
        const uint32_t smem = shared_stack_bytes(128, c->t.g.depth);
        const uint32_t blocks = uint32_t(std::min<uint64_t>(
            (tiles * n_views + 3) / 4,
            resident_blocks(reinterpret_cast<const void*>(kernel), 128, smem)));
        kernel<<<blocks, 128, smem, st>>>(c->t, rt, d_cams, w, h, n_views, out, l, bias, d_mask, list, head, tables,
                                          reinterpret_cast<uint4*>(d_paths_copied));
    };
    if (c->fp_mode)
        launch(k_camera_tables<1>, k_trace_views<1>);
    else
        launch(k_camera_tables<0>, k_trace_views<0>);
    HD_LAUNCH_CHECK();
    if (mid)
        HD_CUDA(cudaEventRecord(mid, st));
    shadow_walks(c, px, light, d_mask, nullptr, st, rt, list, head);
}

// DAGUtils::get_value
__global__ void k_get_values(Table t, const uint32_t* __restrict__ d_root, const uint32_t* __restrict__ xyz,
                             uint64_t n, uint8_t* __restrict__ out)
{
    const uint32_t root = *d_root;
    HD_GRID_STRIDE(i, n)
    {
        const uint32_t x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
        uint32_t index = root;
        uint8_t v = 0;
        for (uint32_t level = 0; level < t.g.depth; level++) {
            if (level < t.g.leaf_level) {
                // one translation per node: its child pointers follow the
                // header in the same page
                const uint32_t* p = t.sys(index);
                const uint32_t mask = __ldg(p) & 0xffu;
                const uint32_t s = t.g.depth - (level + 1);
                const uint32_t child = (((x >> s) & 1) << 2) | (((y >> s) & 1) << 1) | ((z >> s) & 1);
                if (!(mask & (1u << child)))
                    break;
                index = __ldg(p + child_offset(mask, child));
            } else {
                const uint32_t* p = t.sys(index);
                const uint64_t leaf = uint64_t(__ldg(p)) | (uint64_t(__ldg(p + 1)) << 32);
                v = uint8_t((leaf >> leaf_bit(x, y, z)) & 1);
                break;
            }
        }
        out[i] = v;
    }
}

void get_values(hd_ctx* c, const uint32_t* d_xyz, uint64_t n, uint8_t* d_out)
{
    if (!n)
        return;
    k_get_values<<<grid_for(n, 256), 256, 0, c->stream>>>(c->t, c->d_root, d_xyz, n, d_out);
    HD_LAUNCH_CHECK();
}

} // namespace hd

// ---------------------------------------------------------------------------
// Traversal counters without any device allocation.
//
// Some callers cannot call cudaMalloc at the time they trace: an embedding
// application (a game engine, a plugin host) that reserves the device
// memory budget at start-up and forbids allocations afterwards, or a
// real-time loop in which cudaMalloc / cudaFree, which may synchronise the
// whole device, would stall the other streams' work.  This variant of
// hd_trace_counters keeps its scratch (one partial sum per 8x8-pixel block
// and the six totals) in a file-scope device array instead of the context's
// scratch buffers.  The array holds kNoAllocMaxBlocks blocks, i.e. images of
// up to 16,777,216 pixels (4096 x 4096); larger images, and images taller
// than 65535 rows of blocks (524,280 pixels), are rejected.  The
// array lives on every GPU that loads the library until the process exits.
// All calls share it: each call writes every slot it later reads, so
// nothing needs clearing, but calls that overlap on the GPU (other streams,
// other threads) race on it.
// ---------------------------------------------------------------------------
namespace hd {

constexpr uint32_t kNoAllocMaxBlocks = 262144;
__device__ __align__(256) unsigned long long g_noalloc_scratch[3 * kNoAllocMaxBlocks + 8];

HD_D void block_sum3(uint32_t a, uint32_t b, uint32_t c, unsigned long long* dst)
{
    __shared__ unsigned long long part[2][3];
    unsigned long long v[3] = {a, b, c};
    for (int k = 0; k < 3; k++)
        for (int o = 16; o; o >>= 1)
            v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; k++)
            part[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < 3; k++)
            dst[k] = part[0][k] + part[1][k];
}

template <int FMA>
__global__ void __launch_bounds__(64) k_trace_primary_partials(Table t, const uint32_t* __restrict__ d_root,
                                                               hd_camera cam, uint32_t W, uint32_t H,
                                                               uint4* __restrict__ out,
                                                               unsigned long long* __restrict__ partial)
{
    const uint32_t x = blockIdx.x * 8 + (threadIdx.x & 7);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 3);
    uint32_t rays = 0, descents = 0, leaves = 0;
    if (x < W && y < H) {
        double dd[3];
        camera_dir<FMA>(cam, double(x), double(y), dd);
        const F3 d = {float(dd[0]), float(dd[1]), float(dd[2])};
        const F3 o = {float(cam.position[0]), float(cam.position[1]), float(cam.position[2])};
        uint32_t hit[3];
        walk<FMA>(t, *d_root, o, d, inverse_dir(d), hit, descents, leaves);
        out[uint64_t(H - 1 - y) * W + x] = make_uint4(hit[0], hit[1], hit[2], 0);
        rays = 1;
    }
    block_sum3(rays, descents, leaves, partial + 3 * (uint64_t(blockIdx.y) * gridDim.x + blockIdx.x));
}

template <int FMA>
__global__ void __launch_bounds__(64) k_trace_shadow_partials(Table t, const uint32_t* __restrict__ d_root,
                                                              hd_camera cam, uint32_t W, uint32_t H,
                                                              const uint4* __restrict__ paths, F3 light, float bias,
                                                              uint8_t* __restrict__ mask,
                                                              unsigned long long* __restrict__ partial)
{
    const uint32_t x = blockIdx.x * 8 + (threadIdx.x & 7);
    const uint32_t r = blockIdx.y * 8 + (threadIdx.x >> 3);
    uint32_t rays = 0, descents = 0, leaves = 0;
    if (x < W && r < H) {
        const uint64_t i = uint64_t(r) * W + x;
        const uint4 p = paths[i];
        if (p.x == 0 && p.y == 0 && p.z == 0) {
            mask[i] = 2;
        } else {
            // the same origin and front-to-back order as the shadow pass
            const F3 dir = light_dir<FMA>(light);
            const F3 o = shadow_origin<FMA>(cam, H, x, r, p, dir, bias);
            uint32_t hit[3];
            mask[i] = walk<FMA>(t, *d_root, o, dir, inverse_dir(dir), hit, descents, leaves) ? 1 : 0;
            rays = 1;
        }
    }
    block_sum3(rays, descents, leaves, partial + 3 * (uint64_t(blockIdx.y) * gridDim.x + blockIdx.x));
}

// One block: column sums of the partials into totals[0..2].
__global__ void k_sum_partials(const unsigned long long* __restrict__ partial, uint32_t nblocks,
                               unsigned long long* __restrict__ totals)
{
    __shared__ unsigned long long acc[3][256];
    for (int k = 0; k < 3; k++) {
        unsigned long long s = 0;
        for (uint32_t b = threadIdx.x; b < nblocks; b += blockDim.x)
            s += partial[3 * uint64_t(b) + k];
        acc[k][threadIdx.x] = s;
    }
    __syncthreads();
    for (uint32_t w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int k = 0; k < 3; k++)
                acc[k][threadIdx.x] += acc[k][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 3)
        totals[threadIdx.x] = acc[threadIdx.x][0];
}

} // namespace hd

namespace {
// Device address of g_noalloc_scratch per device, resolved on the first
// call made with that device current.
std::mutex g_noalloc_mutex;
unsigned long long* g_noalloc_ptr[256] = {};

unsigned long long* noalloc_scratch()
{
    int dev = 0;
    HD_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256)
        throw hd::StatusError{HD_ERR_INVALID, "device ordinal out of range"};
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        HD_CUDA(cudaGetSymbolAddress(&p, hd::g_noalloc_scratch));
        g_noalloc_ptr[dev] = static_cast<unsigned long long*>(p);
    }
    return g_noalloc_ptr[dev];
}
} // namespace

extern "C" hd_status hd_trace_counters_noalloc(hd_ctx* c, const hd_camera* cam, uint32_t w, uint32_t h,
                                               const float light[3], float bias, uint32_t* d_paths, uint8_t* d_mask,
                                               uint64_t out[6])
{
    using namespace hd;
    if (!c || !cam || !d_paths || !d_mask || !light || !out || !w || !h)
        return HD_ERR_INVALID;
    const uint64_t bx = (w + 7) / 8, by = (h + 7) / 8;
    if (bx * by > kNoAllocMaxBlocks) {
        c->err = "hd_trace_counters_noalloc: image of " + std::to_string(uint64_t(w) * h) +
                 " pixels exceeds the fixed scratch (at most 262144 blocks of 8x8 pixels, 16777216 pixels)";
        return HD_ERR_INVALID;
    }
    if (by > kMaxGridRows) {
        c->err = "hd_trace_counters_noalloc: image height " + std::to_string(h) + " exceeds " +
                 std::to_string(8 * kMaxGridRows) + " rows";
        return HD_ERR_INVALID;
    }
    try {
        unsigned long long* scratch = noalloc_scratch();
        unsigned long long* partial = scratch;
        unsigned long long* totals = scratch + 3 * uint64_t(kNoAllocMaxBlocks);
        const dim3 grid{uint32_t(bx), uint32_t(by), 1u};
        const uint32_t nb = uint32_t(bx * by);
        const F3 l = {light[0], light[1], light[2]};
        uint4* paths = reinterpret_cast<uint4*>(d_paths);
        if (c->fp_mode)
            k_trace_primary_partials<1><<<grid, 64, 0, c->stream>>>(c->t, c->d_root, *cam, w, h, paths, partial);
        else
            k_trace_primary_partials<0><<<grid, 64, 0, c->stream>>>(c->t, c->d_root, *cam, w, h, paths, partial);
        HD_LAUNCH_CHECK();
        k_sum_partials<<<1, 256, 0, c->stream>>>(partial, nb, totals);
        HD_LAUNCH_CHECK();
        if (c->fp_mode)
            k_trace_shadow_partials<1><<<grid, 64, 0, c->stream>>>(c->t, c->d_root, *cam, w, h, paths, l, bias,
                                                                   d_mask, partial);
        else
            k_trace_shadow_partials<0><<<grid, 64, 0, c->stream>>>(c->t, c->d_root, *cam, w, h, paths, l, bias,
                                                                   d_mask, partial);
        HD_LAUNCH_CHECK();
        k_sum_partials<<<1, 256, 0, c->stream>>>(partial, nb, totals + 3);
        HD_LAUNCH_CHECK();
        HD_CUDA(cudaMemcpyAsync(out, totals, 6 * sizeof(uint64_t), cudaMemcpyDeviceToHost, c->stream));
        HD_CUDA(cudaStreamSynchronize(c->stream));
        return HD_OK;
    } catch (const StatusError& e) {
        c->err = e.msg;
        return e.status;
    } catch (const CudaError& e) {
        c->err = std::string("CUDA error ") + cudaGetErrorString(e.code) + " in " + e.where;
        return HD_ERR_CUDA;
    }
}
