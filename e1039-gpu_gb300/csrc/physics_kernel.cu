// physics_kernel.cu -- the stages after global tracking: vertexing, dimuon
// building and the monitoring histograms.
//
// Replaces gKernel_Vertexing (OnlineReconstruction/reconstruction_kernels.cuh
// :2542-2810), gKernel_DimuonBuilding (:2820-3090, with
// FindDimuonClosestApproach, reconstruction_helper.cuh:1269-1477) and
// gKernel_fill_display_histograms (:3100-3195), launched in that order after
// the post-global selection (online_reconstruction.cu:939-983).
//
//  - Vertexing swims each global track (stationID >= 6) back through FMag in
//    double, 100 magnet steps with energy loss and 100 target steps, and keeps
//    the point of closest approach to the beam line: stationID 7, vertex
//    position and momentum.  The reference gives a thread to each slot, so a
//    warp works for the one or two lanes whose slot holds a global track;
//    here a warp gathers the global tracks of some events into a shared list
//    and swims them one per lane, which keeps the lanes of the double-
//    precision loop busy (FP64 is the scarce unit of this GPU).  The swim is
//    not stored: the closest-approach scan visits the points in step order
//    with a strict "smaller than" test, so it runs as the points are made.
//  - Dimuons: the two swims of a pair depend on its tracks alone and are made
//    by two lanes side by side; the pairs of an event are then gone through in
//    order by its own lane, as the reference's pair loop carries state from
//    one pair to the next (the swum momenta of the current track stay in
//    p_pos / p_neg).
//  - Histograms: one warp per event, lanes over the (trigger, variable)
//    tables, each searched by halves; counts go in with atomics, so the result is the exact
//    count whatever the order (the reference's plain "+=" from concurrent
//    blocks loses updates).
//
// Every expression keeps the operand types of the reference expression it
// restates (float track parameters, double step and energy-loss constants,
// sqrtf on double expressions), so promotions and roundings are the same.
#include <algorithm>

#include "or_device.cuh"

namespace orgpu {

namespace phys {
constexpr float X_BEAM = 0.f, Y_BEAM = 0.f;          // K0:75-76
constexpr double PTKICK_UNIT = -0.006096568;         // K0:93
constexpr double FMAG_LENGTH = 502.92;               // K0:110
constexpr double FMAG_HOLE_LENGTH = 27.94;           // K0:111
constexpr double FMAG_HOLE_RADIUS = 1.27;            // K0:112
constexpr int NSTEPS_FMAG = 100;                     // K0:113
constexpr double STEP_FMAG = 2.514600;               // K0:114
constexpr double DEDX_UNIT_0 = 0.014282073;          // K0:115-119
constexpr double DEDX_UNIT_1 = 7.1869681e-05;
constexpr double DEDX_UNIT_2 = -1.4279150e-06;
constexpr double DEDX_UNIT_3 = 1.5853655e-08;
constexpr double DEDX_UNIT_4 = -6.0741470e-11;
constexpr int NSTEPS_TARGET = 100;                   // K0:120
constexpr double STEP_TARGET = 5.0;                  // K0:121
constexpr float EBEAM = 120.f, MP = 0.938272f, PBEAM = 119.996331801f, MMU = 0.105658f;  // K0:210-213
constexpr float CHI2DOF_MAX = 250.f;                 // K0:194
constexpr int VTX_LIST = 256;                        // vertexing list entries per warp
}  // namespace phys

// gTracks::get_firsthitdetid (reconstruction_classes.cuh:517-532)
__device__ __forceinline__ short first_hit_detid(const float *T, const float *z) {
    const int nhits = (int)T[OR_TRK_NHITS];
    short detid_min = 30;
    float z_min = 10000.f;
    for (int i = 0; i < nhits && i < OR_MAXHITS_PER_TRACK; ++i) {
        const short d = (short)T[OR_TRK_HIT_DETID + i];
        if (d > 0 && z[d] < z_min) {
            detid_min = d;
            z_min = z[d];
        }
    }
    return detid_min;
}

// calculate_x0_tx_st1 (H:622-626)
__device__ __forceinline__ void x0_tx_st1(float x0, float tx, float invP, short charge, float &x0_st1, float &tx_st1) {
    tx_st1 = tx + PT_KICK_KMAG * invP * charge;
    x0_st1 = tx * Z_KMAG_BEND + x0 - tx_st1 * Z_KMAG_BEND;
}

__device__ __forceinline__ double dedx_poly(double p) {
    using namespace phys;
    return DEDX_UNIT_0 + DEDX_UNIT_1 * p + DEDX_UNIT_2 * p * p + DEDX_UNIT_3 * p * p * p + DEDX_UNIT_4 * p * p * p * p;
}

// ---------------------------------------------------------------------------
// vertexing (K:2594-2803)

#ifndef OR_VTX_GROUP
#define OR_VTX_GROUP 16
#endif
static_assert(OR_VTX_GROUP <= 32, "a flag of a warp's events per lane");

// The z of every step: the same subtractions for every track.
struct VtxZ {
    double z[phys::NSTEPS_FMAG + phys::NSTEPS_TARGET + 1];
    int first_half, second_half;  // steps whose first (second) half ends above the hole's length
};
constexpr VtxZ vtx_z() {
    using namespace phys;
    VtxZ o{};
    double z = FMAG_LENGTH;
    o.z[0] = z;
    for (int k = 1; k <= NSTEPS_FMAG; ++k) {
        const double b = z - STEP_FMAG;
        z = b - STEP_FMAG;
        o.z[k] = z;
        if (b > FMAG_HOLE_LENGTH) o.first_half = k;
        if (z > FMAG_HOLE_LENGTH) o.second_half = k;
    }
    for (int k = NSTEPS_FMAG + 1; k <= NSTEPS_FMAG + NSTEPS_TARGET; ++k) {
        z = z - STEP_TARGET;
        o.z[k] = z;
    }
    return o;
}
__device__ __constant__ VtxZ c_vtx = vtx_z();
constexpr int VTX_FIRST = vtx_z().first_half, VTX_SECOND = vtx_z().second_half;

// The helpers below work on the bits of doubles with integer and float
// instructions, without branches; each clears `ok` outside the range it is
// exact for, and its caller then evaluates the double expression.

// The double expressions are calls, so that they are not evaluated beside the
// others (inlined, the compiler did: a step's three square roots took 900
// cycles each instead of 300).
__device__ __noinline__ double slow_sqrt(double s) { return sqrt(s); }
__device__ __noinline__ double slow_div(double m, double p) { return m / p; }
__device__ __noinline__ double slow_loss(double ptot, float len) { return ptot + dedx_poly(ptot) * len; }
__device__ __noinline__ float slow_length(double t, double c1, double c2) { return t * t + c1 + c2; }
__device__ __noinline__ bool slow_closer(float away, double mx, double px, double py, double bx, double by, bool first) {
    using namespace phys;
    const double dca2 = (px - X_BEAM) * (px - X_BEAM) + (py - Y_BEAM) * (py - Y_BEAM);
    const double dca2_min = first ? 1.e18 : (bx - X_BEAM) * (bx - X_BEAM) + (by - Y_BEAM) * (by - Y_BEAM);
    return !(away * mx < 0.) && dca2 < dca2_min;
}

// whether the exponent field of a double lies in [lo, hi)
__device__ __forceinline__ bool dbl_range(int hi_word, int lo, int hi) {
    return (unsigned)(((hi_word >> 20) & 0x7FF) - lo) < (unsigned)(hi - lo);
}
__device__ __forceinline__ bool dbl_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
// a double's leading bits as a float (error below 2^-23)
__device__ __forceinline__ float dbl_lead(double x, bool &ok) {
    const int hi = __double2hiint(x);
    ok &= dbl_range(hi, 896 + 10, 896 + 245);
    // the exponent's low nine bits lead; 0x380 less (modulo 2^9) is the float's
    const unsigned m = __funnelshift_l((unsigned)__double2loint(x), (unsigned)hi, 3) + 0x40000000u;
    return __int_as_float((hi & 0x80000000) | (int)(m & 0x7FFFFFFFu));
}
// a double as two floats, to 46 bits
__device__ __forceinline__ FF dbl_ff(double x, bool &ok) {
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    ok &= dbl_range(hi, 896 + 60, 896 + 245);
    const float h = dbl_lead(x, ok);
    // 23 of the 29 bits left, as the fraction of h's last place
    const int u = (__float_as_int(h) & 0xFF800000) - (23 << 23);
    return FF{h, __int_as_float(u | (int)((lo >> 6) & 0x7FFFFF)) - __int_as_float(u)};
}
// x plus k units of its last place
__device__ __forceinline__ double dbl_ulps(double x, int k) {
    return __longlong_as_double(__double_as_longlong(x) + k);
}
// whether no power of two is within 2048 units of x
__device__ __forceinline__ bool dbl_inside(double x) {
    return (((unsigned long long)__double_as_longlong(x) + 2048) & 0xFFFFFFFFFFFFFull) >= 4096;
}
// the nearest integer, |x| < 2^22
__device__ __forceinline__ int flt_round(float x) { return __float_as_int(x + 0x1.8p23f) - 0x4B400000; }

// m / p for m = the rounded product q * p: the quotient is q or a neighbour,
// decided by the product's rounding error, one FMA (P. Markstein, IA-64 and
// Elementary Functions, 2000, ch. 8: the remainder of an approximate quotient
// is exact).
__device__ __forceinline__ double vtx_ratio(double m, double p, double q, bool &sure) {
    const double r = __fma_rn(-q, p, m);
    const int hq = __double2hiint(q);
    bool ok = dbl_inside(q) & dbl_range(hq, 896 + 30, 896 + 200);
    const float pf = dbl_lead(p, ok);
    ok &= (pf > 0x1p-20f) & (pf < 0x1p20f);
    const bool exact = ok & dbl_zero(r);
    const float rf = dbl_lead(r, ok);
    // half a unit of q's last place, times p; scaled by 2^60 with r
    const int e = (hq >> 20) & 0x7FF;
    const float half = pf * __int_as_float((e - 896 - 53 + 60) << 23);
    const float rs = fabsf(rf) * 0x1p60f;
    ok &= (rs < half * (1.f - 0x1p-16f)) | (rs > half * (1.f + 0x1p-16f));
    const int k = (rs < half) | exact ? 0 : ((__float_as_int(rf) ^ hq) < 0 ? -1 : 1);
    sure = ok | exact;
    return dbl_ulps(q, k);
}

// h + c (|c| some 2^-22 of h) as a double; `scale` becomes one over a unit of
// its last place
__device__ __forceinline__ double dbl_join(float h, float c, float &scale, bool &ok) {
    const int u = __float_as_int(h), e = u & 0x7F800000;
    ok &= (unsigned)(e - ((127 - 40) << 23)) < (80u << 23);
    scale = __int_as_float(((52 + 127 + 127) << 23) - e);
    const float ks = (u < 0 ? -c : c) * (0x1p-9f * scale);  // in units of 2^9
    const float k1 = (ks + 0x1.8p23f) - 0x1.8p23f;
    const int lo = flt_round((ks - k1) * 0x1p9f);
    const double x = __hiloint2double((u & 0x80000000) | ((u & 0x7FFFFFFF) >> 3) + 0x38000000, u << 29);
    const double g = __longlong_as_double(__double_as_longlong(x) + (long long)flt_round(ks) * 512 + lo);
    ok &= dbl_inside(g) & (((__double2hiint(g) ^ __double2hiint(x)) & 0x7FF00000) == 0) & (fabsf(ks) < 0x1p22f);
    return g;
}
// moves g by x units of its last place, x known to 2^-9, rounded to whole
// units; `ok` is cleared when the rounding is not sure
__device__ __forceinline__ double dbl_settle(double g, float x, bool &ok) {
    const float k = (x + 0x1.8p23f) - 0x1.8p23f;
    ok &= (fabsf(x) < 1024.f) & (fabsf(x - k) < 0.498f);
    return dbl_ulps(g, flt_round(x));
}

// sqrt(s): two floats' worth of it, then one FMA gives what is left, exactly
// enough to round (the remainder of an approximate root, as that of a quotient
// above: Markstein 2000).  y is 1 / sqrt(s) to a float.
__device__ __forceinline__ double vtx_sqrt(double s, float &y, bool &sure) {
    bool ok = true;
    const FF a = dbl_ff(s, ok);
    y = rsqrtf(a.h);
    const float h = a.h * y, c = (__fmaf_rn(-h, h, a.h) + a.l) * (0.5f * y);
    float scale;
    const double g = dbl_join(h, c, scale, ok);
    const double d = __fma_rn(-g, g, s);
    const bool exact = ok & dbl_zero(d);
    const double r = dbl_settle(g, dbl_lead(d, ok) * (0.5f * y) * scale, ok);
    sure = ok | exact;
    return exact ? g : r;
}

// m / p, y being 1 / p to a float, the same way (Markstein's remainder of the
// quotient)
__device__ __forceinline__ double vtx_div(double m, double p, float y, bool &sure) {
    bool ok = y > 0.f;
    const FF a = dbl_ff(m, ok), b = dbl_ff(p, ok);
    const float h = a.h * y, c = (__fmaf_rn(-h, b.h, a.h) + (a.l - h * b.l)) * y;
    float scale;
    const double q = dbl_join(h, c, scale, ok);
    const double d = __fma_rn(-q, p, m);
    const bool exact = ok & dbl_zero(d);
    const float x = dbl_lead(d, ok) * y * scale;
    const double r = dbl_settle(q, h < 0.f ? -x : x, ok);
    sure = ok | exact;
    return exact ? q : r;
}

// (float)(t * t + c), c = the other two squares' sum
__device__ __forceinline__ float vtx_length(double t, FF c, bool &sure) {
    bool ok = true;
    const FF a = dbl_ff(t, ok);
    const float p = a.h * a.h;
    const FF v = ff_add(ff_fast(p, __fmaf_rn(a.h, a.h, -p) + 2.f * a.h * a.l), c);
    sure = ok & ff_sure(v);
    return v.h;
}

// ptot + dedx_poly(ptot) * len.  For 4 <= ptot < 128 the loss is formed in
// fixed point (Horner in units of 2^-67) and added to ptot's significand with
// ten more bits; the double expression's own rounding errors come to at most
// `margin` of those units (a bound over each binade: j roundings in the
// power j, one in each of the four sums, one in the product by len < 3, plus
// two units for the truncations here), so the sum decides the result unless it is that close to
// the middle of two doubles (some 2 % of the tracks' steps).
__host__ __device__ constexpr long long loss_coef(double c) { return (long long)(c * 0x1p67); }
__device__ __forceinline__ double vtx_loss(double ptot, float len, bool &sure) {
    using namespace phys;
    const long long bits = __double_as_longlong(ptot);
    const int k = (int)(bits >> 52) - 1023, ul = __float_as_int(len);
    const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    const long long x = (long long)(m << ((k + 4) & 15));  // ptot / 128 in units of 2^-63
    long long a = loss_coef(DEDX_UNIT_4 * 0x1p28);
    a = __mul64hi(a, x) * 2 + loss_coef(DEDX_UNIT_3 * 0x1p21);
    a = __mul64hi(a, x) * 2 + loss_coef(DEDX_UNIT_2 * 0x1p14);
    a = __mul64hi(a, x) * 2 + loss_coef(DEDX_UNIT_1 * 0x1p7);
    a = __mul64hi(a, x) * 2 + loss_coef(DEDX_UNIT_0);
    const long long v = __mul64hi(a, (long long)((ul & 0x7FFFFF) | 0x800000) << 39);  // units of 2^-64
    const unsigned long long w = (m << 10) + (unsigned long long)(v >> ((k + 2) & 15));
    const unsigned long long r = (w + 512) >> 10;
    // the error bound of the double expression: 30, 17, 10, 7, 9 units for k = 2 .. 6
    const int margin = max(10, 136 >> (k & 7));
    sure = ((unsigned)(k - 2) <= 4u) & (ul >= 0x40000000) & (ul < 0x40400000) & ((r >> 52) == 1) &
           (abs((int)(w & 1023) - 512) > margin);
    return __longlong_as_double((bits & 0x7FF0000000000000ll) | (long long)(r & 0xFFFFFFFFFFFFFull));
}

// The swim of one track.  An FP64 instruction takes a warp 64 cycles of its
// quarter of the SM, whatever its active lanes (measured), so what need not be
// FP64 to give the same bits is not: the z of a step is a constant, its hole
// test too; roots and quotients are two floats' worth refined by one FMA; the
// slope of a step is the quotient of a product by its factor; path lengths are
// floats; the energy loss is formed in fixed point; and a point is compared
// with the closest so far by leading bits.  Each of these knows when it cannot
// decide the last bit, and the double expression does then.  Some 25 FP64
// instructions a magnet step remain of 147, 2 of 9 a target step.  Bound: the
// chain of one step into the next, some 4,000 cycles.
__device__ void vertex_track(float *T, const float *z) {
    using namespace phys;
    const float x0 = T[OR_TRK_X0], y0 = T[OR_TRK_Y0], tx = T[OR_TRK_TX], ty = T[OR_TRK_TY];
    const float invP = T[OR_TRK_INVP], charge = T[OR_TRK_CHARGE];
    const short detid_first = first_hit_detid(T, z);
    float x0_st1, tx_st1;
    x0_tx_st1(x0, tx, invP, (short)charge, x0_st1, tx_st1);
    const double z_0 = z[detid_first];
    const double s0 = charge * invP * sqrtf((1.f + tx_st1 * tx_st1) / (1.f + tx_st1 * tx_st1 + ty * ty));
    const double s1 = tx_st1, s2 = ty;
    const double s3 = (float)z_0 * tx_st1 + x0_st1, s4 = (float)z_0 * ty + y0;
    double px = s3 + s1 * (FMAG_LENGTH - z_0), py = s4 + s2 * (FMAG_LENGTH - z_0);
    const double pz_0 = 1.f / (fabs(s0) * sqrtf(1.f + s1 * s1 + s2 * s2));
    double mx = pz_0 * s1, my = pz_0 * s2, mz = pz_0;
    // the closest point: its place, momentum and step; step -1: none yet
    double bx = 0., by = 0., bmx = 0., bmy = 0., bmz = 0.;
    float best = 1.e18f;  // leading bits of its squared distance; NaN: not known
    int bstep = -1;
    const float away = FMAGSTR * charge;
    const bool away_ok = (fabsf(away) > 0x1p-100f) & (fabsf(away) < 0x1p100f);
    static_assert(X_BEAM == 0.f && Y_BEAM == 0.f, "the leading bits are those of the distance");
    auto visit = [&](int step) {
        // FMAGSTR * charge * mx < 0, by signs where the product cannot vanish
        const int hm = __double2hiint(mx);
        const bool out = (hm ^ __float_as_int(away)) < 0;
        bool ok = true;
        const float fx = dbl_lead(px, ok), fy = dbl_lead(py, ok);
        const float d = fx * fx + fy * fy;
        ok &= (d > 1e-20f) & (d < 1e30f);
        const bool nearer = d < best * (1.f - 0x1p-16f), farther = d > best * (1.f + 0x1p-16f);
        bool take = !out & nearer;
        if (!(away_ok & dbl_range(hm, 100, 0x7FF) & (out | (ok & (nearer | farther)))))
            take = slow_closer(away, mx, px, py, bx, by, bstep < 0);
        if (take) {
            best = ok ? d : __int_as_float(0x7FFFFFFF);
            bstep = step;
            bx = px; by = py;
            bmx = mx; bmy = my; bmz = mz;
        }
    };
    visit(0);
    const double kick = 2.f * charge * PTKICK_UNIT * STEP_FMAG;
    const double t1 = ty * STEP_FMAG, t11 = t1 * t1, t12 = STEP_FMAG * STEP_FMAG;
    const double csum = t11 + t12, tyy = ty * ty;
    const FF c = FF{(float)csum, (float)(csum - (double)(float)csum)};
    double slope = s1;  // mx = mz * slope, rounded
#pragma unroll 1
    for (int step = 1; step <= NSTEPS_FMAG; ++step) {
        // what depends on the same values side by side, then one branch for
        // the lanes that need the double expressions
        const double mxx = mx * mx, mzz = mz * mz, sxz = mxx + mzz, sxyz = mxx + my * my + mzz;
        float y_xz, y_p, y_n;
        bool ok1, ok2, ok3, ok4;
        double tx_i = vtx_ratio(mx, mz, slope, ok1);
        double pxz = vtx_sqrt(sxz, y_xz, ok2), ptot_i = vtx_sqrt(sxyz, y_p, ok3);
        if (!(ok1 & ok2 & ok3)) {
            if (!ok1) tx_i = slow_div(mx, mz);
            if (!ok2) pxz = slow_sqrt(sxz);
            if (!ok3) ptot_i = slow_sqrt(sxyz);
        }
        double turn = vtx_div(kick, pxz, y_xz, ok1);
        const double t10 = tx_i * STEP_FMAG, b0 = px - t10, b1 = py - t1;
        float q1 = vtx_length(t10, c, ok2);
        if (!(ok1 & ok2)) {
            if (!ok1) turn = slow_div(kick, pxz);
            if (!ok2) q1 = slow_length(t10, t11, t12);
        }
        const double tx_f = tx_i + turn, t20 = tx_f * STEP_FMAG, snorm = 1.f + tx_f * tx_f + tyy;
        double norm = vtx_sqrt(snorm, y_n, ok1);
        float q2 = vtx_length(t20, c, ok2);
        const float len1 = sqrtf(q1);
        double ptot_b = vtx_loss(ptot_i, len1, ok3);
        const bool in1 = step <= VTX_FIRST || b0 * b0 + b1 * b1 > FMAG_HOLE_RADIUS;
        if (!(ok1 & ok2 & (ok3 | !in1))) {
            if (!ok1) norm = slow_sqrt(snorm);
            if (!ok2) q2 = slow_length(t20, t11, t12);
            if (!ok3) ptot_b = slow_loss(ptot_i, len1);
        }
        if (!in1) ptot_b = ptot_i;
        px = b0 - t20;
        py = b1 - t1;
        const float len2 = sqrtf(q2);
        double ptot_f = vtx_loss(ptot_b, len2, ok4);
        const bool in2 = step <= VTX_SECOND || px * px + py * py > FMAG_HOLE_RADIUS;
        if (!ok4 & in2) ptot_f = slow_loss(ptot_b, len2);
        if (!in2) ptot_f = ptot_b;
        double pz_f = vtx_div(ptot_f, norm, y_n, ok1);
        if (!ok1) pz_f = slow_div(ptot_f, norm);
        mx = pz_f * tx_f;
        my = pz_f * ty;
        mz = pz_f;
        slope = tx_f;
        visit(step);
    }
    {
        const double dx = mx / mz * STEP_TARGET, dy = ty * STEP_TARGET;
#pragma unroll 1
        for (int step = NSTEPS_FMAG + 1; step <= NSTEPS_FMAG + NSTEPS_TARGET; ++step) {
            px = px - dx;
            py = py - dy;
            visit(step);
        }
    }
    if (bstep < 0) {  // the last point (K:2752)
        bstep = NSTEPS_FMAG + NSTEPS_TARGET;
        bx = px; by = py;
        bmx = mx; bmy = my; bmz = mz;
    }
    T[OR_TRK_STID] = 7.f;  // K:2796
    T[OR_TRK_VX] = (float)bx;
    T[OR_TRK_VX + 1] = (float)by;
    T[OR_TRK_VX + 2] = (float)c_vtx.z[bstep];
    T[OR_TRK_PX] = (float)bmx;
    T[OR_TRK_PX + 1] = (float)bmy;
    T[OR_TRK_PX + 2] = (float)bmz;
}

// One warp per block, so that the warps spread over the SMs before they
// share one: the swim is bound by the FP64 pipes, one to each quarter of an
// SM (a warp's swim takes some 240 us of one, whatever its lanes), and
// blocks of four warps left half of the SMs idle (10,000 events: 1,016 us;
// now 332 us, 2,000 events 1,012 -> 244 us).  A warp gathers the
// tracks (stationID >= 6) of `group` events, lane = slot, into a shared list
// and swims them one per lane.
__global__ void __launch_bounds__(32)
    vertex_kernel(const or_plane_t *__restrict__ gplane, or_tracks_view_t tv, const uint8_t *__restrict__ toomany,
                  int n_events, int group) {
    __shared__ float zs[OR_NDET];
    __shared__ uint32_t list[phys::VTX_LIST];
    const int lane = threadIdx.x;
    for (int i = lane; i < OR_NDET; i += 32) zs[i] = gplane->z[i];
    __syncwarp();
    for (long e0 = (long)blockIdx.x * group; e0 < n_events; e0 += (long)gridDim.x * group) {
        const long e1 = min(e0 + group, (long)n_events);
        const unsigned live = __ballot_sync(0xffffffffu, e0 + lane < e1 && !toomany[min(e0 + lane, e1 - 1)]);
        int waiting = 0;
        for (long eb = e0; eb < e1; eb += 8) {  // eight events' counts and stationIDs in flight
            int n[8], most = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const bool have = eb + i < e1 && ((live >> (int)(eb + i - e0)) & 1u);
                n[i] = have ? min((int)tv.ntracks[(eb + i) * OR_NSLOTS + lane], OR_SLOTCAP) : 0;
                most = max(most, n[i]);
            }
            most = __reduce_max_sync(0xffffffffu, most);
#pragma unroll 1
            for (int k = 0; k < most; ++k) {
                unsigned take = 0u;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (k < n[i] && trk_rec(tv, eb + i, lane, k)[OR_TRK_STID] >= 6) take |= 1u << i;  // K:2594
#pragma unroll 1
                for (int i = 0; i < 8; ++i) {
                    const unsigned m = __ballot_sync(0xffffffffu, (take >> i) & 1u);
                    if ((take >> i) & 1u)
                        list[waiting + __popc(m & lanemask_lt())] =
                            (uint32_t)(eb + i - e0) << 9 | (uint32_t)(lane * OR_SLOTCAP + k);
                    waiting += __popc(m);
                    __syncwarp();
                    // swim full warps of tracks as the list fills
                    while (waiting >= phys::VTX_LIST - 32) {
                        waiting -= 32;
                        const uint32_t c = list[waiting + lane];
                        vertex_track(trk_rec(tv, e0 + (c >> 9), (int)(c & 511u) / OR_SLOTCAP, (int)(c & 511u) % OR_SLOTCAP),
                                     zs);
                        __syncwarp();
                    }
                }
            }
        }
#pragma unroll 1
        for (int i = lane; i < waiting; i += 32) {
            const uint32_t c = list[i];
            vertex_track(trk_rec(tv, e0 + (c >> 9), (int)(c & 511u) / OR_SLOTCAP, (int)(c & 511u) % OR_SLOTCAP), zs);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// dimuons (K:2820-3090, H:1269-1477), in float as there

struct SwimPt {
    float x, y, z, mx, my, mz;
};

__device__ __forceinline__ float E4(float m, const float *p) { return sqrtf(m * m + p[0] * p[0] + p[1] * p[1] + p[2] * p[2]); }
__device__ __forceinline__ float mult4(const float *a, const float *b) {
    return a[3] * b[3] - (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]);
}

// start of a track's swim (K:2927-2947)
__device__ __forceinline__ SwimPt dim_start(const float *T, const float *z, float &ty, float &charge) {
    using namespace phys;
    const float x0 = T[OR_TRK_X0], y0 = T[OR_TRK_Y0], tx = T[OR_TRK_TX];
    ty = T[OR_TRK_TY];
    const float invP = T[OR_TRK_INVP];
    charge = T[OR_TRK_CHARGE];
    const short detid_first = first_hit_detid(T, z);
    float x0_st1, tx_st1;
    x0_tx_st1(x0, tx, invP, (short)charge, x0_st1, tx_st1);
    const float z_0 = z[detid_first];
    const float s0 = charge * invP * sqrtf((1.f + tx_st1 * tx_st1) / (1.f + tx_st1 * tx_st1 + ty * ty));
    const float s1 = tx_st1, s2 = ty;
    const float s3 = z_0 * tx_st1 + x0_st1, s4 = z_0 * ty + y0;
    SwimPt p;
    p.x = (float)(s3 + s1 * (FMAG_LENGTH - z_0));
    p.y = (float)(s4 + s2 * (FMAG_LENGTH - z_0));
    p.z = (float)FMAG_LENGTH;
    const float pz_0 = 1.f / (fabsf(s0) * sqrtf(1.f + s1 * s1 + s2 * s2));
    p.mx = pz_0 * s1;
    p.my = pz_0 * s2;
    p.mz = pz_0;
    return p;
}

// Largest floats not above the hole's length and radius: for a float x,
// x > FMAG_HOLE_LENGTH (a double) exactly when x > this, without the FP64 pipe.
constexpr float HOLE_LENGTH_F = 0x1.bf0a3cp+4f, HOLE_RADIUS_F = 0x1.451eb8p+0f;
static_assert((double)HOLE_LENGTH_F <= phys::FMAG_HOLE_LENGTH && (double)0x1.bf0a3ep+4f > phys::FMAG_HOLE_LENGTH, "");
static_assert((double)HOLE_RADIUS_F <= phys::FMAG_HOLE_RADIUS && (double)0x1.451ebap+0f > phys::FMAG_HOLE_RADIUS, "");

// p(ptot) of the energy loss (dedx_poly with the linear coefficient d1)
__device__ __forceinline__ FF ff_dedx(float p, FF d1) {
    using namespace phys;
    constexpr FF d0 = ff_const(DEDX_UNIT_0), d2 = ff_const(DEDX_UNIT_2), d3 = ff_const(DEDX_UNIT_3),
                 d4 = ff_const(DEDX_UNIT_4);
    FF a = ff_add(ff_mul(d4, p), d3);
    a = ff_add(ff_mul(a, p), d2);
    a = ff_add(ff_mul(a, p), d1);
    return ff_add(ff_mul(a, p), d0);
}

// the double statements themselves, as calls (see slow_sqrt)
__device__ __noinline__ float slow_energy(float ptot, float len, double d1) {
    using namespace phys;
    return (float)(ptot + (DEDX_UNIT_0 + d1 * ptot + DEDX_UNIT_2 * ptot * ptot + DEDX_UNIT_3 * ptot * ptot * ptot +
                           DEDX_UNIT_4 * ptot * ptot * ptot * ptot) *
                              len);
}
__device__ __noinline__ float slow_step(float t) { return (float)(t * phys::STEP_FMAG); }
__device__ __noinline__ float slow_kick(float tx, double kick, float len) { return (float)(tx + kick / len); }

// (float)(ptot + p(ptot) * len) as the reference rounds it
__device__ __forceinline__ float dim_energy(float ptot, float len, FF d1f, bool &sure) {
    const FF v = ff_add(ff_mul(ff_dedx(ptot, d1f), len), FF{ptot, 0.f});
    // up to these bounds the loss stays well below ptot, and the polynomial's
    // terms below 2^6
    sure = (ptot < 1000.f) & (len < 16.f) & ff_sure(v);
    return v.h;
}

// (float)(t * STEP_FMAG)
__device__ __forceinline__ float dim_step(float t, bool &sure) {
    const FF v = ff_mul(ff_const(phys::STEP_FMAG), t);
    sure = ff_sure(v);
    return v.h;
}

// (float)(tx + kick / len)
__device__ __forceinline__ float dim_kick(float tx, FF kf, float len, bool &sure) {
    const float q = kf.h / len;
    const FF s = ff_sum(tx, q);
    const FF v = ff_fast(s.h, s.l + (__fmaf_rn(-q, len, kf.h) + kf.l) / len);
    // (a sum that all but cancels keeps the quotient's error)
    sure = (fabsf(v.h) > 0x1p-8f * fabsf(q)) & ff_sure(v);
    return v.h;
}

// What a track's steps have in common.
struct DimTrack {
    float ty, t1;          // t1 = (float)(ty * STEP_FMAG)
    double kick, d1;       // d1 = the linear energy-loss coefficient of the first update, DEDX_UNIT_2 for the
    FF kickf, d1f;         // reference's second track (H:1354)
};

// one FMag step (H:1290-1333)
__device__ __forceinline__ void dim_fmag_step(SwimPt &s, const DimTrack &k) {
    using namespace phys;
    // what depends on the same values side by side, then one branch for the
    // lanes that need the double statements
    const float t2 = (float)STEP_FMAG;
    bool ok1, ok2;
    const float tx_i = s.mx / s.mz, pxz = sqrtf(s.mx * s.mx + s.mz * s.mz);
    const float ptot_i = sqrtf(s.mx * s.mx + s.my * s.my + s.mz * s.mz);
    float tx_f = dim_kick(tx_i, k.kickf, pxz, ok1), t10 = dim_step(tx_i, ok2);
    if (!(ok1 & ok2)) {
        if (!ok1) tx_f = slow_kick(tx_i, k.kick, pxz);
        if (!ok2) t10 = slow_step(tx_i);
    }
    const float b0 = s.x - t10, b1 = s.y - k.t1, b2 = s.z - t2;
    const float len1 = sqrtf(t10 * t10 + k.t1 * k.t1 + t2 * t2);
    float t20 = dim_step(tx_f, ok1), ptot_b = dim_energy(ptot_i, len1, k.d1f, ok2);
    const bool in1 = b2 > HOLE_LENGTH_F || b0 * b0 + b1 * b1 > HOLE_RADIUS_F;
    if (!(ok1 & (ok2 | !in1))) {
        if (!ok1) t20 = slow_step(tx_f);
        if (!ok2) ptot_b = slow_energy(ptot_i, len1, k.d1);
    }
    if (!in1) ptot_b = ptot_i;
    s.x = b0 - t20;
    s.y = b1 - k.t1;
    s.z = b2 - t2;
    const float len2 = sqrtf(t20 * t20 + k.t1 * k.t1 + t2 * t2);
    float ptot_f = dim_energy(ptot_b, len2, ff_const(DEDX_UNIT_1), ok1);
    const bool in2 = s.z > HOLE_LENGTH_F || s.x * s.x + s.y * s.y > HOLE_RADIUS_F;
    if (!ok1 & in2) ptot_f = slow_energy(ptot_b, len2, DEDX_UNIT_1);
    if (!in2) ptot_f = ptot_b;
    const float pz_f = ptot_f / sqrtf(1.f + tx_f * tx_f + k.ty * k.ty);
    s.mx = pz_f * tx_f;
    s.my = pz_f * k.ty;
    s.mz = pz_f;
}

// H:1395-1408; a float times 5.0 rounds once, in float or in double
static_assert(phys::STEP_TARGET == 5.0, "");
__device__ __forceinline__ void dim_target_step(SwimPt &s, float tx_i, float t1) {
    s.x = s.x - tx_i * 5.f;
    s.y = s.y - t1;
    s.z = s.z - 5.f;
}

// a pair's two swims, one per lane, and the point of closest approach
// (FindDimuonClosestApproach, H:1269-1477)
struct SwimResult {
    float b[6];       // x, y, z, mx, my, mz at the closest approach
    float z66;        // z of step 66: element 200 of the reference's flat arrays (H:1447-1449)
    float single[6];  // momentum and vertex of the track as vertexed
    int found;
};

// Both lanes of a pair (lane, lane ^ 1) call this with their own track; d1 =
// the linear energy-loss coefficient of the first update of a step.
__device__ __noinline__ void pair_swim(SwimPt s, float charge, float ty, double d1, SwimResult &o) {
    using namespace phys;
    DimTrack k;
    k.ty = ty;
    k.t1 = (float)(ty * STEP_FMAG);
    k.kick = 2.f * charge * PTKICK_UNIT * STEP_FMAG;
    k.kickf = FF{(float)k.kick, (float)(k.kick - (double)(float)k.kick)};
    k.d1 = d1;
    k.d1f = FF{(float)d1, (float)(d1 - (double)(float)d1)};
    float tx_t = 0.f;  // the slope in the target steps, which keep the momentum
    float dca2_min = 1.e18f;
    SwimPt b = s;
    int found = 0;
    float z66 = 0.f;
#pragma unroll 1
    for (int j = 0; j <= NSTEPS_FMAG + NSTEPS_TARGET; ++j) {
        if (j >= 1 && j <= NSTEPS_FMAG) {
            dim_fmag_step(s, k);
            if (j == NSTEPS_FMAG) tx_t = s.mx / s.mz;
        } else if (j > NSTEPS_FMAG) {
            dim_target_step(s, tx_t, ty * 5.f);
        }
        if (j == 66) z66 = s.z;
        const int away = FMAGSTR * charge * s.mx < 0.f;
        const float ox = __shfl_xor_sync(0xffffffffu, s.x, 1), oy = __shfl_xor_sync(0xffffffffu, s.y, 1);
        const int oaway = __shfl_xor_sync(0xffffffffu, away, 1);
        if (away && oaway) continue;
        const float dx = s.x - ox, dy = s.y - oy;  // squared: the same for both lanes
        const float dca2 = dx * dx + dy * dy;
        if (dca2 < dca2_min) {
            dca2_min = dca2;
            found = 1;
            b = s;
        }
    }
    o.b[0] = b.x; o.b[1] = b.y; o.b[2] = b.z;
    o.b[3] = b.mx; o.b[4] = b.my; o.b[5] = b.mz;
    o.z66 = z66;
    o.found = found;
}

// What the pair loop carries within an event.
struct DimState {
    float p_pos[4], p_neg[4], pos_v[3], neg_v[3];
    int ndim;
};

// One pair of the loop, with its swims (r1: the first track's, r2: the second
// track's); `fresh`: the first track is new to the loop.
__device__ __noinline__ void dim_pair(DimState &S, bool fresh, float qi, float qj, const SwimResult &r1,
                                      const SwimResult &r2, float c1, float *__restrict__ out) {
    using namespace phys;
    float *p_pos = S.p_pos, *p_neg = S.p_neg, *pos_v = S.pos_v, *neg_v = S.neg_v;
    const float p_beam[4] = {0, 0, PBEAM, EBEAM};
    const float p_target[4] = {0, 0, 0, MP};
    const float p_cms[4] = {0, 0, PBEAM, EBEAM + MP};
    const float s = p_cms[3] * p_cms[3] - (p_cms[0] * p_cms[0] + p_cms[1] * p_cms[1] + p_cms[2] * p_cms[2]);
    const float sqrt_s = sqrtf(s);
    const float cms_bz = p_cms[2] / p_cms[3];
    if (fresh) {
        float *pv = qi > 0 ? p_pos : p_neg, *vv = qi > 0 ? pos_v : neg_v;
        for (int k = 0; k < 3; ++k) {
            pv[k] = r1.single[k];
            vv[k] = r1.single[3 + k];
        }
        pv[3] = E4(MMU, pv);
    }
    {
        float *qv = qj > 0 ? p_pos : p_neg, *wv = qj > 0 ? pos_v : neg_v;
        for (int k = 0; k < 3; ++k) {
            qv[k] = r2.single[k];
            wv[k] = r2.single[3 + k];
        }
        qv[3] = E4(MMU, qv);
    }
    float p_pos_single[4], p_neg_single[4], v_1[3], v_2[3], dim_v[3], p_sum[4];
    for (int k = 0; k < 4; ++k) {
        p_pos_single[k] = p_pos[k];
        p_neg_single[k] = p_neg[k];
    }
    for (int k = 0; k < 3; ++k) v_1[k] = (pos_v[k] + neg_v[k]) * 0.5f;
    float vz_2;
    if (!r1.found) {
        const float m = (float)((r1.z66 + r2.z66) * 0.5);
        v_2[0] = v_2[1] = v_2[2] = m;
        vz_2 = Z_DUMP;
    } else {
        const float *bp = c1 > 0 ? r1.b : r2.b, *bn = c1 > 0 ? r2.b : r1.b;
        for (int k = 0; k < 3; ++k) {
            p_pos[k] = bp[3 + k];
            p_neg[k] = bn[3 + k];
            v_2[k] = (float)((r1.b[k] + r2.b[k]) * 0.5);
        }
        vz_2 = r1.b[2];
    }
    p_pos[3] = E4(MMU, p_pos);
    p_neg[3] = E4(MMU, p_neg);
    if (fabsf(vz_2 - v_2[2]) < STEP_FMAG) {
        for (int k = 0; k < 4; ++k) p_sum[k] = p_pos[k] + p_neg[k];
        for (int k = 0; k < 3; ++k) dim_v[k] = v_2[k];
    } else {
        for (int k = 0; k < 4; ++k) p_sum[k] = p_pos_single[k] + p_neg_single[k];
        for (int k = 0; k < 3; ++k) dim_v[k] = v_1[k];
    }
    const float m = sqrtf(p_sum[3] * p_sum[3] - (p_sum[0] * p_sum[0] + p_sum[1] * p_sum[1] + p_sum[2] * p_sum[2]));
    const float pT = sqrtf(p_sum[0] * p_sum[0] + p_sum[1] * p_sum[1]);
    const float x1 = mult4(p_target, p_sum) / mult4(p_target, p_cms);
    const float x2 = mult4(p_beam, p_sum) / mult4(p_beam, p_cms);
    {  // Boost(p_sum, cms_bv, -1), H:1245-1267
        const float bx = 0.0f * -1, by = 0.0f * -1, bz = cms_bz * -1;
        const float b2 = bx * bx + by * by + bz * bz;
        const float gamma = 1.0f / sqrtf(1.0f - b2);
        const float bp = p_sum[0] * bx + p_sum[1] * by + p_sum[2] * bz;
        const float gamma2 = b2 > 0.0f ? (gamma - 1.0f) / b2 : 0.0f;
        p_sum[0] = p_sum[0] + gamma2 * bp * bx + gamma * bx * p_sum[3];
        p_sum[1] = p_sum[1] + gamma2 * bp * by + gamma * by * p_sum[3];
        p_sum[2] = p_sum[2] + gamma2 * bp * bz + gamma * bz * p_sum[3];
        p_sum[3] = gamma * (p_sum[3] + bp);
    }
    const float xF = 2.0f * p_sum[2] / (sqrt_s * (1.f - m * m / s));
    const float costheta = 2 * (p_neg[3] * p_pos[2] - p_neg[2] * p_pos[3]) / (m * sqrtf(m * m + pT * pT));
    const float phi = atan2f(2 * sqrtf(m * m + pT * pT) * (p_neg[0] * p_pos[1] - p_neg[1] * p_pos[0]),
                             m * (p_pos[0] * p_pos[0] - p_neg[0] * p_neg[0] + p_pos[1] * p_pos[1] - p_neg[1] * p_neg[1]));
    // K:3028-3042
    if (FMAGSTR * (p_pos[0] - p_neg[0]) < 0.) return;
    if (m < 0 || m > 10.f) return;
    if (fabsf(xF) > 1.f) return;
    if (x1 < 0.f || x1 > 1.f) return;
    if (x2 < 0.f || x2 > 1.f) return;
    if (fabsf(costheta) > 1.f) return;
    if (p_pos[2] + p_neg[2] > 120.f || p_pos[2] + p_neg[2] < 30.f) return;
    if (fabsf(p_pos[0] + p_neg[0]) > 3.f) return;
    if (dim_v[0] * dim_v[0] + dim_v[1] * dim_v[1] > 225.f) return;
    // the reference writes a 17th record past its event's 16 (K:3059); the
    // event's 16 records are the limit here
    if (S.ndim >= OR_DIMUON_MAX) return;
    float *D = out + (size_t)S.ndim * OR_NDIMUONPARAM;
    D[OR_DIM_MASS] = m;
    D[OR_DIM_PT] = pT;
    D[OR_DIM_XF] = xF;
    D[OR_DIM_X1] = x1;
    D[OR_DIM_X2] = x2;
    D[OR_DIM_COSTHETA] = costheta;
    D[OR_DIM_PHI] = phi;
    D[OR_DIM_MASS_SINGLE] = 0.f;
    D[OR_DIM_CHI2_SINGLE] = 0.f;
    for (int k = 0; k < 3; ++k) {
        D[OR_DIM_VTX + k] = dim_v[k];
        D[OR_DIM_POS_VTX + k] = pos_v[k];
        D[OR_DIM_NEG_VTX + k] = neg_v[k];
    }
    for (int k = 0; k < 4; ++k) {
        D[OR_DIM_POS_P + k] = p_pos[k];
        D[OR_DIM_NEG_P + k] = p_neg[k];
        D[OR_DIM_POS_P_SINGLE + k] = p_pos_single[k];
        D[OR_DIM_NEG_P_SINGLE + k] = p_neg_single[k];
    }
    D[OR_DIM_CHI2_VTX] = 0.f;
    D[OR_DIM_CHI2_KF] = 0.f;
    ++S.ndim;
}

#ifndef OR_DIM_GROUP
#define OR_DIM_GROUP 16
#endif
constexpr int DIM_LIST = 1024;   // vertexed tracks a warp lists at a time
constexpr int DIM_PAIRS = 16;    // pairs swum at a time, two lanes each
static_assert(OR_DIM_GROUP <= 32 && DIM_LIST >= OR_TRKMAX, "lane = event; one event's tracks fit");

// One warp per block, as in vertexing: the FP64 pipe bounds the energy-loss
// terms, so the warps spread over the SMs first.  The vertexed tracks of the
// warp's events are listed in (slot, position) order; lane e then goes
// through event e's pairs in the reference's order (i_trd, j_trd >= i_trd, i,
// j; opposite charges), sixteen pairs over the events at a time being swum
// by the whole warp.  A thread per event swimming its pairs one after the
// other, both tracks in turn, in blocks of 128 took 947 us for 10,000 events
// and for 2,000; this takes 117 and 106 us.  The events' flags and counts are
// read side by side, so that a batch with nothing to do costs what its reads
// do (3,000 events without tracks 17 us with each event's after the last's, 11
// us so).
__global__ void __launch_bounds__(32)
    dimuon_kernel(const or_plane_t *__restrict__ gplane, or_tracks_view_t tv, or_dimuons_view_t dv,
                  const uint8_t *__restrict__ toomany, int n_events, int group) {
    using namespace phys;
    __shared__ float zs[OR_NDET];
    __shared__ uint16_t code[DIM_LIST];  // slot * 16 + position
    __shared__ float chg[DIM_LIST];
    __shared__ SwimResult res[DIM_PAIRS][2];
    __shared__ float c1s[DIM_PAIRS];
    __shared__ int2 pairs[DIM_PAIRS];  // event << 16 | first track, second track (list entries)
    const int lane = threadIdx.x;
    const unsigned lt = lanemask_lt();
    for (int i = lane; i < OR_NDET; i += 32) zs[i] = gplane->z[i];
    for (long g0 = (long)blockIdx.x * group; g0 < n_events; g0 += (long)gridDim.x * group) {
        const int ng = (int)min((long)group, n_events - g0);
        const unsigned live = __ballot_sync(0xffffffffu, lane < ng && !toomany[g0 + min(lane, ng - 1)]);
        if (!live) continue;
        for (int ev0 = 0; ev0 < ng;) {
            // --- list the vertexed tracks of events ev0 .. ev1 that fit --------
            __syncwarp();
            int listed = 0, ev1 = ev0, first = 0, last = 0;  // the lane's event: entries [first, last)
            for (bool fits = true; fits && ev1 < ng;) {
                int n[8];  // eight events' counts in flight
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    n[i] = ev1 + i < ng && ((live >> (ev1 + i)) & 1u)
                               ? min((int)tv.ntracks[(g0 + ev1 + i) * OR_NSLOTS + lane], OR_SLOTCAP)
                               : 0;
#pragma unroll 1
                for (int i = 0; i < 8 && ev1 < ng; ++i, ++ev1) {
                    const long e = g0 + ev1;
                    int c = 0, ne = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k == i) ne = n[k];
                    int tot = 0, incl = 0;
                    if (__any_sync(0xffffffffu, ne > 0)) {
                        unsigned mask = 0u;
#pragma unroll 4
                        for (int k = 0; k < ne; ++k)
                            if (trk_rec(tv, e, lane, k)[OR_TRK_STID] >= 7) mask |= 1u << k;
                        c = __popc(mask);
                        incl = c;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int v = __shfl_up_sync(0xffffffffu, incl, o);
                            if (lane >= o) incl += v;
                        }
                        tot = __shfl_sync(0xffffffffu, incl, 31);
                        if (listed + tot > DIM_LIST) {
                            fits = false;
                            break;
                        }
                        int at = listed + incl - c;
                        for (unsigned m = mask; m; m &= m - 1) {
                            const int k = __ffs(m) - 1;
                            code[at] = (uint16_t)(lane * OR_SLOTCAP + k);
                            chg[at] = trk_rec(tv, e, lane, k)[OR_TRK_CHARGE];
                            ++at;
                        }
                    }
                    if (lane == ev1) {
                        first = listed;
                        last = listed + tot;
                    }
                    listed += tot;
                }
            }
            __syncwarp();
            // --- the pair loop of the lane's event ------------------------------
            const bool own = lane >= ev0 && lane < ev1;
            const long e = g0 + lane;
            DimState S;
            for (int k = 0; k < 4; ++k) S.p_pos[k] = S.p_neg[k] = 0.f;
            for (int k = 0; k < 3; ++k) S.pos_v[k] = S.neg_v[k] = 0.f;
            S.ndim = 0;
            // slot groups [a0, a1) of the first and [b0, b1) of the second track
            auto group_end = [&](int i) {
                const int sl = code[i] / OR_SLOTCAP;
                while (i < last && code[i] / OR_SLOTCAP == sl) ++i;
                return i;
            };
            int a0 = first, a1 = own && first < last ? group_end(first) : first;
            int b0 = a0, b1 = a1, i = a0, j = b0;
            bool busy = own && first < last, fresh = true;
            // A first track without a pair leaves nothing behind, unless a
            // charge is neither positive nor negative: then its momentum may
            // stand where the next pair's second track does not overwrite it.
            bool odd = false;
            for (int k = first; own && k < last; ++k) odd |= !(chg[k] > 0 || chg[k] < 0);
            while (listed) {
                // the lane's next pair
                bool have = false;
                while (busy) {
                    if (j == b1) {  // next first track of the group, with the same second group
                        if (odd && fresh) {
                            const float *T = trk_rec(tv, e, code[i] / OR_SLOTCAP, code[i] % OR_SLOTCAP);
                            float *pv = chg[i] > 0 ? S.p_pos : S.p_neg, *vv = chg[i] > 0 ? S.pos_v : S.neg_v;
                            for (int k = 0; k < 3; ++k) {
                                pv[k] = T[OR_TRK_PX + k];
                                vv[k] = T[OR_TRK_VX + k];
                            }
                            pv[3] = E4(MMU, pv);
                        }
                        ++i;
                        fresh = true;
                        j = b0;
                        if (i == a1) {
                            if (b1 < last) {  // next second group
                                b0 = b1;
                                b1 = group_end(b0);
                            } else if (a1 < last) {  // next first group
                                a0 = a1;
                                a1 = group_end(a0);
                                b0 = a0;
                                b1 = a1;
                            } else {
                                busy = false;
                                break;
                            }
                            i = a0;
                            j = b0;
                        }
                        continue;
                    }
                    if (!(chg[j] * chg[i] > 0)) {
                        have = true;
                        break;
                    }
                    ++j;
                }
                const unsigned hm = __ballot_sync(0xffffffffu, have);
                if (!hm) break;
                // up to sixteen of them, in lane order
                const int at = __popc(hm & lt);
                const bool take = have && at < DIM_PAIRS;
                if (take) pairs[at] = make_int2(lane << 16 | i, j);
                __syncwarp();
                const int np = min(__popc(hm), DIM_PAIRS);
                {
                    const int p = min(lane >> 1, np - 1);
                    const int2 pr = pairs[p];
                    const int c = code[(lane & 1) ? pr.y : pr.x & 0xFFFF];
                    const float *T = trk_rec(tv, g0 + (pr.x >> 16), c / OR_SLOTCAP, c % OR_SLOTCAP);
                    SwimResult o;
                    for (int k = 0; k < 3; ++k) {
                        o.single[k] = T[OR_TRK_PX + k];
                        o.single[3 + k] = T[OR_TRK_VX + k];
                    }
                    float ty, ch;
                    const SwimPt s = dim_start(T, zs, ty, ch);
                    pair_swim(s, ch, ty, (lane & 1) ? DEDX_UNIT_2 : DEDX_UNIT_1, o);
                    if ((lane >> 1) < np) {
                        res[p][lane & 1] = o;
                        if (!(lane & 1)) c1s[p] = ch;
                    }
                }
                __syncwarp();
                if (take) {
                    dim_pair(S, fresh, chg[i], chg[j], res[at][0], res[at][1], c1s[at],
                             dv.dimuons + (size_t)e * OR_EVT_DIM_FLOATS);
                    fresh = false;
                    ++j;
                }
                __syncwarp();
            }
            if (own && ((live >> lane) & 1u)) dv.ndimuons[e] = (uint16_t)S.ndim;
            ev0 = ev1;
        }
    }
}

// ---------------------------------------------------------------------------
// histograms (K:3100-3195)

// Count v in table i: every bin j with x[j] - h <= v < x[j] + h.  With the
// centres in order both tests are monotone in j, so the bins that hold v
// follow the first one whose upper edge lies above it; a table out of order
// is gone through whole.
__device__ __forceinline__ void hist_add(or_hists_t *H, int i, int nb, float h, bool sorted, float v) {
    const float *xp = H->xpts + (size_t)i * OR_HIST_NBINS_MAX;
    float *val = H->values + (size_t)i * OR_HIST_NBINS_MAX;
    int j = 0;
    if (sorted) {
        int hi = nb;
        while (j < hi) {
            const int mid = (j + hi) >> 1;
            if (v < __ldg(xp + mid) + h) hi = mid;
            else j = mid + 1;
        }
    }
    for (; j < nb; ++j) {
        const float x = __ldg(xp + j);
        const bool below = x - h <= v;
        if (below && v < x + h) atomicAdd(val + j, 1.f);
        else if (sorted && !below) break;
    }
}

__device__ __constant__ unsigned char c_hist_dim[12] = {OR_DIM_MASS, OR_DIM_XF,    OR_DIM_X1,     OR_DIM_X2,
                                                        OR_DIM_PT,   OR_DIM_PHI,   OR_DIM_POS_P,  OR_DIM_POS_P + 1,
                                                        OR_DIM_POS_P + 2, OR_DIM_VTX, OR_DIM_VTX + 1, OR_DIM_VTX + 2};

// A warp per event; its lanes take (variable, trigger) pairs of a track or a
// dimuon, and each searches its table.  Bound: the search's L1 latency and
// the atomics.  With the lanes over the bins of one table at a time, every
// table of every value was read whole: 151 us for 10,000 one-dimuon events;
// this takes 35 us.
template <int W>
__global__ void __launch_bounds__(W * 32)
    hist_kernel(or_tracks_view_t tv, or_dimuons_view_t dv, const int32_t *__restrict__ trigger_bits,
                const uint8_t *__restrict__ toomany, or_hists_t *H, int n_events) {
    constexpr int NT = OR_HIST_NTRIGGERS * OR_HIST_NVARS;
    __shared__ int16_t nbins[NT];
    __shared__ float hw[NT];
    __shared__ uint8_t ordered[NT];
    __shared__ uint8_t trig[W][OR_HIST_NTRIGGERS];  // the event's trigger classes
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < NT; i += blockDim.x) {
        nbins[i] = min((int)H->nbins[i], OR_HIST_NBINS_MAX);
        hw[i] = H->pts_hw[i];
    }
    // the tables' order is looked at by blocks that may have something to
    // count: some event of theirs has tracks or dimuons (3,000 rejected events
    // 21 -> 8 us)
    bool some = false;
    for (long e = (long)blockIdx.x * W + w; e < n_events && !some; e += (long)gridDim.x * W)
        if (!toomany[e]) some = __any_sync(0xffffffffu, tv.ntracks[e * OR_NSLOTS + lane] != 0 || dv.ndimuons[e] != 0);
    if (!__syncthreads_or(some)) return;
    for (int i = w; i < NT; i += W) {
        const float *xp = H->xpts + (size_t)i * OR_HIST_NBINS_MAX;
        bool ok = true;
#pragma unroll 4
        for (int j = lane; j + 1 < nbins[i]; j += 32) ok &= xp[j] <= xp[j + 1];
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) ordered[i] = ok;
    }
    __syncthreads();
    for (long e = (long)blockIdx.x * W + w; e < n_events; e += (long)gridDim.x * W) {
        if (toomany[e]) continue;
        const int tb = trigger_bits ? trigger_bits[e] : 0;
        // K:3108: the bit test the reference makes; the last class is "all triggers" (K:3110)
        const bool in = lane < OR_HIST_NTRIGGERS && (lane == OR_HIST_NTRIGGERS - 1 || (tb & lane));
        const unsigned tmask = __ballot_sync(0xffffffffu, in);
        const int nt = __popc(tmask);
        __syncwarp();  // every lane is done with the previous event's classes
        if (in) trig[w][__popc(tmask & lanemask_lt())] = (uint8_t)lane;
        __syncwarp();
        auto add = [&](int q, int k0, float v) {
            const int i = trig[w][q % nt] * OR_HIST_NVARS + k0 + q / nt;
            hist_add(H, i, nbins[i], hw[i], ordered[i], v);
        };
        const int nslot = min((int)tv.ntracks[e * OR_NSLOTS + lane], OR_SLOTCAP);
        const int most = __reduce_max_sync(0xffffffffu, nslot);
#pragma unroll 1
        for (int k = 0; k < most; ++k) {
            bool take = false;
            if (k < nslot) {
                const float *T = trk_rec(tv, e, lane, k);
                take = !(T[OR_TRK_STID] < 7 || T[OR_TRK_CHI2] / (T[OR_TRK_NHITS] - 5) > phys::CHI2DOF_MAX);
            }
            for (unsigned m = __ballot_sync(0xffffffffu, take); m; m &= m - 1) {
                const float *T = trk_rec(tv, e, __ffs(m) - 1, k);
                for (int q = lane; q < OR_HIST_NVARS_TRACKS * nt; q += 32) {
                    const int v = q / nt;
                    add(q, 0, T[v < 3 ? OR_TRK_PX + v : OR_TRK_VX + v - 3]);
                }
            }
        }
        const int nd = min((int)dv.ndimuons[e], OR_DIMUON_MAX);
        for (int i = 0; i < nd; ++i) {
            const float *D = dv.dimuons + (size_t)e * OR_EVT_DIM_FLOATS + (size_t)i * OR_NDIMUONPARAM;
            for (int q = lane; q < 12 * nt; q += 32) {
                const int v = q / nt, f = c_hist_dim[v];
                const float x = D[f];
                add(q, OR_HIST_NVARS_TRACKS, v >= 6 && v < 9 ? x + D[f + OR_DIM_NEG_P - OR_DIM_POS_P] : x);
            }
        }
    }
}

// ---------------------------------------------------------------------------

cudaError_t launch_vertexing(const or_plane_t *d_plane, or_tracks_view_t tv, const uint8_t *toomany, int n_events,
                             cudaStream_t stream, int sm_count) {
    if (n_events <= 0) return cudaSuccess;
    // events per warp: a warp to each quarter of an SM first, and at most
    // OR_VTX_GROUP events, whose tracks fill about one warp (2,000 events, 2 /
    // 4 / 8 / 13 events a warp: 300 / 244 / 253 / 274 us; 10,000 events, 4 / 8
    // / 16 / 32: 764 / 455 / 332 / 559 us)
    const int group = std::max(1, std::min(OR_VTX_GROUP, (n_events + 4 * sm_count - 1) / (4 * sm_count)));
    const long blocks = std::min(((long)n_events + group - 1) / group, (long)sm_count * 32);
    vertex_kernel<<<(unsigned)blocks, 32, 0, stream>>>(d_plane, tv, toomany, n_events, group);
    return cudaGetLastError();
}

cudaError_t launch_dimuons(const or_plane_t *d_plane, or_tracks_view_t tv, or_dimuons_view_t dv,
                           const uint8_t *toomany, int n_events, cudaStream_t stream, int sm_count) {
    if (n_events <= 0) return cudaSuccess;
    // a warp per SM first, then up to OR_DIM_GROUP events per warp
    const int group = std::max(1, std::min(OR_DIM_GROUP, n_events / sm_count));
    const long blocks = std::min(((long)n_events + group - 1) / group, (long)sm_count * 32);
    dimuon_kernel<<<(unsigned)blocks, 32, 0, stream>>>(d_plane, tv, dv, toomany, n_events, group);
    return cudaGetLastError();
}

cudaError_t launch_histograms(or_tracks_view_t tv, or_dimuons_view_t dv, const int32_t *trigger_bits,
                              const uint8_t *toomany, or_hists_t *d_hists, int n_events, cudaStream_t stream,
                              int sm_count) {
    if (n_events <= 0) return cudaSuccess;
    // two blocks an SM: each checks the tables' order once (80 KB)
    constexpr int W = 16;
    long blocks = ((long)n_events + W - 1) / W;
    blocks = min(blocks, (long)sm_count * 2);
    hist_kernel<W><<<(unsigned)blocks, W * 32, 0, stream>>>(tv, dv, trigger_bits, toomany, d_hists, n_events);
    return cudaGetLastError();
}

}  // namespace orgpu
