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
//    here a warp gathers the global tracks of 32 events into a shared list
//    and swims them one per lane, which keeps the lanes of the double-
//    precision loop busy (FP64 is the scarce unit of this GPU).  The swim is
//    not stored: the closest-approach scan visits the points in step order
//    with a strict "smaller than" test, so it runs as the points are made.
//  - Dimuons: the two swims of a pair depend on its tracks alone and are made
//    by two lanes side by side; the pairs of an event are then gone through in
//    order by its own lane, as the reference's pair loop carries state from
//    one pair to the next (the swum momenta of the current track stay in
//    p_pos / p_neg).
//  - Histograms: one warp per event, lanes over the bins of one (trigger,
//    variable) table; counts go in with atomics, so the result is the exact
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
    double px = s3 + s1 * (FMAG_LENGTH - z_0), py = s4 + s2 * (FMAG_LENGTH - z_0), pz = FMAG_LENGTH;
    const double pz_0 = 1.f / (fabs(s0) * sqrtf(1.f + s1 * s1 + s2 * s2));
    double mx = pz_0 * s1, my = pz_0 * s2, mz = pz_0;
    double dca2_min = 1.e18;
    bool found = false;
    double v[6];
    auto visit = [&]() {
        if (!(FMAGSTR * charge * mx < 0.)) {
            const double dca2 = (px - X_BEAM) * (px - X_BEAM) + (py - Y_BEAM) * (py - Y_BEAM);
            if (dca2 < dca2_min) {
                dca2_min = dca2;
                found = true;
                v[0] = px; v[1] = py; v[2] = pz;
                v[3] = mx; v[4] = my; v[5] = mz;
            }
        }
    };
    visit();
    for (int step = 1; step <= NSTEPS_FMAG; ++step) {
        const double tx_i = mx / mz;
        const double tx_f = tx_i + 2.f * charge * PTKICK_UNIT * STEP_FMAG / sqrt(mx * mx + mz * mz);
        const double t10 = tx_i * STEP_FMAG, t11 = ty * STEP_FMAG, t12 = STEP_FMAG;
        const double b0 = px - t10, b1 = py - t11, b2 = pz - t12;
        const double ptot_i = sqrt(mx * mx + my * my + mz * mz);
        double ptot_b = ptot_i;
        if (b2 > FMAG_HOLE_LENGTH || b0 * b0 + b1 * b1 > FMAG_HOLE_RADIUS)
            ptot_b += dedx_poly(ptot_i) * sqrtf(t10 * t10 + t11 * t11 + t12 * t12);
        const double t20 = tx_f * STEP_FMAG, t21 = ty * STEP_FMAG, t22 = STEP_FMAG;
        px = b0 - t20;
        py = b1 - t21;
        pz = b2 - t22;
        double ptot_f = ptot_b;
        if (pz > FMAG_HOLE_LENGTH || px * px + py * py > FMAG_HOLE_RADIUS)
            ptot_f += dedx_poly(ptot_b) * sqrtf(t20 * t20 + t21 * t21 + t22 * t22);
        const double pz_f = ptot_f / sqrt(1.f + tx_f * tx_f + ty * ty);
        mx = pz_f * tx_f;
        my = pz_f * ty;
        mz = pz_f;
        visit();
    }
    for (int step = NSTEPS_FMAG + 1; step <= NSTEPS_FMAG + NSTEPS_TARGET; ++step) {
        const double tx_i = mx / mz;
        px = px - tx_i * STEP_TARGET;
        py = py - ty * STEP_TARGET;
        pz = pz - STEP_TARGET;
        visit();
    }
    if (!found) {  // the last point (K:2752)
        v[0] = px; v[1] = py; v[2] = pz;
        v[3] = mx; v[4] = my; v[5] = mz;
    }
    T[OR_TRK_STID] = 7.f;  // K:2796
    T[OR_TRK_VX] = (float)v[0];
    T[OR_TRK_VX + 1] = (float)v[1];
    T[OR_TRK_VX + 2] = (float)v[2];
    T[OR_TRK_PX] = (float)v[3];
    T[OR_TRK_PX + 1] = (float)v[4];
    T[OR_TRK_PX + 2] = (float)v[5];
}

// One warp per block, so that the warps spread over the SMs before they
// share one: the swim is bound by the FP64 pipes, one to each quarter of an
// SM (a warp's swim takes some 460 us of one, whatever its lanes), and
// blocks of four warps left half of the SMs idle (10,000 events: 1,016 us;
// now 652 us, 2,000 events 1,012 -> 463 us).  A warp gathers the
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
        int waiting = 0;
        for (long eb = e0; eb < e1; eb += 8) {  // eight events' counts and stationIDs in flight
            int n[8], most = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                n[i] = eb + i < e1 && !toomany[eb + i] ? min((int)tv.ntracks[(eb + i) * OR_NSLOTS + lane], OR_SLOTCAP) : 0;
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

// one FMag step (H:1290-1333); d1 = the linear energy-loss coefficient of the
// first update, DEDX_UNIT_2 for the reference's second track (H:1354)
__device__ __forceinline__ void dim_fmag_step(SwimPt &s, float charge, float ty, double d1) {
    using namespace phys;
    const float tx_i = s.mx / s.mz;
    const float tx_f = (float)(tx_i + 2.f * charge * PTKICK_UNIT * STEP_FMAG / sqrtf(s.mx * s.mx + s.mz * s.mz));
    const float t10 = (float)(tx_i * STEP_FMAG), t11 = (float)(ty * STEP_FMAG), t12 = (float)STEP_FMAG;
    const float b0 = s.x - t10, b1 = s.y - t11, b2 = s.z - t12;
    const float ptot_i = sqrtf(s.mx * s.mx + s.my * s.my + s.mz * s.mz);
    float ptot_b = ptot_i;
    if (b2 > HOLE_LENGTH_F || b0 * b0 + b1 * b1 > HOLE_RADIUS_F)
        ptot_b = (float)(ptot_b + (DEDX_UNIT_0 + d1 * ptot_i + DEDX_UNIT_2 * ptot_i * ptot_i +
                                   DEDX_UNIT_3 * ptot_i * ptot_i * ptot_i + DEDX_UNIT_4 * ptot_i * ptot_i * ptot_i * ptot_i) *
                                      sqrtf(t10 * t10 + t11 * t11 + t12 * t12));
    const float t20 = (float)(tx_f * STEP_FMAG), t21 = (float)(ty * STEP_FMAG), t22 = (float)STEP_FMAG;
    s.x = b0 - t20;
    s.y = b1 - t21;
    s.z = b2 - t22;
    float ptot_f = ptot_b;
    if (s.z > HOLE_LENGTH_F || s.x * s.x + s.y * s.y > HOLE_RADIUS_F)
        ptot_f = (float)(ptot_f + dedx_poly(ptot_b) * sqrtf(t20 * t20 + t21 * t21 + t22 * t22));
    const float pz_f = ptot_f / sqrtf(1.f + tx_f * tx_f + ty * ty);
    s.mx = pz_f * tx_f;
    s.my = pz_f * ty;
    s.mz = pz_f;
}

__device__ __forceinline__ void dim_target_step(SwimPt &s, float ty) {  // H:1395-1408
    using namespace phys;
    const float tx_i = s.mx / s.mz;
    const float t0 = (float)(tx_i * STEP_TARGET), t1 = (float)(ty * STEP_TARGET), t2 = (float)STEP_TARGET;
    s.x = s.x - t0;
    s.y = s.y - t1;
    s.z = s.z - t2;
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
    float dca2_min = 1.e18f;
    SwimPt b = s;
    int found = 0;
    float z66 = 0.f;
#pragma unroll 1
    for (int j = 0; j <= NSTEPS_FMAG + NSTEPS_TARGET; ++j) {
        if (j >= 1 && j <= NSTEPS_FMAG) dim_fmag_step(s, charge, ty, d1);
        else if (j > NSTEPS_FMAG) dim_target_step(s, ty);
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
// and for 2,000; this takes 300 and 227 us.
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
        for (int ev0 = 0; ev0 < ng;) {
            // --- list the vertexed tracks of events ev0 .. ev1 that fit --------
            __syncwarp();
            int listed = 0, ev1 = ev0, first = 0, last = 0;  // the lane's event: entries [first, last)
            for (; ev1 < ng; ++ev1) {
                const long e = g0 + ev1;
                unsigned mask = 0u;
                if (!toomany[e]) {
                    const int n = min((int)tv.ntracks[e * OR_NSLOTS + lane], OR_SLOTCAP);
#pragma unroll 4
                    for (int k = 0; k < n; ++k)
                        if (trk_rec(tv, e, lane, k)[OR_TRK_STID] >= 7) mask |= 1u << k;
                }
                const int c = __popc(mask);
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                const int tot = __shfl_sync(0xffffffffu, incl, 31);
                if (listed + tot > DIM_LIST) break;
                int at = listed + incl - c;
                for (unsigned m = mask; m; m &= m - 1) {
                    const int k = __ffs(m) - 1;
                    code[at] = (uint16_t)(lane * OR_SLOTCAP + k);
                    chg[at] = trk_rec(tv, e, lane, k)[OR_TRK_CHARGE];
                    ++at;
                }
                if (lane == ev1) {
                    first = listed;
                    last = listed + tot;
                }
                listed += tot;
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
            for (;;) {
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
            if (own && !toomany[e]) dv.ndimuons[e] = (uint16_t)S.ndim;
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
// this takes 36 us.
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
    __syncthreads();
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
    // events per warp: a warp per SM first, and at most OR_VTX_GROUP events,
    // whose tracks fill about one warp
    const int group = std::max(1, std::min(OR_VTX_GROUP, n_events / sm_count));
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
