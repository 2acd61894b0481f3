// global_kernel.cu -- global tracking across KMag (station-1 extension).
//
// Replaces gKernel_Global_tracking<<<N,32>>> (OnlineReconstruction/
// reconstruction_kernels.cuh:1841-2534).
//
// Per YZ track (stationID >= 5) the reference finds station-1 x/u/v hit
// pairs in sagitta windows (reconstruction_helper.cuh:556-613), then for
// each x1 pair fits the x hits plus the KMag bend point, derives charge and
// 1/p (H:652-691), and for each (u1, v1) combination fits y with the
// station-2/3 u/v hits, resolves left/right, and keeps the best chi2.
// State carried by the reference, reproduced here:
//   - y0/ty are overwritten by every (u1,v1) fit and feed the next x1 pair's
//     x positions (K:2120, K:2370-2377);
//   - on the x' hit alone, the walk pairs it with the first u1 hit (planes
//     3/2) and re-sets its sign whenever that resolution succeeds;
//   - the scratch entry past the hit count (x part and uv part of the walk).
//
// A warp takes one slot; its tracks and their x1 pairs are in order.  The
// state between x1 pairs needs no (u1, v1) loop: whether a station-1 hit is
// accepted depends on the x1 pair and the hit alone, so the last combination
// that reaches the y fit is the last accepted v1 pair with the last accepted
// u1 pair, and the last writer of each scratch entry follows from the two
// lists in the same way (the end of gl_track's loop).  So
//   - the x fits of up to 32 x1 pairs are made at once, one per lane, up to
//     the first one inside the momentum window (only that one changes y0 and
//     ty);
//   - its station-1 hits are accepted once, one per lane;
//   - its (u1, v1) combinations then cost a few additions and the 2-sigma
//     cut, and those that pass wait in a ring, across x1 pairs, until 32 of
//     them can be walked and fitted with every lane in use (gl_pass).
//
// Bound: instruction fetch (a slot's track runs through some 80 KB of code
// once; with 99 KB two thirds of the warps' stalls were instruction misses),
// and the serial chain of one slot's tracks on small batches.  Evaluating
// each (u1, v1) combination with its hits' acceptance and the scratch
// entries' scan, 32 of one x1 pair at a time, took 13.7 ms for 100,000 uneven
// events and 1,223 us for 333 of them; this takes 8.4 ms and 385 us (11.8 ms
// with the windows and pairs walked plane by plane).
#include "window_pairs.cuh"

namespace orgpu {

constexpr int GL_PAIRCAP = 128;
constexpr unsigned GL_NONE = 0xFFFFu;

// A combination that passed the first y cut.
struct __align__(8) GlSurv {
    float xs0, xst, yc, tyc;
    // ix | x hits << 7 | x signs (2 bits each, two's complement) << 9 | v1 pair << 13 | x' alone << 20 | tries the
    // x', u1 pair << 21
    unsigned a;
    unsigned b;  // u1 pair | planes u1 u1' v1 v1' << 7 | scratch entry past the hit count << 16
};

struct GlWarp {
    GlSurv ring[64];
    // (eY * Y, eY * Y * z) of the u1 u1' hits in the windows for the current x1 pair, then of the v1 v1' hits
    float2 term[2 * GL_PAIRCAP];
    float2 bu[GL_PAIRCAP];       // accepted u1 pairs: the y fit's right-hand side after them
    HitPlane hc[6];              // station-1 plane views of the event
    unsigned char wl[6 * GL_PAIRCAP];  // hit index of each hit in the windows, list after list
    int woff[7];                       // where each list starts
    int start[6], np[3];
    unsigned short st[8];              // the slot's scratch entries 0..6: codes list << 12 | hit index
    float lo[3], hi[3];
    uchar2 pairs[3][GL_PAIRCAP];       // x1, u1, v1: positions in the lists (255 = none)
    unsigned short ua[GL_PAIRCAP];    // accepted u1 pairs: pair | planes << 7
    unsigned va[GL_PAIRCAP];          // accepted v1 pairs: pair | planes << 7 | latest earlier pair with two attempts << 16
    unsigned acc[2][2 * GL_PAIRCAP / 32];   // accepted u1 u1' hits, v1 v1' hits
    unsigned fl[6 * GL_PAIRCAP / 32];
    // station-2/3 hits of the current track
    float p1x[12], p1y[12], p1z[12], dpx[12], dpy[12], dpz[12], drift[12], res2[12];
    short sign[12];
    float Y[12], eY[12], Zy[12];
    // the current track's (u1, v1) y fit by plane set (gl_tab_entry)
    float tab[9][8];
    // best
    float b_chi2, b_ty, b_y0, b_xst, b_ety, b_ey0;
    int b_n;
    float b_det[6], b_el[6], b_pos[6], b_drift[6], b_sign[6], b_tdc[6], b_res[18];
};

// station-1 planes x x' u u' v v' (K:1880-1923, E1039 chamber ids)
__device__ __forceinline__ constexpr int gl_det(int l) {
    return l == 0 ? 4 : l == 1 ? 3 : l == 2 ? 2 : l == 3 ? 1 : l == 4 ? 6 : 5;
}

// The y fit of a (u1, v1) combination (K:2368-2379) adds the track's
// station-2/3 y hits and then the accepted u1 u1' v1 v1' hits, each with its
// plane's weight (calculate_y_uvhit's error, a plane constant) and z: its
// normal matrix, inverse and errors depend only on which station-1 planes
// gave a hit.  Entry (gu - 1) * 3 + gv - 1 (plane bits of the u1 and v1
// groups, 1..3) holds Fit2::solve's inverse A^-1 (4), the 2-sigma bounds of
// the first cut Y0_MAX + 2 err_y0, TY_MAX + 2 err_ty, and err_y0, err_ty --
// computed as Fit2 accumulates (the station-2/3 hits first, the station-1
// planes in attempt order), so a combination needs only its right-hand side.
__device__ __forceinline__ void gl_tab_entry(const float *eY, const float *Zy, int nyh, int gu, int gv,
                                             const or_plane_t &P, float *out) {
    Fit2 f;
#pragma unroll 1
    for (int k = 0; k < nyh; ++k) f.add(0.f, Zy[k], eY[k]);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (!((a < 2 ? gu >> a : gv >> (a - 2)) & 1)) continue;
        const int d = gl_det(a + 2);
        f.add(0.f, P.z[d], P.resolution[d] * fabsf(P.deltapy[d] / P.deltapx[d]));
    }
    const float A[4] = {f.A0, f.A1, f.A2, f.A3};
    float Ai[4];
    matinv_2x2(A, Ai);
    const float e0 = sqrtf(fabsf(Ai[0])), e1 = sqrtf(fabsf(Ai[3]));
    out[0] = Ai[0];
    out[1] = Ai[1];
    out[2] = Ai[2];
    out[3] = Ai[3];
    out[4] = Y0_MAX + 2 * e0;
    out[5] = TY_MAX + 2 * e1;
    out[6] = e0;
    out[7] = e1;
}

// SagittaRatioInStation1 (H:556-613) for plane pair i = 0..2: the expected
// position and half window of projection idx.
__device__ __forceinline__ void sagitta_st1(int i, float x0, float tx, float y0, float ty, int detid_lasthit, int &idx,
                                            float &pos_exp, float &window, const or_plane_t &P) {
    const float z_st3 = P.z[detid_lasthit];
    const float x_st3 = x0 + tx * z_st3;
    const float y_st3 = y0 + ty * z_st3;
    const short detid = (short)(2 * i + 2);
    idx = c_planetype[detid / 2 - 1];
    const short detid_2 = (short)(c_detsuperid[2][idx] * 2);
    const float pos_st3 = x_st3 * P.costheta[detid_2] + y_st3 * P.sintheta[detid_2];
    const float z_st1 = P.z[detid];
    const float z_st2 = P.z[detid_2];
    const float x_st2 = x0 + tx * z_st2;
    const float y_st2 = y0 + ty * z_st2;
    const float pos_st2 = x_st2 * P.costheta[detid_2] + y_st2 * P.sintheta[detid_2];
    const float s2_target = pos_st2 - pos_st3 * (z_st2 - Z_TARGET) / (z_st3 - Z_TARGET);
    const float s2_dump = pos_st2 - pos_st3 * (z_st2 - Z_DUMP) / (z_st3 - Z_DUMP);
    const float pe_t = SAGITTA_TARGET_CENTER * s2_target + pos_st3 * (z_st1 - Z_TARGET) / (z_st3 - Z_TARGET);
    const float pe_d = SAGITTA_DUMP_CENTER * s2_dump + pos_st3 * (z_st1 - Z_DUMP) / (z_st3 - Z_DUMP);
    const float win_t = fabsf(s2_target * SAGITTA_TARGET_WIDTH);
    const float win_d = fabsf(s2_dump * SAGITTA_DUMP_WIDTH);
    const float p_min = fminf(pe_t - win_t, pe_d - win_d);
    const float p_max = fmaxf(pe_t + win_t, pe_d + win_d);
    pos_exp = (float)(0.5 * (double)(p_max + p_min));
    window = (float)(0.5 * (double)(p_max - p_min));
}

// list of entry i of an index space whose lists start at s[0..5]
__device__ __forceinline__ int gl_list_of(const int *s, int i) {
    int l = 0;
#pragma unroll
    for (int k = 1; k < 6; ++k) l += i >= s[k];
    return l;
}

// The station-1 hits in the windows S.lo / S.hi and their pairs
// (make_hitpairs_in_station, H:464-549), in the reference's order: pairs in
// (hit1, hit2) order, the unpaired hits of plane 1, those of plane 2.  The
// hits of the six planes, the candidate pairs of the three projections and
// the unpaired hits are one index space each, 32 entries at a time.  Returns
// false when a projection has more pairs than the cap.
__device__ __forceinline__ bool gl_windows(GlWarp &S, const or_plane_t &P) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    int start = lane < 6 ? min(S.hc[lane].n, WP_MAXHITS) : 0;
    const int n = start;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, start, o);
        if (lane >= o) start += v;
    }
    const int total = __shfl_sync(0xffffffffu, start, 5);
    start -= n;
    if (lane < 6) S.start[lane] = start;
    if (lane < 3) S.np[lane] = 0;
    if (lane < 6 * GL_PAIRCAP / 32) S.fl[lane] = 0u;
    __syncwarp();
    int nwin = 0, wo = -1;
#pragma unroll 1
    for (int b0 = 0; b0 < total; b0 += 32) {
        const int f = b0 + lane;
        bool in = false;
        int i = 0;
        if (f < total) {
            const int l = gl_list_of(S.start, f);
            i = f - S.start[l];
            in = wp_in_window(gl_det(l), S.hc[l].chan(i), S.lo[l >> 1], S.hi[l >> 1], P);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        const int k = nwin + __popc(m & lt);
        if (in && k < 6 * GL_PAIRCAP) S.wl[k] = (unsigned char)i;
        if (lane < 6 && start >= b0 && start < b0 + 32) wo = nwin + __popc(m & ((1u << (start - b0)) - 1u));
        nwin += __popc(m);
    }
    if (wo < 0) wo = nwin;
    const int next = __shfl_down_sync(0xffffffffu, wo, 1);
    const int nw = (lane == 5 ? nwin : next) - wo;
    if (__any_sync(0xffffffffu, lane < 6 && nw > GL_PAIRCAP)) return false;  // each of them is in a pair
    if (lane < 6) S.woff[lane] = wo;
    if (lane == 6) S.woff[6] = nwin;
    const int n2 = __shfl_down_sync(0xffffffffu, nw, 1);
    const int c12 = lane < 6 && (lane & 1) == 0 ? nw * n2 : 0;  // lane 2q: projection q
    int incl = c12;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const int npair = __shfl_sync(0xffffffffu, incl, 5);
    __syncwarp();
    if (lane < 6 && (lane & 1) == 0) S.start[lane >> 1] = incl - c12;
    __syncwarp();
    auto append = [&](bool take, int q, uchar2 v) {
        const unsigned peers = __match_any_sync(0xffffffffu, take ? q : 4 + lane);
        int at = 0;
        if (take) {
            at = S.np[q];
            const int k = at + __popc(peers & lt);
            if (k < GL_PAIRCAP) S.pairs[q][k] = v;
        }
        __syncwarp();
        if (take && (peers & lt) == 0u) S.np[q] = at + __popc(peers);
        __syncwarp();
    };
#pragma unroll 1
    for (int b0 = 0; b0 < npair; b0 += 32) {
        const int f = b0 + lane;
        bool take = false;
        int q = 0, ia = 0, ib = 0;
        if (f < npair) {
            q = (f >= S.start[1]) + (f >= S.start[2]);
            const int oa = S.woff[2 * q], ob = S.woff[2 * q + 1], c2 = S.woff[2 * q + 2] - ob, c = f - S.start[q];
            ia = c / c2;
            ib = c - ia * c2;
            const float spacing = c_spacingplane[c_detsuperid[0][q]];
            if (!(fabsf(S.hc[2 * q].pos(S.wl[oa + ia]) - S.hc[2 * q + 1].pos(S.wl[ob + ib])) > spacing)) {
                take = true;
                atomicOr(&S.fl[(oa + ia) >> 5], 1u << ((oa + ia) & 31));
                atomicOr(&S.fl[(ob + ib) >> 5], 1u << ((ob + ib) & 31));
            }
        }
        append(take, q, make_uchar2((unsigned char)ia, (unsigned char)ib));
    }
#pragma unroll 1
    for (int b0 = 0; b0 < nwin; b0 += 32) {
        const int k = b0 + lane;
        const bool take = k < nwin && !((S.fl[b0 >> 5] >> lane) & 1u);
        const int l = take ? gl_list_of(S.woff, k) : 0;
        const unsigned char i = (unsigned char)(k - S.woff[l]);
        append(take, l >> 1, (l & 1) ? make_uchar2(255, i) : make_uchar2(i, 255));
    }
    return S.np[0] <= GL_PAIRCAP && S.np[1] <= GL_PAIRCAP && S.np[2] <= GL_PAIRCAP;
}

// one x1 pair's fit (K:2108-2203) for the state (y0, ty) it finds; `sdet`,
// `sdrift` = scratch entry 1
struct GlX {
    float xs0, xst;
    int nhx, signs;  // signs: 2 bits each, two's complement
    unsigned c0, c1; // codes of its hits
    bool pass;
};

__device__ __forceinline__ GlX gl_xfit(const GlWarp &S, uchar2 px, float x0, float tx, float ex0, float etx, float y0,
                                       float ty, int sdet, float sdrift, const or_plane_t &P) {
    GlX o;
    // first (only) hit in index 0, x' hit of a pair in index 1
    const bool two = px.x != 255 && px.y != 255;
    const int la = px.x != 255 ? 0 : 1;
    const int ha = S.wl[S.woff[la] + (la ? px.y : px.x)], hb = two ? S.wl[S.woff[1] + px.y] : 0;
    const int d0 = gl_det(la);
    o.nhx = two ? 2 : 1;
    o.c0 = (unsigned)(la << 12 | ha);
    o.c1 = two ? (unsigned)(1 << 12 | hb) : GL_NONE;
    float X0 = 0.f, Z0 = 0.f, X1 = 0.f, Z1 = 0.f;
    const float dr0 = S.hc[la].drift(ha), dr1 = two ? S.hc[1].drift(hb) : 0.f;
    const float r0 = P.resolution[d0], r1 = P.resolution[3];
#pragma unroll 1
    for (int k = 0; k < o.nhx; ++k) {
        float X, Z;
        calculate_xz_fy(k ? 3 : d0, (short)(k ? S.hc[1].chan(hb) : S.hc[la].chan(ha)), k ? dr1 : dr0, 0, y0, ty, P, X, Z);
        if (k) {
            X1 = X;
            Z1 = Z;
        } else {
            X0 = X;
            Z0 = Z;
        }
    }
    const float Xk = x0 + tx * Z_KMAG_BEND;  // K:2163-2165
    const float ek = ex0 + etx * Z_KMAG_BEND;
    float xs0, xst, e0, e1;
    int s0 = 0, s1 = 0;
    // the fit, the signs it gives, and the fit with the drift distances
#pragma unroll 1
    for (int pass = 0;; ++pass) {
        Fit2 f;
        f.add(X0, Z0, r0);
        if (two) f.add(X1, Z1, r1);
        f.add(Xk, Z_KMAG_BEND, ek);
        f.solve(xs0, xst, e0, e1);
        if (pass) break;
        // resolve_leftright_xhits (H:820-871): the two hits, or the one hit
        // with scratch entry 1 (whose position is the KMag point)
        const int dj = two ? 3 : sdet;
        if (abs(d0 - dj) == 1) {
            const int k = lr_pair_xhits(xs0, xst, xs0, xst, (short)d0, (short)dj, X0, dr0, two ? X1 : Xk,
                                        two ? dr1 : sdrift, P.z, 150.f);
            if (k >= 0) {
                s0 = c_lrpossibility[k][0];
                if (two) s1 = c_lrpossibility[k][1];
            }
        }
        if (!s0) s0 = single_sign_xhits(xs0, xst, (short)d0, X0, P.z);
        if (two && !s1) s1 = single_sign_xhits(xs0, xst, 3, X1, P.z);
        X0 += (float)s0 * dr0;
        X1 += (float)s1 * dr1;
    }
    o.xs0 = xs0;
    o.xst = xst;
    o.signs = (s0 & 3) | ((s1 & 3) << 2);
    const short charge = calculate_charge(tx, x0);  // K:2198-2203
    const float invP = (xst - tx) * (float)charge / PT_KICK_KMAG;
    const float einvP = (etx - etx) / PT_KICK_KMAG;
    o.pass = !(invP > INVP_MAX + einvP || invP < INVP_MIN - einvP);
    return o;
}

// place of hit k of list l (u1 u1' v1 v1') among its projection's hits
__device__ __forceinline__ int gl_place(const GlWarp &S, int l, int k) {
    return (l & 1) ? S.woff[l + 2] - S.woff[l + 1] + k : k;
}
__device__ __forceinline__ bool gl_acc(const GlWarp &S, int l, int k) {
    const int f = gl_place(S, l, k);
    return (S.acc[l >> 1][f >> 5] >> (f & 31)) & 1u;
}
// which of pair p's two hits (lists l, l + 1 of u1 u1' v1 v1') are accepted
__device__ __forceinline__ int gl_group(const GlWarp &S, int l, uchar2 p) {
    return (p.x != 255 && gl_acc(S, l, p.x) ? 1 : 0) | (p.y != 255 && gl_acc(S, l + 1, p.y) ? 2 : 0);
}
__device__ __forceinline__ unsigned gl_code(const GlWarp &S, int l, int k) { return (unsigned)((l + 2) << 12 | S.wl[S.woff[l + 2] + k]); }
// the hit a v1 (u1) pair leaves at its first offset: the second one when the
// first is refused or missing
__device__ __forceinline__ unsigned gl_rel0(const GlWarp &S, int l, uchar2 p) {
    const bool second = p.x == 255 || (!gl_acc(S, l, p.x) && p.y != 255);
    return second ? gl_code(S, l + 1, p.y) : gl_code(S, l, p.x);
}

// sign state of a lone x' hit carried from one chunk of survivors to the next
struct GlCarry {
    int ix = -1;
    bool has = false;
    int sign = 0;
};

struct Stale3 {
    short det;
    float pos, drift;
};

__device__ __forceinline__ Stale3 gl_decode(const GlWarp &S, unsigned code) {
    if (code == GL_NONE) return Stale3{DET_SENTINEL, 0.f, 0.f};
    const int l = (int)(code >> 12), h = (int)(code & 0xFFFu);
    return Stale3{(short)gl_det(l), S.hc[l].pos(h), S.hc[l].drift(h)};
}

// A survivor's hits in order (x1 then u1 u1' v1 v1'), codes of 16 bits.
struct GlHits {
    unsigned long long lo, hi;
    unsigned sign;
    int n;
    __device__ __forceinline__ unsigned code(int k) const {
        return (unsigned)((k < 4 ? lo >> (16 * k) : hi >> (16 * (k - 4))) & 0xFFFFull);
    }
    __device__ __forceinline__ void push(unsigned c) {
        if (n < 4) lo |= (unsigned long long)c << (16 * n);
        else hi |= (unsigned long long)c << (16 * (n - 4));
        ++n;
    }
    __device__ __forceinline__ int get_sign(int k) const { return (int)(sign << (30 - 2 * k)) >> 30; }
    __device__ __forceinline__ void set_sign(int k, int s) { sign = (sign & ~(3u << (2 * k))) | (((unsigned)s & 3u) << (2 * k)); }
};

// residual_line out of line: one copy for the chi2 sums and the winner
__device__ __noinline__ float gl_residual(float p1x, float p1y, float p1z, float dpx, float dpy, float dpz, float drift,
                                          int sign, float x0, float y0, float tx, float ty) {
    return residual_line(p1x, p1y, p1z, dpx, dpy, dpz, drift, (short)sign, x0, y0, tx, ty);
}

__device__ __forceinline__ float gl_res1(const GlWarp &S, const GlHits &h, int k, const or_plane_t &P, float xs0,
                                         float xst, float yc, float tyc, int &d) {
    const unsigned c = h.code(k);
    const int l = (int)(c >> 12), hi = (int)(c & 0xFFFu);
    d = gl_det(l);
    const short el = (short)S.hc[l].chan(hi);
    return gl_residual(x_bep(d, el, P), y_bep(d, el, P), z_bep(d, el, P), P.deltapx[d], P.deltapy[d], P.deltapz[d],
                       S.hc[l].drift(hi), h.get_sign(k), xs0, yc, xst, tyc);
}

// The left/right walk and chi2 of n (<= 32) survivors from the ring, in order
// (K:2380-2501), and the best combination so far.
__device__ __noinline__ void gl_pass(GlWarp &S, int head, int n, int nst, float x0, float tx, const or_plane_t &P,
                                     GlCarry &cs, float &chi2min, bool &update) {
    const int lane = lane_id();
    const bool valid = lane < n;
    const GlSurv q = S.ring[(head + lane) & 63];
    const int ix = valid ? (int)(q.a & 127u) : -2 - lane;
    const float xs0 = q.xs0, xst = q.xst, yc = q.yc, tyc = q.tyc;
    const int g = (int)(q.b >> 7) & 15;
    float eyc = 0.f, etyc = 0.f;
    GlHits h{0ull, 0ull, 0u, 0};
    if (valid) {
        const float *te = S.tab[((g & 3) - 1) * 3 + (g >> 2) - 1];
        eyc = te[6];
        etyc = te[7];
        const uchar2 px = S.pairs[0][ix], pu = S.pairs[1][q.b & 127u], pv = S.pairs[2][(q.a >> 13) & 127u];
        if (px.x != 255) h.push((unsigned)S.wl[px.x]);
        if (px.y != 255) h.push((unsigned)(1 << 12 | S.wl[S.woff[1] + px.y]));
        h.sign = (q.a >> 9) & 15u;
        if (g & 1) h.push(gl_code(S, 0, pu.x));
        if (g & 2) h.push(gl_code(S, 1, pu.y));
        if (g & 4) h.push(gl_code(S, 2, pv.x));
        if (g & 8) h.push(gl_code(S, 3, pv.y));
    }
    // x' hit alone, paired with the first u1 hit (planes 3, 2): the sign of
    // the last earlier combination of the x1 pair that resolved it
    const bool alone = valid && ((q.a >> 20) & 1u);
    if (__any_sync(0xffffffffu, alone)) {
        bool xok = false;
        int xval = 0;
        if (valid && ((q.a >> 21) & 1u)) {
            const Stale3 h0 = gl_decode(S, h.code(0)), h1 = gl_decode(S, h.code(1));
            const int k = lr_pair_newhits_ool(xs0, xst, yc, tyc, xs0, xst, eyc, etyc, h0.det, h1.det, h0.pos, h0.drift,
                                              h1.pos, h1.drift, P, 150.f);
            if (k >= 0) {
                xok = true;
                xval = c_lrpossibility[k][0];
            }
        }
        const unsigned seg = __match_any_sync(0xffffffffu, ix);
        const unsigned xm = __ballot_sync(0xffffffffu, xok);
        const int xs = last_lane(xm & seg & lanemask_lt());
        const int xprev = __shfl_sync(0xffffffffu, xval, xs < 0 ? 0 : xs);
        if (alone) {
            if (xs >= 0) h.set_sign(0, xprev);
            else if (ix == cs.ix && cs.has) h.set_sign(0, cs.sign);
        }
        const int il = __shfl_sync(0xffffffffu, ix, n - 1);
        const int xl = last_lane(xm & __ballot_sync(0xffffffffu, ix == il));
        const int nx = __shfl_sync(0xffffffffu, xval, xl < 0 ? 0 : xl);
        if (xl >= 0) {
            cs.has = true;
            cs.sign = nx;
        } else if (il != cs.ix) {
            cs.has = false;
        }
        cs.ix = il;
    }
    const bool in = valid && !(fabsf(yc) > Y0_MAX || fabsf(tyc) > TY_MAX);  // K:2410
    bool pass = false;
    float chi2 = 0.f;
    if (in) {
        // resolve_leftright_newhits over the x + uv hits (H:714-780), with
        // the scratch entry past the end, then the singles (H:785-804)
#pragma unroll 1
        for (int i = 0; i < h.n;) {
            const int j = i + 1;
            const unsigned ci = h.code(i), cj = j < h.n ? h.code(j) : q.b >> 16;
            const int di = gl_det((int)(ci >> 12)), dj = cj == GL_NONE ? (int)DET_SENTINEL : gl_det((int)(cj >> 12));
            if (abs(di - dj) != 1) {
                i += 1;
                continue;
            }
            const int sj = j < h.n ? h.get_sign(j) : 0;
            if (h.get_sign(i) * sj == 0) {
                const Stale3 hi = gl_decode(S, ci), hj = gl_decode(S, cj);
                const int k = lr_pair_newhits_ool(xs0, xst, yc, tyc, xs0, xst, eyc, etyc, (short)di, (short)dj, hi.pos,
                                                  hi.drift, hj.pos, hj.drift, P, 150.f);
                if (k >= 0) {
                    h.set_sign(i, c_lrpossibility[k][0]);
                    if (j < h.n) h.set_sign(j, c_lrpossibility[k][1]);
                }
            }
            i += 2;
        }
#pragma unroll 1
        for (int k = 0; k < h.n; ++k) {
            if (h.get_sign(k)) continue;
            const Stale3 hk = gl_decode(S, h.code(k));
            h.set_sign(k, single_sign_newhits(xs0, xst, yc, tyc, hk.det, hk.pos, P));
        }
        // chi2 over the station-2/3 hits (H:1149-1180) plus chi2_track over
        // the station-1 hits (K:2449-2461)
#pragma unroll 1
        for (int m = 0; m < nst; ++m) {
            const float r = gl_residual(S.p1x[m], S.p1y[m], S.p1z[m], S.dpx[m], S.dpy[m], S.dpz[m], S.drift[m], S.sign[m],
                                        x0, yc, tx, tyc);
            chi2 += r * r / S.res2[m];
        }
        float c1 = 0.f;
#pragma unroll 1
        for (int k = 0; k < h.n; ++k) {
            int d;
            const float r = gl_res1(S, h, k, P, xs0, xst, yc, tyc, d);
            c1 += r * r / P.resolution[d] / P.resolution[d];
        }
        chi2 += c1;
        pass = !(chi2 > 10000.f);
    }
    // best chi2, strict < in combination order (K:2470)
    const bool elig = pass && chi2 < chi2min;
    const unsigned key = elig ? __float_as_uint(chi2) : 0xffffffffu;
    const unsigned kmin = __reduce_min_sync(0xffffffffu, key);
    if (kmin != 0xffffffffu) {
        const int winl = __ffs(__ballot_sync(0xffffffffu, key == kmin)) - 1;
        if (lane == winl) {
            S.b_n = h.n;
            S.b_chi2 = chi2;
            S.b_ty = tyc;
            S.b_y0 = yc;
            S.b_xst = xst;
            S.b_ety = etyc;
            S.b_ey0 = eyc;
        }
        // the winner's hits and residuals, one per lane
        GlHits w;
        w.lo = __shfl_sync(0xffffffffu, h.lo, winl);
        w.hi = __shfl_sync(0xffffffffu, h.hi, winl);
        w.sign = __shfl_sync(0xffffffffu, h.sign, winl);
        w.n = __shfl_sync(0xffffffffu, h.n, winl);
        const float wx = __shfl_sync(0xffffffffu, xs0, winl), wt = __shfl_sync(0xffffffffu, xst, winl);
        const float wy = __shfl_sync(0xffffffffu, yc, winl), wty = __shfl_sync(0xffffffffu, tyc, winl);
        if (lane < nst) {
            S.b_res[lane] = gl_residual(S.p1x[lane], S.p1y[lane], S.p1z[lane], S.dpx[lane], S.dpy[lane], S.dpz[lane],
                                        S.drift[lane], S.sign[lane], x0, wy, tx, wty);
        } else if (lane >= 16 && lane < 16 + w.n) {
            const int k = lane - 16;
            const unsigned c = w.code(k);
            const int l = (int)(c >> 12), hi = (int)(c & 0xFFFu);
            int d;
            S.b_res[nst + k] = gl_res1(S, w, k, P, wx, wt, wy, wty, d);
            S.b_det[k] = (float)d;
            S.b_el[k] = (float)(short)S.hc[l].chan(hi);
            S.b_pos[k] = S.hc[l].pos(hi);
            S.b_drift[k] = S.hc[l].drift(hi);
            S.b_sign[k] = (float)w.get_sign(k);
            S.b_tdc[k] = S.hc[l].tdc(hi);
        }
        chi2min = __uint_as_float(kmin);
        update = true;
    }
    __syncwarp();
}

// One track of the slot; S.st is the slot's scratch state.
__device__ __forceinline__ void gl_track(GlWarp &S, float *T, const or_plane_t &P, uint32_t *__restrict__ errw) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const float stid = T[OR_TRK_STID];
    if (stid < 5) return;  // K:2053
    const int nst = (int)(short)min((int)T[OR_TRK_NHITS], 12);  // YZ tracks carry <= 12 hits
    const float x0 = T[OR_TRK_X0], tx = T[OR_TRK_TX], ex0 = T[OR_TRK_ERR_X0], etx = T[OR_TRK_ERR_TX];
    float y0 = T[OR_TRK_Y0], ty = T[OR_TRK_TY];
    // the track's station-2/3 hits, one per lane
    int det = 0, chan = 0;
    float dr = 0.f;
    short sg = 0;
    const bool mine = lane < nst;
    if (mine) {
        det = (int)(short)T[OR_TRK_HIT_DETID + lane];
        chan = (int)T[OR_TRK_HIT_CHAN + lane];
        dr = T[OR_TRK_HIT_DRIFT + lane];
        sg = (short)T[OR_TRK_HIT_SIGN + lane];
    }
    // get_lasthitdetid (reconstruction_classes.cuh:500-515): the first of the
    // hits with the largest z
    int dmax = 1;
    {
        float z = mine && det > 0 ? P.z[det] : -10000.f;
        int who = mine && det > 0 && z > -10000.f ? lane : 32;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const float oz = __shfl_xor_sync(0xffffffffu, z, o);
            const int ow = __shfl_xor_sync(0xffffffffu, who, o);
            if (ow < 32 && (who == 32 || oz > z || (oz == z && ow < who))) {
                z = oz;
                who = ow;
            }
        }
        who = __shfl_sync(0xffffffffu, who, 0);
        const int d = __shfl_sync(0xffffffffu, det, who & 31);
        if (who < 32) dmax = d;
    }
    // station-1 windows, one projection per lane
    __syncwarp();  // every lane is done with the previous track's lists
    if (lane < 3) {
        int idx;
        float pe, wi;
        sagitta_st1(lane, x0, tx, y0, ty, dmax, idx, pe, wi, P);
        S.lo[idx] = pe - wi * 1.0f;
        S.hi[idx] = pe + wi * 1.0f;
    }
    __syncwarp();
    if (!gl_windows(S, P)) {
        if (lane == 0) atomicOr(errw, ERRW_CAPACITY);
        return;
    }
    const int nx1 = S.np[0], nu1 = S.np[1], nv1 = S.np[2];
    if (nx1 == 0 || nu1 == 0 || nv1 == 0) return;
    // station-2/3 hits and their y (K:2086-2102)
    int nyh;
    {
        bool acc = false;
        float yy = 0.f, ey = 0.f;
        if (mine) {
            S.p1x[lane] = x_bep(det, (short)chan, P);
            S.p1y[lane] = y_bep(det, (short)chan, P);
            S.p1z[lane] = z_bep(det, (short)chan, P);
            S.dpx[lane] = P.deltapx[det];
            S.dpy[lane] = P.deltapy[det];
            S.dpz[lane] = P.deltapz[det];
            S.drift[lane] = dr;
            S.sign[lane] = sg;
            S.res2[lane] = P.resolution[det] * P.resolution[det];
            if (!((double)P.costheta[det] > 0.99))
                acc = calculate_y_uvhit((int)T[OR_TRK_HIT_DETID + lane], chan, dr, sg, x0, tx, P, yy, ey);
        }
        const unsigned m = __ballot_sync(0xffffffffu, acc);
        if (acc) {
            const int k = __popc(m & lt);
            S.Y[k] = yy;
            S.eY[k] = ey;
            S.Zy[k] = P.z[det];
        }
        nyh = __popc(m);
    }
    __syncwarp();
    // the y fit's station-1 plane sets, one per lane, and the right-hand side
    // of the station-2/3 hits (Fit2::add order)
    if (lane < 9) gl_tab_entry(S.eY, S.Zy, nyh, lane / 3 + 1, lane % 3 + 1, P, S.tab[lane]);
    float bs0 = 0.f, bs1 = 0.f;
#pragma unroll 1
    for (int k = 0; k < nyh; ++k) {
        bs0 += S.eY[k] * S.Y[k];
        bs1 += S.eY[k] * S.Y[k] * S.Zy[k];
    }
    __syncwarp();
    float chi2min = 10000.1f;
    bool update = false;
    GlCarry cs;
    int head = 0, waiting = 0;
#pragma unroll 1
    for (int ib = 0; ib < nx1;) {
        // --- x fits of x1 pairs ib .. ib+31, up to the first that passes ----
        const int ix = ib + lane;
        const bool in = ix < nx1;
        const uchar2 px = S.pairs[0][in ? ix : ib];
        const bool two = in && px.x != 255 && px.y != 255;
        const unsigned twom = __ballot_sync(0xffffffffu, two);
        // scratch entry 1: the x' hit of the last earlier pair of two
        const int pt = last_lane(twom & lt);
        const unsigned x1code = two ? (unsigned)(1 << 12 | S.wl[S.woff[1] + px.y]) : GL_NONE;
        const unsigned prev = __shfl_sync(0xffffffffu, x1code, pt < 0 ? 0 : pt);
        const unsigned e1 = pt >= 0 ? prev : S.st[1];
        GlX x;
        x.pass = false;
        x.nhx = x.signs = 0;
        x.xs0 = x.xst = 0.f;
        x.c0 = x.c1 = GL_NONE;
        if (in) {
            int sdet = DET_SENTINEL;
            float sdr = 0.f;
            if (!two && e1 != GL_NONE) {
                const int l = (int)(e1 >> 12);
                sdet = gl_det(l);
                sdr = S.hc[l].drift((int)(e1 & 0xFFFu));
            }
            x = gl_xfit(S, px, x0, tx, ex0, etx, y0, ty, sdet, sdr, P);
        }
        const unsigned pm = __ballot_sync(0xffffffffu, x.pass);
        const int p = pm ? __ffs(pm) - 1 : min(32, nx1 - ib) - 1;  // the pair to go on with, or the last one
        // entries 0 and 1 as pairs ib .. ib+p leave them
        const int lt2 = last_lane(twom & (p == 31 ? ~0u : (2u << p) - 1u));
        const unsigned c1 = __shfl_sync(0xffffffffu, x1code, lt2 < 0 ? 0 : lt2);
        __syncwarp();  // every lane has read entry 1
        if (lane == p) S.st[0] = (unsigned short)x.c0;
        if (lane == 0 && lt2 >= 0) S.st[1] = (unsigned short)c1;
        __syncwarp();
        const int ixp = ib + p;
        ib += p + 1;
        if (!pm) continue;
        const float xs0 = __shfl_sync(0xffffffffu, x.xs0, p), xst = __shfl_sync(0xffffffffu, x.xst, p);
        const int nhx = __shfl_sync(0xffffffffu, x.nhx, p), signs = __shfl_sync(0xffffffffu, x.signs, p);
        const bool alone = nhx == 1 && (S.st[0] >> 12) == 1u;  // x' alone
        // its station-1 hits of projection h (0: u1, 1: v1): acceptance and fit terms
        auto accept = [&](int h) {
            const int o0 = S.woff[2 * h + 2], o1 = S.woff[2 * h + 3], n = S.woff[2 * h + 4] - o0;
            __syncwarp();  // every lane is done with the previous terms
#pragma unroll 1
            for (int b0 = 0; b0 < n; b0 += 32) {
                const int f = b0 + lane;
                bool a = false;
                if (f < n) {
                    const int l = 2 * h + 2 + (f >= o1 - o0), d = gl_det(l), hi = S.wl[o0 + f];
                    float yy = 0.f, ey = 0.f;
                    a = calculate_y_uvhit(d, (short)S.hc[l].chan(hi), S.hc[l].drift(hi), 0, xs0, xst, P, yy, ey);
                    if (a) S.term[f] = make_float2(ey * yy, ey * yy * P.z[d]);
                }
                const unsigned m = __ballot_sync(0xffffffffu, a);
                if (lane == 0) S.acc[h][b0 >> 5] = m;
            }
            __syncwarp();
        };
        accept(0);
        // --- accepted u1 pairs --------------------------------------------
        int nua = 0, firstU2 = 1 << 20, lastU1 = -1, lastU2 = -1;
#pragma unroll 1
        for (int b0 = 0; b0 < nu1; b0 += 32) {
            const int iu = b0 + lane;
            int g = 0;
            float t0 = bs0, t1 = bs1;
            if (iu < nu1) {
                const uchar2 pu = S.pairs[1][iu];
                g = gl_group(S, 0, pu);
                if (g & 1) {
                    const float2 t = S.term[pu.x];
                    t0 += t.x;
                    t1 += t.y;
                }
                if (g & 2) {
                    const float2 t = S.term[gl_place(S, 1, pu.y)];
                    t0 += t.x;
                    t1 += t.y;
                }
            }
            const unsigned am = __ballot_sync(0xffffffffu, g != 0);
            const unsigned m2 = __ballot_sync(0xffffffffu, g == 3);
            if (g) {
                const int k = nua + __popc(am & lt);
                S.ua[k] = (unsigned short)(iu | g << 7);
                S.bu[k] = make_float2(t0, t1);
            }
            nua += __popc(am);
            if (m2) {
                if (lastU2 < 0) firstU2 = b0 + __ffs(m2) - 1;
                lastU2 = b0 + last_lane(m2);
            }
            if (am & ~m2) lastU1 = b0 + last_lane(am & ~m2);
        }
        // --- accepted v1 pairs --------------------------------------------
        // r1: the pair's second hit is tried after its first was accepted
        accept(1);
        int nva = 0, lastR1 = 255;
#pragma unroll 1
        for (int b0 = 0; b0 < nv1; b0 += 32) {
            const int iv = b0 + lane;
            int g = 0;
            bool r1 = false;
            if (iv < nv1) {
                const uchar2 pv = S.pairs[2][iv];
                g = gl_group(S, 2, pv);
                r1 = (g & 1) && pv.y != 255;
            }
            const unsigned am = __ballot_sync(0xffffffffu, g != 0);
            const unsigned rm = __ballot_sync(0xffffffffu, r1);
            const int pr = last_lane(rm & lt);
            if (g) {
                const int k = nva + __popc(am & lt);
                S.va[k] = (unsigned)(iv | g << 7 | (pr >= 0 ? b0 + pr : lastR1) << 16);
            }
            nva += __popc(am);
            if (rm) lastR1 = b0 + last_lane(rm);
        }
        __syncwarp();
        // --- combinations ----------------------------------------------------
        const int nc = nua * nva;
        if (nc > 0) {
            const int sv = 32 / nua, su = 32 - sv * nua;
            int kv = lane / nua, ku = lane - kv * nua;
            float yl = 0.f, tl = 0.f;  // the fit of the last combination
#pragma unroll 1
            for (int b0 = 0; b0 < nc; b0 += 32) {
                bool keep = false;
                float yc = 0.f, tyc = 0.f;
                unsigned u = 0u, v = 0u;
                if (b0 + lane < nc) {
                    u = S.ua[ku];
                    v = S.va[kv];
                    const int gu = (int)(u >> 7), gv = (int)(v >> 7) & 3;
                    const float2 b = S.bu[ku];
                    float f0 = b.x, f1 = b.y;
                    const uchar2 pv = S.pairs[2][v & 127u];
                    if (gv & 1) {
                        const float2 t = S.term[pv.x];
                        f0 += t.x;
                        f1 += t.y;
                    }
                    if (gv & 2) {
                        const float2 t = S.term[gl_place(S, 3, pv.y)];
                        f0 += t.x;
                        f1 += t.y;
                    }
                    // K:2368-2379, Fit2::solve with the plane set's inverse
                    const float *te = S.tab[(gu - 1) * 3 + gv - 1];
                    yc = 0.0f;
                    yc += te[0] * f0;
                    yc += te[1] * f1;
                    tyc = 0.0f;
                    tyc += te[2] * f0;
                    tyc += te[3] * f1;
                    // past the hard cut a combination only matters for the
                    // x' sign it may set
                    keep = !(fabsf(yc) > te[4] || fabsf(tyc) > te[5]) &&
                           (!(fabsf(yc) > Y0_MAX || fabsf(tyc) > TY_MAX) || (alone && (gu & 1)));
                }
                if (b0 + 32 >= nc) {
                    yl = __shfl_sync(0xffffffffu, yc, nc - 1 - b0);
                    tl = __shfl_sync(0xffffffffu, tyc, nc - 1 - b0);
                }
                const unsigned km = __ballot_sync(0xffffffffu, keep);
                if (km) {
                    if (keep) {
                        const int iu = (int)(u & 127u), iv = (int)(v & 127u);
                        const int gu = (int)(u >> 7), gv = (int)(v >> 7) & 3;
                        const uchar2 pv = S.pairs[2][iv];
                        // The scratch entry past the hits is only read by a
                        // v1 hit left without its partner plane's, and only
                        // pairs with a hit of that plane.
                        unsigned code = GL_NONE;
                        if (gv != 3) {
                            const int prevR1 = (int)(v >> 16);
                            if (gv == 1 && pv.y != 255) {
                                code = gl_code(S, 3, pv.y);  // its own refused v1' hit
                            } else if (gu == 3) {  // entry nhx + 3
                                code = prevR1 != 255 ? gl_code(S, 3, S.pairs[2][prevR1].y) : S.st[nhx + 3];
                            } else if (firstU2 < iu) {
                                code = GL_NONE;  // entry nhx + 2: this v1 pair's own hit, after two u1 hits
                            } else if (lastU2 >= 0) {
                                if (iv == 0) {
                                    code = S.st[nhx + 2];
                                } else {
                                    const uchar2 pp = S.pairs[2][iv - 1];
                                    code = lastU1 > lastU2 && prevR1 == iv - 1 ? gl_code(S, 3, pp.y) : gl_rel0(S, 2, pp);
                                }
                            } else {
                                code = prevR1 != 255 ? gl_code(S, 3, S.pairs[2][prevR1].y) : S.st[nhx + 2];
                            }
                        }
                        GlSurv o;
                        o.xs0 = xs0;
                        o.xst = xst;
                        o.yc = yc;
                        o.tyc = tyc;
                        o.a = (unsigned)ixp | (unsigned)nhx << 7 | (unsigned)signs << 9 | (unsigned)iv << 13 |
                              (alone ? 1u << 20 : 0u) | (alone && (gu & 1) ? 1u << 21 : 0u);
                        o.b = (unsigned)iu | (unsigned)(gu | gv << 2) << 7 | code << 16;
                        S.ring[(head + waiting + __popc(km & lt)) & 63] = o;
                    }
                    waiting += __popc(km);
                    __syncwarp();
                    if (waiting >= 32) {
                        gl_pass(S, head, 32, nst, x0, tx, P, cs, chi2min, update);
                        head = (head + 32) & 63;
                        waiting -= 32;
                    }
                }
                ku += su;
                const int cy = ku >= nua;
                ku -= cy ? nua : 0;
                kv += sv + cy;
            }
            y0 = yl;
            ty = tl;
        }
        // --- scratch entries as this x1 pair leaves them --------------------
        // lane m = 0..3: entry nhx + m.  0: every combination tries its u1
        // pair; 1: the last combination with an accepted u1 hit; 2: v1 hits
        // after two u1 hits, or a second v1 attempt after one; 3: a second
        // v1 attempt after two u1 hits
        if (lane < 4) {
            unsigned c = GL_NONE;
            const int iv = nv1 - 1;
            const bool second = lastR1 != 255;
            if (lane == 0) {
                c = gl_rel0(S, 0, S.pairs[1][nu1 - 1]);
            } else if (lane == 1 && lastU2 > lastU1) {
                c = gl_code(S, 1, S.pairs[1][lastU2].y);
            } else if ((lane == 1 && lastU1 >= 0) || (lane == 2 && lastU2 >= 0 && !(lastU1 > lastU2 && lastR1 == iv))) {
                c = gl_rel0(S, 2, S.pairs[2][iv]);
            } else if (second && ((lane == 2 && lastU1 >= 0) || (lane == 3 && lastU2 >= 0))) {
                c = gl_code(S, 3, S.pairs[2][lastR1].y);
            }
            if (c != GL_NONE) S.st[nhx + lane] = (unsigned short)c;
        }
        __syncwarp();
    }
    if (waiting) gl_pass(S, head, waiting, nst, x0, tx, P, cs, chi2min, update);
    if (update) {  // K:2504-2528
        const int n1 = S.b_n;
        const short charge = calculate_charge(tx, x0);
        if (lane == 0) {
            T[OR_TRK_STID] = 6.f;
            T[OR_TRK_NHITS] = (float)nst + (float)n1;
            T[OR_TRK_CHI2] = S.b_chi2;
            T[OR_TRK_TY] = S.b_ty;
            T[OR_TRK_Y0] = S.b_y0;
            T[OR_TRK_INVP] = (S.b_xst - tx) * (float)charge / PT_KICK_KMAG;
            T[OR_TRK_ERR_TY] = S.b_ety;
            T[OR_TRK_ERR_Y0] = S.b_ey0;
            T[OR_TRK_ERR_INVP] = (etx - etx) / PT_KICK_KMAG;
            T[OR_TRK_CHARGE] = (float)charge;
        }
        if (mine) T[OR_TRK_HIT_RESID + lane] = S.b_res[lane];
        if (lane < n1) {
            const int n = lane;
            T[OR_TRK_HIT_DETID + nst + n] = S.b_det[n];
            T[OR_TRK_HIT_CHAN + nst + n] = S.b_el[n];
            T[OR_TRK_HIT_POS + nst + n] = S.b_pos[n];
            T[OR_TRK_HIT_DRIFT + nst + n] = S.b_drift[n];
            T[OR_TRK_HIT_SIGN + nst + n] = S.b_sign[n];
            T[OR_TRK_HIT_TDC + nst + n] = S.b_tdc[n];
            T[OR_TRK_HIT_RESID + nst + n] = S.b_res[nst + n];
        }
    }
    __syncwarp();
}

constexpr int GL_LIST_THREADS = 1024;
// Slots that hold a track to extend (stationID >= 5) of events not rejected,
// in four classes by the work they are about to make (tracks times the square
// of the event's station-1 hits), sched[1 + class] = their numbers.  The warps
// take the largest class first, so that a long slot does not start last, and
// those that run side by side do the same kind of work (100,000 uneven events
// 9.2 -> 8.4 ms with the lowest bound at 3,000; 8.5 at 6,000, 8.7 at 12,000;
// 10,000 of them 1,376 -> 1,290 us).
constexpr int GL_CLASSES = 4;
constexpr int GL_WORK = 3000;  // the classes' bounds: this, twice and four times this
// where unit i of class c stands: classes 0 and 1 grow from the two ends of
// the first n places, 2 and 3 from those of the second
__device__ __forceinline__ unsigned long long gl_list_at(int c, unsigned long long i, unsigned long long n) {
    return (c >> 1) * n + ((c & 1) ? n - 1 - i : i);
}
__global__ void __launch_bounds__(GL_LIST_THREADS)
    global_list_kernel(or_hits_view_t hv, or_tracks_view_t tv, const uint8_t *__restrict__ toomany, int n_events,
                       unsigned long long *__restrict__ sched, unsigned *__restrict__ list) {
    __shared__ int warp_n[GL_LIST_THREADS / 32][GL_CLASSES];
    __shared__ unsigned base[GL_CLASSES];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long e = (long)blockIdx.x * (GL_LIST_THREADS / 32) + w;
    const int n = e < n_events && !toomany[e] ? min((int)tv.ntracks[e * OR_NSLOTS + lane], OR_SLOTCAP) : 0;
    const int most = __reduce_max_sync(0xffffffffu, n);
    int ntake = 0;
#pragma unroll 4
    for (int k = 0; k < most; ++k)
        if (k < n) ntake += trk_rec(tv, e, lane, k)[OR_TRK_STID] >= 5;
    const int hits = __reduce_add_sync(0xffffffffu, most && lane < 6 ? (int)hv.nhits_cham[e * OR_NCHAM + lane] : 0);
    const int work = ntake * hits * hits;
    const int cls = ntake == 0 ? -1 : work >= 4 * GL_WORK ? 0 : work >= 2 * GL_WORK ? 1 : work >= GL_WORK ? 2 : 3;
    const unsigned mine = __match_any_sync(0xffffffffu, cls);
    if (lane < GL_CLASSES) warp_n[w][lane] = 0;
    __syncwarp();
    const int rank = __popc(mine & lanemask_lt());
    if (cls >= 0 && rank == 0) warp_n[w][cls] = __popc(mine);
    __syncthreads();
    if (w < GL_CLASSES) {
        const int v = warp_n[lane][w];
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        warp_n[lane][w] = incl - v;
        if (lane == 31) base[w] = incl ? (unsigned)atomicAdd(sched + 1 + w, (unsigned long long)incl) : 0u;
    }
    __syncthreads();
    if (cls >= 0)
        list[gl_list_at(cls, base[cls] + warp_n[w][cls] + rank, (unsigned long long)n_events * OR_NSLOTS)] =
            (unsigned)(e * OR_NSLOTS + lane);
}

#ifndef OR_GL_WARPS_SM
#define OR_GL_WARPS_SM 20
#endif

// Work units are slots, taken from a device counter: slots are independent
// in the reference (one thread each, state kept per thread), and the cost per
// slot is very uneven, so warps that finish early keep taking units.
template <int W>
__global__ void __launch_bounds__(W * 32, (OR_GL_WARPS_SM / W > 0 ? OR_GL_WARPS_SM / W : 1))
    global_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv,
                  const uint8_t *__restrict__ toomany, int n_events, uint32_t *__restrict__ errw,
                  unsigned long long *__restrict__ sched, const unsigned *__restrict__ list) {
    extern __shared__ __align__(16) unsigned char gl_smem[];
    or_plane_t &P = *reinterpret_cast<or_plane_t *>(gl_smem);
    GlWarp *warps = reinterpret_cast<GlWarp *>(gl_smem + ((sizeof(or_plane_t) + 15) & ~size_t(15)));
    load_plane_smem(&P, gplane);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    GlWarp &S = warps[threadIdx.x >> 5];
    const unsigned long long nall = (unsigned long long)n_events * OR_NSLOTS;
    unsigned long long end[GL_CLASSES] = {nall, nall, nall, nall};  // units up to each class's last
    if (list) {
        end[0] = sched[1];
#pragma unroll
        for (int c = 1; c < GL_CLASSES; ++c) end[c] = end[c - 1] + sched[1 + c];
    }
    const unsigned long long nunits = end[GL_CLASSES - 1];
    // the next slot is taken while the current one is worked on; with no more
    // slots than warps each warp has its own (one taken ahead would wait while
    // other warps are idle)
    const bool own = nunits <= (unsigned long long)gridDim.x * W;
    unsigned long long nxt = own ? (unsigned long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x : 0ull;
    if (!own && lane == 0) nxt = atomicAdd(sched, 1ull);
    for (;;) {
        unsigned long long u = __shfl_sync(0xffffffffu, nxt, 0);
        if (u >= nunits) break;
        nxt = nunits;
        if (!own && lane == 0) nxt = atomicAdd(sched, 1ull);
        if (list) {
            int c = 0;
#pragma unroll
            for (int k = 0; k < GL_CLASSES - 1; ++k)
                if (u >= end[k]) c = k + 1;
            u = list[gl_list_at(c, u - (c ? end[c - 1] : 0ull), nall)];
        }
        const long e = (long)(u / OR_NSLOTS);
        const int slot = (int)(u % OR_NSLOTS);
        if (toomany[e]) continue;
        const int ntr = min((int)tv.ntracks[u], OR_SLOTCAP);
        if (ntr == 0) continue;
        __syncwarp();  // every lane is done with the previous event's views
        if (lane < 6) {  // chambers all
            const int d = gl_det(lane) - 1;
            S.hc[lane] = HitPlane{hv.hits_cham + e * OR_EVT_CHAM_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_CHAM * d,
                                  (int)hv.nhits_cham[e * OR_NCHAM + d]};
        }
        __syncwarp();
        if (lane < 8) S.st[lane] = (unsigned short)GL_NONE;
        __syncwarp();
#pragma unroll 1
        for (int it = 0; it < ntr; ++it) gl_track(S, trk_rec(tv, e, slot, it), P, errw);
    }
}

size_t global_smem_bytes(int warps) {
    return ((sizeof(or_plane_t) + 15) & ~size_t(15)) + sizeof(GlWarp) * (size_t)warps;
}

// `sched`: 256 bytes of counters and, after them, twice the room for list_cap
// slots (gl_list_at)
size_t global_sched_bytes(int list_cap) { return 256 + 2 * sizeof(unsigned) * (size_t)list_cap; }

template <int W>
static cudaError_t global_launch(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv,
                                 const uint8_t *toomany, int n_events, uint32_t *errw, unsigned long long *sched,
                                 int list_cap, cudaStream_t stream, int sm_count, bool cleared) {
    const size_t smem = global_smem_bytes(W);
    cudaError_t err = smem_attr_once((const void *)global_kernel<W>, (int)smem);
    if (err != cudaSuccess) return err;
    if (!cleared && (err = cudaMemsetAsync(sched, 0, (1 + GL_CLASSES) * sizeof(unsigned long long), stream)) != cudaSuccess)
        return err;
    const long nslots = (long)n_events * OR_NSLOTS;
    // the list saves an atomic per slot without a track; a batch beyond its
    // room visits every slot
    unsigned *list = nslots <= list_cap ? reinterpret_cast<unsigned *>(reinterpret_cast<char *>(sched) + 256) : nullptr;
    if (list) {
        global_list_kernel<<<(unsigned)((nslots + GL_LIST_THREADS - 1) / GL_LIST_THREADS), GL_LIST_THREADS, 0, stream>>>(
            hv, tv, toomany, n_events, sched, list);
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
    long blocks = (nslots + W - 1) / W;
    const long cap = (long)sm_count * (OR_GL_WARPS_SM / W > 0 ? OR_GL_WARPS_SM / W : 1);
    if (blocks > cap) blocks = cap;
    global_kernel<W><<<(unsigned)blocks, W * 32, smem, stream>>>(d_plane, hv, tv, toomany, n_events, errw, sched, list);
    return cudaGetLastError();
}

// `warps` = slots in flight per CTA: 1, 2, 4, 8 or 16; `cleared`: the counters
// are zero already (ChainClear)
cudaError_t launch_global(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv, const uint8_t *toomany,
                          int n_events, uint32_t *errw, unsigned long long *sched, int list_cap, cudaStream_t stream,
                          int sm_count, int warps, bool cleared) {
    if (n_events <= 0) return cudaSuccess;
#define OR_GL_LAUNCH(W) \
    global_launch<W>(d_plane, hv, tv, toomany, n_events, errw, sched, list_cap, stream, sm_count, cleared)
    switch (warps) {
    case 1: return OR_GL_LAUNCH(1);
    case 2: return OR_GL_LAUNCH(2);
    case 8: return OR_GL_LAUNCH(8);
    case 16: return OR_GL_LAUNCH(16);
    default: return OR_GL_LAUNCH(4);
    }
#undef OR_GL_LAUNCH
}

}  // namespace orgpu
