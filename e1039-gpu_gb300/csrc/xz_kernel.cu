// xz_kernel.cu -- station-2/3 XZ tracklets.
//
// Replaces gKernel_XZ_tracking<<<N,32>>> (OnlineReconstruction/
// reconstruction_kernels.cuh:182-855) with make_hitpairs_in_station_bins
// (reconstruction_helper.cuh:368-460) and the fit / left-right / prop / hodo
// helpers it calls.
//
// GPU layout: one warp per event, or for small batches one CTA of eight.
//  1. The hits of the six x planes are one index space: each hit's x and z
//     (calculate_xz_fy with y0 = ty = 0, so a property of the hit) is
//     computed once, not once per candidate.  So are the candidate pairs of
//     the three stations and the hits left unpaired; each bin's list keeps
//     the reference order (pairs in (i,j) order, then unpaired x, then
//     unpaired x') through __match_any_sync ranks.  A bin with more than 20
//     entries rejects the event (K:359-375).
//  2. The reference splits the 28x28 bin space over 32 threads (K:217-219);
//     every thread enumerates 49 bin pairs and, in each, all (pair2, pair3)
//     candidates.  Here the candidates of all 32 threads are one index space,
//     32 at a time; a thread's number of candidates is the product of the
//     entries in its seven station-2 and seven station-3 bins, so a
//     candidate's place follows from 32 prefix sums and three divisions.
//  3. The reference's per-thread scratch arrays persist across candidates,
//     and its left/right walk reads the entry just past the hit count when it
//     lands on the last hit (H:820-828).  That entry holds hit #2 (#3) of the
//     latest earlier candidate of the same thread with >= 3 (4) hits; a
//     segmented last-writer scan over the candidates (ballot + shuffle,
//     carried across chunks) gives each lane exactly that hit.
//  4. Candidates that pass the first fit's cut wait in a ring until 32 of
//     them can go through the left/right walk, the second fit and the gates
//     with every lane in use.
//  5. Surviving tracklets are written in order, each record by the whole
//     warp; the k-th tracklet of station-3 half p goes to slot 2*(k%16)+p,
//     position k/16 -- the round-robin the reference's least-populated-slot
//     balancing (K:675-807) performs when adds come one at a time.
//  With a CTA per event its warps take equal runs of candidates (the state
//  of 3. at the start of a run is found by walking back) and keep their
//  tracklets until the counts of the runs before are known.
//
// Bound: instruction issue on large batches, instruction fetch and the
// serial chain of one event on small ones.  With a prefix over the 1,568 bin
// pairs, the fits and gates of every candidate in the lane that held it,
// records written by single lanes and a warp per event always (80 KB of code)
// this took 7.87 ms for 100,000 uneven events, 555 us for 10,000 one-dimuon
// ones and 180 us for a single uneven one; it takes 4.16 ms, 263 us and 50 us.
#include "or_device.cuh"

namespace orgpu {

constexpr int XZ_MAXPLANEHITS = 200;
constexpr int XZ_HITS = 320;   // x-plane hits with x and z in shared memory (an accepted event has at most 300)
constexpr int XZ_GATE = 256;   // prop-tube and hodoscope hits kept there
constexpr int XZ_TEAM = 8;     // warps of an event's CTA on small batches
constexpr int XZ_STASH = 96;   // tracklets a warp of it keeps

// A candidate past the first cut, or a tracklet.
struct __align__(16) XzCand {
    float x0, tx, ex0, etx;
    unsigned long long hits;  // in order, 11 bits each (index over the six planes)
    unsigned stale;  // the scratch entry past the hits: same index, 0xFFFF = none
    unsigned place;  // t | cell << 8 | hit count << 16 | a tracklet's signs (2 bits each) << 24
};

struct XzWarp {
    XzCand ring[64];
    float rec[OR_NTRKPARAM];
};

struct XzEvent {
    HitPlane hc[6];              // x x' of stations 2, 3+, 3-
    int start[7];                // first hit of each plane in the index space
    int cpair[4];                // candidate pairs before each station
    const float *gpos[10];       // prop tubes 50 49 52 51, hodoscopes of stations 2-4
    int gn[10], goff[11], staged;
    float X[XZ_HITS], Z[XZ_HITS], drift[XZ_HITS];
    float gate[XZ_GATE];
    unsigned paired[(6 * XZ_MAXPLANEHITS + 31) / 32];
    uchar2 pairs[3][28][MAXHITS_PROJ_X];  // 255 = none
    int np[3][28], off[3][29];            // entries of each bin, of the bins before it
    int tpre[33];                         // candidates of the reference threads before each
    bool over;
};

// warps of one event together: a warp, or the CTA
template <int WPE>
__device__ __forceinline__ void xz_sync() {
    if (WPE == 1) __syncwarp();
    else __syncthreads();
}
template <int WPE>
__device__ __forceinline__ int xz_thread() { return WPE == 1 ? (int)lane_id() : (int)threadIdx.x; }

__device__ __forceinline__ int xz_det(int l) { return (l < 2 ? DET_X2 : l < 4 ? 22 : 28) - (l & 1); }

__device__ __forceinline__ int xz_list_of(const int *s, int i) {
    int l = 0;
#pragma unroll
    for (int k = 1; k < 6; ++k) l += i >= s[k];
    return l;
}

// x, z and drift of hit f of the index space
__device__ __noinline__ float3 xz_hit_direct(const XzEvent &E, int f, const or_plane_t &P) {
    const int l = xz_list_of(E.start, f), i = f - E.start[l];
    const float dr = E.hc[l].drift(i);
    float X, Z;
    calculate_xz_fy(xz_det(l), (short)E.hc[l].chan(i), dr, 0, 0.f, 0.f, P, X, Z);
    return make_float3(X, Z, dr);
}
__device__ __forceinline__ float3 xz_hit(const XzEvent &E, int f, const or_plane_t &P) {
    if (E.start[6] <= XZ_HITS) return make_float3(E.X[f], E.Z[f], E.drift[f]);
    return xz_hit_direct(E, f, P);
}

// append an entry to bin `key` = station * 28 + bin, in lane order
__device__ __forceinline__ void xz_append(XzEvent &E, bool take, int key, uchar2 v) {
    const unsigned lt = lanemask_lt();
    const unsigned peers = __match_any_sync(0xffffffffu, take ? key : 128 + (int)lane_id());
    int at = 0;
    if (take) {
        at = E.np[0][key];
        const int k = at + __popc(peers & lt);
        if (k < MAXHITS_PROJ_X) E.pairs[0][key][k] = v;
    }
    __syncwarp();
    if (take && (peers & lt) == 0u) E.np[0][key] = at + __popc(peers);
    __syncwarp();
}

// Steps 1 and 2 up to the prefix sums.  False: a plane states more hits than
// the reference's scratch holds (before any hit is read: a view's stride is
// the stated count), or a bin has too many entries.
template <int WPE>
__device__ __forceinline__ bool xz_lists(XzEvent &E, const or_hits_view_t &hv, long e, const or_plane_t &P) {
    const int lane = lane_id(), tid = xz_thread<WPE>(), w = WPE == 1 ? 0 : threadIdx.x >> 5;
    constexpr int NT = 32 * WPE;
    xz_sync<WPE>();  // everyone is done with the previous event
    if (tid < 6) {
        const int d = xz_det(tid) - 1;
        E.hc[tid] = HitPlane{hv.hits_cham + e * OR_EVT_CHAM_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_CHAM * d,
                             (int)hv.nhits_cham[e * OR_NCHAM + d]};
    } else if (tid >= 8 && tid < 18) {
        const int k = tid - 8;
        const int det = k < 4 ? (k == 0 ? DET_P1X1 : k == 1 ? DET_P1X2 : k == 2 ? DET_P2X1 : DET_P2X2)
                              : c_hodoplanesx[((k - 4) >> 1) + 1][k & 1];
        const HitPlane h = hits_of(hv, e, det);
        E.gpos[k] = h.d + h.n;
        E.gn[k] = h.n;
    }
    for (int i = tid; i < 3 * 28; i += NT) E.np[0][i] = 0;
    for (int i = tid; i < (6 * XZ_MAXPLANEHITS + 31) / 32; i += NT) E.paired[i] = 0u;
    xz_sync<WPE>();
    // prefix sums over the planes (lanes 0-5) and the gates' planes (8-17)
    if (w == 0) {
        const int n = lane < 6 ? max(0, E.hc[lane].n) : 0;
        // a gate plane that states more hits than its slot holds is not staged
        const unsigned graw = lane >= 8 && lane < 18 ? (unsigned)E.gn[lane - 8] : 0u;
        const int g = graw > (lane < 12 ? OR_MAXHITS_PROP : OR_MAXHITS_HODO) ? XZ_GATE + 1 : (int)graw;
        int a = n, b = g;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) {
                a += x;
                b += y;
            }
        }
        const int n2 = __shfl_down_sync(0xffffffffu, n, 1);
        int c = lane < 6 && (lane & 1) == 0 ? n * n2 : 0;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c += x;
        }
        if (lane < 7) E.start[lane] = a - n;
        if (lane < 6 && (lane & 1)) E.cpair[(lane >> 1) + 1] = c;
        if (lane == 6) E.cpair[0] = 0;
        const bool many = __any_sync(0xffffffffu, n > XZ_MAXPLANEHITS);
        if (lane == 0) E.over = many;
        // the gates' hits go to shared memory as far as whole planes fit
        if (lane >= 8 && lane < 18) E.goff[lane - 8] = b <= XZ_GATE ? b - g : XZ_GATE;
        if (lane == 18) E.goff[10] = XZ_GATE;
        const unsigned fit = __ballot_sync(0xffffffffu, lane >= 8 && lane < 18 && b <= XZ_GATE);
        const int staged = __shfl_sync(0xffffffffu, b, fit ? last_lane(fit) : 7);
        if (lane == 0) E.staged = fit ? staged : 0;
    }
    xz_sync<WPE>();
    if (E.over) return false;
    const int total = E.start[6];
#pragma unroll 1
    for (int f = tid; f < E.staged; f += NT) {
        int l = 0;
#pragma unroll
        for (int k = 1; k < 10; ++k) l += f >= E.goff[k];
        E.gate[f] = E.gpos[l][f - E.goff[l]];
    }
    if (total <= XZ_HITS) {
#pragma unroll 1
        for (int f = tid; f < total; f += NT) {
            const float3 h = xz_hit_direct(E, f, P);
            E.X[f] = h.x;
            E.Z[f] = h.y;
            E.drift[f] = h.z;
        }
    }
    // pairs: with a CTA per event warp q takes station q
    const int q0 = WPE == 1 ? 0 : w, q1 = WPE == 1 ? 3 : w + 1;
    if (q0 < 3) {
#pragma unroll 1
        for (int b0 = E.cpair[q0]; b0 < E.cpair[q1]; b0 += 32) {
            const int f = b0 + lane;
            bool take = false;
            int key = 0, i = 0, j = 0;
            if (f < E.cpair[q1]) {
                const int q = (f >= E.cpair[1]) + (f >= E.cpair[2]);
                const int n2 = E.start[2 * q + 2] - E.start[2 * q + 1], c = f - E.cpair[q];
                i = c / n2;
                j = c - i * n2;
                if (!(fabsf(E.hc[2 * q].pos(i) - E.hc[2 * q + 1].pos(j)) > c_spacingplane[c_detsuperid[2 + q][0]])) {
                    const int a = E.start[2 * q] + i, b = E.start[2 * q + 1] + j;
                    atomicOr(&E.paired[a >> 5], 1u << (a & 31));
                    atomicOr(&E.paired[b >> 5], 1u << (b & 31));
                    const int bin = x_bin_of(2 + q, E.hc[2 * q].chan(i));
                    take = bin >= 0;
                    key = q * 28 + bin;
                }
            }
            xz_append(E, take, key, make_uchar2((unsigned char)i, (unsigned char)j));
        }
        __syncwarp();
#pragma unroll 1
        for (int b0 = E.start[2 * q0]; b0 < E.start[2 * q1]; b0 += 32) {
            const int f = b0 + lane;
            bool take = false;
            int key = 0;
            uchar2 v = make_uchar2(255, 255);
            if (f < E.start[2 * q1] && !((E.paired[f >> 5] >> (f & 31)) & 1u)) {
                const int l = xz_list_of(E.start, f), i = f - E.start[l];
                const int bin = x_bin_of(2 + (l >> 1), E.hc[l].chan(i));
                take = bin >= 0;
                key = (l >> 1) * 28 + bin;
                if (l & 1) v.y = (unsigned char)i;
                else v.x = (unsigned char)i;
            }
            xz_append(E, take, key, v);
        }
    }
    xz_sync<WPE>();
    if (tid < 10 && E.goff[tid] + E.gn[tid] <= E.staged) E.gpos[tid] = E.gate + E.goff[tid];
    bool over = false;
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {
        const int n = lane < 28 ? E.np[q][lane] : 0;
        over |= __any_sync(0xffffffffu, n > MAXHITS_PROJ_X);
        int a = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= o) a += x;
        }
        if (w == 0 && lane < 29) E.off[q][lane] = a - n;
    }
    xz_sync<WPE>();
    if (over) return false;
    if (w == 0) {
        const int b2 = (lane >> 3) * 7, b3 = ((lane & 7) >> 1) * 7, q3 = 1 + (lane & 1);
        const int n = (E.off[0][b2 + 7] - E.off[0][b2]) * (E.off[q3][b3 + 7] - E.off[q3][b3]);
        int a = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= o) a += x;
        }
        E.tpre[lane] = a - n;
        if (lane == 31) E.tpre[32] = a;
    }
    xz_sync<WPE>();
    return true;
}

// Candidate c: its reference thread t, its cell there (bin2 + 7 bin3) and its
// hits, 11 bits each; returns the hit count.
__device__ __noinline__ int xz_decode(const XzEvent &E, int c, int &t, int &cell, unsigned long long &hits) {
    t = 0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
        if (E.tpre[t + s] <= c) t += s;
    const int b2 = (t >> 3) * 7, b3 = ((t & 7) >> 1) * 7, q3 = 1 + (t & 1);
    const int *o2 = E.off[0] + b2, *o3 = E.off[q3] + b3;
    const int n2 = o2[7] - o2[0];
    int r = c - E.tpre[t];
    const int e3 = r / n2 + o3[0];
    int k3 = 0;
#pragma unroll
    for (int k = 1; k < 7; ++k) k3 += e3 >= o3[k];
    r -= n2 * (o3[k3] - o3[0]);
    const int m3 = E.np[q3][b3 + k3];
    const int e2 = r / m3 + o2[0];
    int k2 = 0;
#pragma unroll
    for (int k = 1; k < 7; ++k) k2 += e2 >= o2[k];
    r -= m3 * (o2[k2] - o2[0]);
    const int m2 = E.np[0][b2 + k2];
    const int i3 = r / m2, i2 = r - i3 * m2;
    cell = k2 + 7 * k3;
    const uchar2 p2 = E.pairs[0][b2 + k2][i2], p3 = E.pairs[q3][b3 + k3][i3];
    hits = 0ull;
    int nh = 0;
    auto push = [&](int l, int i) {
        hits |= (unsigned long long)(E.start[l] + i) << (11 * nh);
        ++nh;
    };
    if (p2.x != 255) push(0, p2.x);
    if (p2.y != 255) push(1, p2.y);
    if (p3.x != 255) push(2 * q3, p3.x);
    if (p3.y != 255) push(2 * q3 + 1, p3.y);
    return nh;
}
__device__ __forceinline__ int xz_code(unsigned long long hits, int k) { return (int)(hits >> (11 * k)) & 0x7FF; }

// Scratch entries 2 and 3 (low and high half: hit index, 0xFFFF = none) of
// thread t.
struct XzStale {
    int t;
    unsigned e;
};

// The fit of a candidate's hits, with the drift distances when `signs` >= 0.
__device__ __noinline__ void xz_fit(const XzEvent &E, const or_plane_t &P, unsigned long long hits, int nh, int signs,
                                    float &x0, float &tx, float &ex0, float &etx) {
    Fit2 f;
#pragma unroll 1
    for (int k = 0; k < nh; ++k) {
        const int h = xz_code(hits, k);
        const float3 v = xz_hit(E, h, P);
        const float w = P.resolution[xz_det(xz_list_of(E.start, h))];
        if (signs < 0) f.add(v.x, v.y, w);
        else f.add_drift(v.x, v.z, (short)((signs << (30 - 2 * k)) >> 30), v.y, w);
    }
    f.solve(x0, tx, ex0, etx);
}

// The left/right walk, the second fit and the gates (K:547-672) of n <= 32
// candidates from the ring; returns whether the lane's candidate stays, with
// its fit and signs in c.
__device__ __noinline__ bool xz_finish(const XzEvent &E, const or_plane_t &P, XzCand &c, bool valid) {
    if (!valid) return false;
    const int nh = (int)(c.place >> 16) & 7;
    int signs = 0;
    float x0 = c.x0, tx = c.tx, ex0 = c.ex0, etx = c.etx;
    auto det_of = [&](int h) { return xz_det(xz_list_of(E.start, h)); };
    // resolve_leftright_xhits walk (H:820-871)
#pragma unroll 1
    for (int n = 0; n < nh;) {
        const int j = n + 1;
        const int hi = xz_code(c.hits, n), hj = j < nh ? xz_code(c.hits, j) : (int)c.stale;
        const int di = det_of(hi), dj = hj == 0xFFFF ? (int)DET_SENTINEL : det_of(hj);
        if (abs(di - dj) != 1) {
            n += 1;
            continue;
        }
        const float3 a = xz_hit(E, hi, P), b = xz_hit(E, hj, P);
        const int k = lr_pair_xhits(x0, tx, ex0, etx, (short)di, (short)dj, a.x, a.z, b.x, b.z, P.z, 150.f);
        if (k >= 0) {
            signs |= (c_lrpossibility[k][0] & 3) << (2 * n);
            if (j < nh) signs |= (c_lrpossibility[k][1] & 3) << (2 * j);
        }
        n += 2;
    }
#pragma unroll 1
    for (int k = 0; k < nh; ++k) {
        if ((signs >> (2 * k)) & 3) continue;
        const int h = xz_code(c.hits, k);
        signs |= (single_sign_xhits(x0, tx, (short)det_of(h), xz_hit(E, h, P).x, P.z) & 3) << (2 * k);
    }
    xz_fit(E, P, c.hits, nh, signs, x0, tx, ex0, etx);
    if (fabsf(x0) > X0_MAX || fabsf(tx) > TX_MAX) return false;
    c.x0 = x0;
    c.tx = tx;
    c.ex0 = ex0;
    c.etx = etx;
    c.place |= (unsigned)signs << 24;
    // prop tubes (K:577-640)
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
        bool ok = false;
#pragma unroll 1
        for (int k = 2 * s; k < 2 * s + 2 && !ok; ++k) {
            const float ex = tx * P.z[DET_P1X1 - k + (k > 1 ? 4 : 0)] + x0;
            const float *p = E.gpos[k];
            const int n = E.gn[k];
#pragma unroll 1
            for (int i = 0; i < n && !ok; ++i) ok = fabsf(p[i] - ex) < (s ? 7.62f : 5.08f);
        }
        if (!ok) return false;
    }
    // hodoscopes (H:1090-1144): the plane's positions are the second field of
    // a view
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {
        bool ok = false;
#pragma unroll 1
        for (int k = 0; k < 2 && !ok; ++k) {
            const int n = E.gn[4 + 2 * q + k];
            ok = match_track_XZ_to_hodo(q + 1, c_hodoplanesx[q + 1][k], HitPlane{E.gpos[4 + 2 * q + k] - n, n}, x0, tx, ex0,
                                        etx, P.z);
        }
        if (!ok) return false;
    }
    return true;
}

// Write tracklet c as number k of station-3 half p; every lane of the warp
// with the same arguments.
__device__ __noinline__ void xz_write(XzWarp &S, const XzEvent &E, const or_plane_t &P, const or_tracks_view_t &tv,
                                      long e, const XzCand &c, int k) {
    const int lane = lane_id();
    const int t = (int)(c.place & 255u), cell = (int)(c.place >> 8) & 255, nh = (int)(c.place >> 16) & 7;
    const int slot = 2 * (k % 16) + (t & 1), posn = k / 16;
    if (posn >= OR_SLOTCAP) return;
#pragma unroll
    for (int f = lane; f < OR_NTRKPARAM; f += 32) S.rec[f] = 0.f;
    __syncwarp();
    if (lane < nh) {
        const int h = xz_code(c.hits, lane), l = xz_list_of(E.start, h), i = h - E.start[l];
        const float3 v = xz_hit(E, h, P);
        S.rec[OR_TRK_HIT_DETID + lane] = (float)xz_det(l);
        S.rec[OR_TRK_HIT_CHAN + lane] = (float)(short)E.hc[l].chan(i);
        S.rec[OR_TRK_HIT_POS + lane] = v.x;
        S.rec[OR_TRK_HIT_DRIFT + lane] = v.z;
        S.rec[OR_TRK_HIT_SIGN + lane] = (float)((int)((c.place >> 24) << (30 - 2 * lane)) >> 30);
        S.rec[OR_TRK_HIT_TDC + lane] = E.hc[l].tdc(i);
    } else if (lane == 8) {
        S.rec[OR_TRK_STID] = (float)(t + 32 * cell);
        S.rec[OR_TRK_THREAD] = (float)t;
        S.rec[OR_TRK_NHITS] = (float)nh;
        S.rec[OR_TRK_TX] = c.tx;
        S.rec[OR_TRK_X0] = c.x0;
        S.rec[OR_TRK_ERR_TX] = c.etx;
        S.rec[OR_TRK_ERR_X0] = c.ex0;
    }
    __syncwarp();
    float *r = trk_rec(tv, e, slot, posn);
#pragma unroll
    for (int f = lane; f < OR_NTRKPARAM; f += 32) r[f] = S.rec[f];
    __syncwarp();
}

// Steps 2 to 4 for candidates [c0, c1): the surviving tracklets go, in order,
// to `sink(candidate of lane src, parity)`, called by the whole warp.
template <class Sink>
__device__ __forceinline__ void xz_walk(XzWarp &S, const XzEvent &E, const or_plane_t &P, int c0, int c1, XzStale cs,
                                        Sink sink) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    int head = 0, waiting = 0;
#pragma unroll 1
    for (int base = c0;; base += 32) {
        const bool more = base < c1;
        if (more) {
            const int c = base + lane;
            const bool valid = c < c1;
            int t = 32 + lane, cell = 0, nh = 0;  // distinct keys for invalid lanes
            unsigned long long hits = 0ull;
            if (valid) nh = xz_decode(E, c, t, cell, hits);
            // segmented last-writer scan of scratch entries 2 and 3
            const unsigned same = __match_any_sync(0xffffffffu, t);
            const unsigned w2 = __ballot_sync(0xffffffffu, nh >= 3), w3 = __ballot_sync(0xffffffffu, nh == 4);
            const unsigned mine = (nh >= 3 ? (unsigned)xz_code(hits, 2) : 0xFFFFu) |
                                  (nh == 4 ? (unsigned)xz_code(hits, 3) : 0xFFFFu) << 16;
            const int l2 = last_lane(w2 & same & lt), l3 = last_lane(w3 & same & lt);
            const unsigned s2 = __shfl_sync(0xffffffffu, mine, l2 < 0 ? 0 : l2);
            const unsigned s3 = __shfl_sync(0xffffffffu, mine, l3 < 0 ? 0 : l3);
            const unsigned ce = t == cs.t ? cs.e : ~0u;
            const unsigned e2 = l2 >= 0 ? s2 & 0xFFFFu : ce & 0xFFFFu, e3 = l3 >= 0 ? s3 >> 16 : ce >> 16;
            {  // state after the last valid lane
                const int last = min(31, c1 - 1 - base);
                const int tl = __shfl_sync(0xffffffffu, t, last);
                const unsigned seg = __shfl_sync(0xffffffffu, same, last);
                const unsigned old = tl == cs.t ? cs.e : ~0u;
                const int a2 = last_lane(w2 & seg), a3 = last_lane(w3 & seg);
                const unsigned n2 = __shfl_sync(0xffffffffu, mine, a2 < 0 ? 0 : a2);
                const unsigned n3 = __shfl_sync(0xffffffffu, mine, a3 < 0 ? 0 : a3);
                cs.e = (a2 >= 0 ? n2 & 0xFFFFu : old & 0xFFFFu) | (a3 >= 0 ? n3 & 0xFFFF0000u : old & 0xFFFF0000u);
                cs.t = tl;
            }
            bool pass = false;
            XzCand o;
            if (valid) {
                xz_fit(E, P, hits, nh, -1, o.x0, o.tx, o.ex0, o.etx);
                pass = !(fabsf(o.x0) > X0_MAX + 2 * o.ex0 || fabsf(o.tx) > TX_MAX + 2 * o.etx);
            }
            const unsigned pm = __ballot_sync(0xffffffffu, pass);
            if (pass) {
                o.hits = hits;
                o.stale = nh == 2 ? e2 : nh == 3 ? e3 : 0xFFFFu;
                o.place = (unsigned)t | (unsigned)cell << 8 | (unsigned)nh << 16;
                S.ring[(head + waiting + __popc(pm & lt)) & 63] = o;
            }
            waiting += __popc(pm);
            __syncwarp();
        }
        if (waiting >= 32 || (!more && waiting > 0)) {
            const int n = min(waiting, 32);
            XzCand c = S.ring[(head + lane) & 63];
            const bool keep = xz_finish(E, P, c, lane < n);
            if (keep) S.ring[(head + lane) & 63] = c;
            const unsigned km = __ballot_sync(0xffffffffu, keep);
            __syncwarp();
#pragma unroll 1
            for (unsigned m = km; m; m &= m - 1) sink(S.ring[(head + __ffs(m) - 1) & 63]);
            __syncwarp();
            head = (head + 32) & 63;
            waiting -= n;
        }
        if (!more && waiting == 0) break;
    }
}

// counts and overflow (K:812-839), one warp
__device__ __forceinline__ void xz_counts(const or_tracks_view_t &tv, long e, int kpar0, int kpar1,
                                          int32_t *__restrict__ ntracklets, uint8_t *__restrict__ toomany) {
    const int lane = lane_id();
    const int ntot = kpar0 + kpar1;
    const bool full = ntot >= OR_TRKMAX || kpar0 > 16 * OR_SLOTCAP || kpar1 > 16 * OR_SLOTCAP;
    const int m = lane >> 1, K = (lane & 1) ? kpar1 : kpar0;
    tv.ntracks[e * OR_NSLOTS + lane] = full ? 0 : (uint16_t)(K > m ? (K - m + 15) / 16 : 0);
    if (lane == 0) {
        ntracklets[e] = ntot;
        if (full) toomany[e] = 1;
    }
}

// An event not reconstructed: no tracklets (K:195-200), or a plane or a bin
// with too many entries.  On its own the stage leaves a flagged event's
// tracklet count as it stands, as the reference's kernel does; a whole-chain
// call (`chain`) wants it cleared.
__device__ __forceinline__ void xz_reject(const or_tracks_view_t &tv, long e, bool over, bool chain,
                                          int32_t *__restrict__ ntracklets, uint8_t *__restrict__ toomany) {
    tv.ntracks[e * OR_NSLOTS + lane_id()] = 0;
    if (lane_id() == 0) {
        if (over) toomany[e] = 1;
        if (over || chain) ntracklets[e] = 0;
    }
}

#ifndef OR_XZ_WARPS_SM
#define OR_XZ_WARPS_SM 16
#endif

#ifndef OR_XZ_TEAM_PER_SM
#define OR_XZ_TEAM_PER_SM 8
#endif

struct XzSlot {
    XzEvent ev;
    XzWarp warp;
};

template <int W>
__global__ void __launch_bounds__(W * 32, (OR_XZ_WARPS_SM / W > 0 ? OR_XZ_WARPS_SM / W : 1))
    xz_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv,
              int32_t *__restrict__ ntracklets, uint8_t *__restrict__ toomany, int n_events, bool chain) {
    extern __shared__ __align__(16) unsigned char xz_smem[];
    or_plane_t &P = *reinterpret_cast<or_plane_t *>(xz_smem);
    XzSlot *slots = reinterpret_cast<XzSlot *>(xz_smem + ((sizeof(or_plane_t) + 15) & ~size_t(15)));
    load_plane_smem(&P, gplane);
    __syncthreads();
    const int w = threadIdx.x >> 5;
    XzEvent &E = slots[w].ev;
    XzWarp &S = slots[w].warp;
    for (long e = (long)blockIdx.x * W + w; e < n_events; e += (long)gridDim.x * W) {
        if (toomany[e]) {  // K:195-200
            xz_reject(tv, e, false, chain, ntracklets, toomany);
            continue;
        }
        if (!xz_lists<1>(E, hv, e, P)) {
            xz_reject(tv, e, true, chain, ntracklets, toomany);
            continue;
        }
        int kpar0 = 0, kpar1 = 0;
        xz_walk(S, E, P, 0, E.tpre[32], XzStale{-1, ~0u}, [&](const XzCand &c) {
            const bool odd = c.place & 1u;
            xz_write(S, E, P, tv, e, c, odd ? kpar1 : kpar0);
            kpar0 += !odd;
            kpar1 += odd;
        });
        xz_counts(tv, e, kpar0, kpar1, ntracklets, toomany);
    }
}

struct XzTeam {
    XzEvent ev;
    XzWarp warp[XZ_TEAM];
    XzCand stash[XZ_TEAM][XZ_STASH];
    int n[XZ_TEAM][2];
};

// One event per CTA: what small batches run, where most SMs would hold one
// warp or none.
__global__ void __launch_bounds__(XZ_TEAM * 32)
    xz_team_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv,
                   int32_t *__restrict__ ntracklets, uint8_t *__restrict__ toomany, int n_events, bool chain) {
    extern __shared__ __align__(16) unsigned char xz_smem[];
    or_plane_t &P = *reinterpret_cast<or_plane_t *>(xz_smem);
    XzTeam &M = *reinterpret_cast<XzTeam *>(xz_smem + ((sizeof(or_plane_t) + 15) & ~size_t(15)));
    load_plane_smem(&P, gplane);
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    XzEvent &E = M.ev;
    XzWarp &S = M.warp[w];
    for (long e = blockIdx.x; e < n_events; e += gridDim.x) {
        const bool rejected = toomany[e];
        __syncthreads();  // every warp has read the flag before one of them sets it
        if (rejected) {
            if (w == 0) xz_reject(tv, e, false, chain, ntracklets, toomany);
            continue;
        }
        if (!xz_lists<XZ_TEAM>(E, hv, e, P)) {
            if (w == 0) xz_reject(tv, e, true, chain, ntracklets, toomany);
            continue;
        }
        // the warp's run of candidates: whole chunks, shared out evenly
        const int total = E.tpre[32], chunks = (total + 31) / 32;
        const int c0 = min(total, chunks * w / XZ_TEAM * 32), c1 = min(total, chunks * (w + 1) / XZ_TEAM * 32);
        // scratch entries of the run's first thread, from the candidates before
        XzStale cs{-1, ~0u};
        if (c0 < c1 && c0 > 0) {
            unsigned long long hits;
            int cell;
            xz_decode(E, c0, cs.t, cell, hits);
#pragma unroll 1
            for (int b = c0 - 32; b > E.tpre[cs.t] - 32 && ((cs.e & 0xFFFFu) == 0xFFFFu || (cs.e >> 16) == 0xFFFFu); b -= 32) {
                const int c = b + lane;  // b >= 0: c0 is a multiple of 32 and tpre >= 0
                int t, nh = 0;
                unsigned mine = ~0u;
                if (c >= E.tpre[cs.t]) {
                    nh = xz_decode(E, c, t, cell, hits);
                    mine = (nh >= 3 ? (unsigned)xz_code(hits, 2) : 0xFFFFu) |
                           (nh == 4 ? (unsigned)xz_code(hits, 3) : 0xFFFFu) << 16;
                }
                const unsigned w2 = __ballot_sync(0xffffffffu, nh >= 3), w3 = __ballot_sync(0xffffffffu, nh == 4);
                const unsigned m2 = __shfl_sync(0xffffffffu, mine, w2 ? last_lane(w2) : 0);
                const unsigned m3 = __shfl_sync(0xffffffffu, mine, w3 ? last_lane(w3) : 0);
                if ((cs.e & 0xFFFFu) == 0xFFFFu && w2) cs.e = (cs.e & 0xFFFF0000u) | (m2 & 0xFFFFu);
                if ((cs.e >> 16) == 0xFFFFu && w3) cs.e = (cs.e & 0xFFFFu) | (m3 & 0xFFFF0000u);
            }
        }
        int k0 = 0, k1 = 0;
        xz_walk(S, E, P, c0, c1, cs, [&](const XzCand &c) {
            const int k = k0 + k1;
            if (k < XZ_STASH && lane == 0) M.stash[w][k] = c;
            k0 += !(c.place & 1u);
            k1 += c.place & 1u;
        });
        if (lane == 0) {
            M.n[w][0] = k0;
            M.n[w][1] = k1;
        }
        __syncthreads();
        int p0 = 0, p1 = 0, n0 = 0, n1 = 0;
        bool fits = true;
#pragma unroll 1
        for (int i = 0; i < XZ_TEAM; ++i) {
            if (i == w) {
                p0 = n0;
                p1 = n1;
            }
            n0 += M.n[i][0];
            n1 += M.n[i][1];
            fits &= M.n[i][0] + M.n[i][1] <= XZ_STASH;
        }
        if (fits) {
#pragma unroll 1
            for (int k = 0; k < k0 + k1; ++k) {
                const XzCand c = M.stash[w][k];
                const bool odd = c.place & 1u;
                xz_write(S, E, P, tv, e, c, odd ? p1 : p0);
                p0 += !odd;
                p1 += odd;
            }
        } else if (w == 0) {  // more tracklets than a warp keeps: one warp walks them again
            p0 = p1 = 0;
            xz_walk(S, E, P, 0, total, XzStale{-1, ~0u}, [&](const XzCand &c) {
                const bool odd = c.place & 1u;
                xz_write(S, E, P, tv, e, c, odd ? p1 : p0);
                p0 += !odd;
                p1 += odd;
            });
        }
        if (w == 0) xz_counts(tv, e, n0, n1, ntracklets, toomany);
        __syncthreads();
    }
}

size_t xz_smem_bytes(int warps) {
    return ((sizeof(or_plane_t) + 15) & ~size_t(15)) + sizeof(XzSlot) * (size_t)warps;
}

template <int W>
static cudaError_t xz_launch(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv, int32_t *ntracklets,
                             uint8_t *toomany, int n_events, cudaStream_t stream, int sm_count, bool chain) {
    const size_t smem = xz_smem_bytes(W);
    cudaError_t err = smem_attr_once((const void *)xz_kernel<W>, (int)smem);
    if (err != cudaSuccess) return err;
    long blocks = (n_events + W - 1) / W;
    // An event per warp, as blocks come free, evens out events of different
    // size; on large batches loading the planes for every block costs more
    // than that (W = 4, uneven events, resident blocks that go round -> a block
    // per W events: 10,000 820 -> 702 us, 20,000 1,248 -> 1,231, 40,000 1,906
    // -> 2,238).
    const long cap = (long)sm_count * (32 / W > 0 ? 32 / W : 1);
    if (blocks > cap && n_events > 128 * sm_count) blocks = cap;
    xz_kernel<W><<<(unsigned)blocks, W * 32, smem, stream>>>(d_plane, hv, tv, ntracklets, toomany, n_events,
                                                               chain);
    return cudaGetLastError();
}

// `warps` = events per CTA: 1, 2, 4 or 8 (the per-warp scratch is too large for
// 16); `chain`: every event's tracklet count is written (xz_reject)
cudaError_t launch_xz(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv, int32_t *ntracklets,
                      uint8_t *toomany, int n_events, cudaStream_t stream, int sm_count, int warps, bool chain) {
    if (n_events <= 0) return cudaSuccess;
    // A CTA per event on small batches, where a warp per event leaves a heavy
    // event's chain to itself: 333 uneven events 238 -> 83 us, 1,000 of them
    // 271 -> 96 us and 1,000 one-dimuon events 84 -> 61 us.  From some
    // thousands of events on light ones pay for it (4,000 one-dimuon events
    // 125 -> 196 us, 4,000 uneven ones 420 -> 268 us).
    if (n_events <= OR_XZ_TEAM_PER_SM * sm_count) {
        const size_t smem = ((sizeof(or_plane_t) + 15) & ~size_t(15)) + sizeof(XzTeam);
        cudaError_t err = smem_attr_once((const void *)xz_team_kernel, (int)smem);
        if (err != cudaSuccess) return err;
        xz_team_kernel<<<(unsigned)n_events, XZ_TEAM * 32, smem, stream>>>(d_plane, hv, tv, ntracklets, toomany,
                                                                           n_events, chain);
        return cudaGetLastError();
    }
    switch (warps) {
    case 1: return xz_launch<1>(d_plane, hv, tv, ntracklets, toomany, n_events, stream, sm_count, chain);
    case 2: return xz_launch<2>(d_plane, hv, tv, ntracklets, toomany, n_events, stream, sm_count, chain);
    case 8: return xz_launch<8>(d_plane, hv, tv, ntracklets, toomany, n_events, stream, sm_count, chain);
    default: return xz_launch<4>(d_plane, hv, tv, ntracklets, toomany, n_events, stream, sm_count, chain);
    }
}

}  // namespace orgpu
