// yz_kernel.cu -- YZ extension of the XZ tracklets with U/V hits.
//
// Replaces gKernel_YZ_tracking<<<N,32>>> (OnlineReconstruction/
// reconstruction_kernels.cuh:864-1832).
//
// The reference gives each of its 32 threads one tracklet slot and, for every
// tracklet in it, loops u3 x v3 (outer) and u2 x v2 (inner) hit pairs
// sequentially, keeping the best chi2 (K:1320-1825).  Two pieces of state
// make that loop sequential:
//   - the station-3 hit signs chosen by the left/right resolution survive
//     from one inner iteration to the next: they are fixed by the first
//     combination of a (u3,v3) iteration that passes the first y cut, and on
//     station 3+ the last v3' hit can pair with the first u2 hit
//     (planes 19/18), whose resolution re-sets that sign whenever it
//     succeeds (H:714-780);
//   - the left/right walk reads the scratch entry just past the hit count
//     (H:725-735), which holds the last hit load attempted at that index --
//     possibly by an earlier combination, (u3,v3) iteration or tracklet of
//     the same slot.
// Work per event is heavily skewed (a few events hold most combinations),
// so the GPU version splits it:
//   yz_plan_kernel   a warp per slot (per eight slots with the combination
//                    scorer's rows) walks its tracklets in order; builds each
//                    one's hit windows once (y, error and acceptance of every
//                    windowed hit for this tracklet) and cuts it into units
//                    of whole (u3,v3) iterations on a device queue, storing
//                    its windows as an image; with the scorer's rows it
//                    evaluates light tracklets itself;
//   yz_first_kernel  persistent warps (28 per SM, 72 registers) drain the
//                    queue with the first cut (fit of the station-3 and
//                    station-2 y hits, 2-sigma cut) and the prop-tube and
//                    hodoscope gates; the survivors that pass, and those that
//                    set station-3 signs for them, go in order to a device
//                    pool; with the combination scorer it walks only the
//                    kept (u3,v3) iterations;
//   yz_second_kernel per unit, those survivors replayed in order with the
//                    sign carry: left/right walk and chi2 (28 warps per SM,
//                    72 registers; a survivor's hits are register offsets
//                    into the arena); a unit whose survivors did not fit runs
//                    whole, first cut and survivors together
//                    (yz_work_kernel's path, which also serves contexts
//                    without a pool, such as the no-allocation entry); the
//                    best combination of a tracklet of one unit is written
//                    here;
//   yz_apply_kernel  writes the best combination of tracklets of several
//                    units.
// Inside a range, lanes evaluate 32 combinations at a time in the reference
// order; ballot/shuffle scans recover the sign state and the scratch entry.
// A unit starts with the scratch entries left by everything before it, which
// depend only on which hit loads were attempted (not on any fit), so the plan
// pass and each unit derive them without evaluating the earlier work.  The
// best combination of a tracklet is the minimum of (chi2, combination index),
// the reference's first-strictly-smaller rule.
#include <type_traits>

#include "window_pairs.cuh"

namespace orgpu {

constexpr int YZ_MAXWIN = 100;          // windowed hits per plane (the reference's hitidx arrays)
constexpr int YZ_MAXPAIR = 100;         // pairs per projection (the reference's hitpairs arrays)
// Build-time tunables (-D...); results do not depend on any of them.  On the
// present kernels and the 100,000-event uneven batch: first cut 8.9 / 9.2 /
// 9.9 ms at 28 / 24 / 20 warps per SM, survivors 6.2 / 6.6 / 7.4, planning 5.3
// / 5.1 / 5.8; units of 1,024 / 4,096 / 8,192 / 16,384 combinations 28.6 / 21.4
// / 20.4 / 20.4 ms (the three together).  The others were chosen on earlier
// forms of the kernels.
//   OR_YZ_ARENA          windowed hit records per warp in shared memory
//   OR_YZ_WARPS_SM       warps per SM of the combined work kernel
//   OR_YZ_SPLIT          first-cut / survivor kernels (1) or the combined one (0)
//   OR_YZ_PLAN_WARPS_SM, OR_YZ_FIRST_WARPS_SM, OR_YZ_SECOND_WARPS_SM
//                        warps per SM (register caps) of the other kernels
//   OR_YZ_POOL_PER_UNIT  survivor-pool entries per unit of queue capacity
//   OR_YZ_IMG_PER_UNIT   window-image 16-byte words per unit of queue capacity
//   OR_YZ_LIGHT          combinations a planning warp evaluates itself
//   OR_YZ_PLAN_CHUNK     slots per planning unit
//   OR_YZ_UNIT           live combinations per queued unit
//   OR_YZ_QCAP_CTX       per-warp survivor queue entries of a context
#ifndef OR_YZ_ARENA
#define OR_YZ_ARENA 64
#endif
#ifndef OR_YZ_WARPS_SM
#define OR_YZ_WARPS_SM 16
#endif
#ifndef OR_YZ_SPLIT
#define OR_YZ_SPLIT 1
#endif
#ifndef OR_YZ_PLAN_WARPS_SM
#define OR_YZ_PLAN_WARPS_SM 28
#endif
#ifndef OR_YZ_FIRST_WARPS_SM
#define OR_YZ_FIRST_WARPS_SM 28
#endif
#ifndef OR_YZ_POOL_PER_UNIT
#define OR_YZ_POOL_PER_UNIT 48
#endif
// survivor entries in the pool (16 B each), per unit of queue capacity: a
// context sized for the 100,000-event uneven batch (4 Mi units) holds
// 192 Mi, several times what that batch passes on; units that do not fit run
// on the combined path
constexpr long long YZ_POOL_PER_UNIT = OR_YZ_POOL_PER_UNIT;
#ifndef OR_YZ_IMG_PER_UNIT
#define OR_YZ_IMG_PER_UNIT 80
#endif
// window images (16-byte words) per unit of queue capacity: 320 Mi words
// (5 GiB) for 4 Mi units, and the 100,000-event uneven batch's queued
// tracklets take 128 Mi words (1.9 GiB); the units of tracklets whose image
// does not fit run on the combined path
constexpr long long YZ_IMG_PER_UNIT = OR_YZ_IMG_PER_UNIT;
constexpr int YZ_ARENA_HITS = OR_YZ_ARENA;      // windowed hits kept in shared memory per warp
#ifndef OR_YZ_LIGHT
#define OR_YZ_LIGHT 32
#endif
constexpr long YZ_LIGHT = OR_YZ_LIGHT;         // combinations a planning warp evaluates itself per tracklet
constexpr long YZ_CHUNK_INLINE = OR_YZ_LIGHT;  // ... and per planning unit
#ifndef OR_YZ_PLAN_CHUNK
#define OR_YZ_PLAN_CHUNK 1
#endif
constexpr int YZ_PLAN_CHUNK = OR_YZ_PLAN_CHUNK;  // slots per planning unit
constexpr int YZ_PLAN_CHUNK_SCORED = 8;          // ... with the combination scorer
#ifndef OR_YZ_UNIT
#define OR_YZ_UNIT 8192
#endif
constexpr long YZ_UNIT = OR_YZ_UNIT;    // live combinations per queued unit (whole (u3,v3) iterations)
constexpr int YZ_GARENA_HITS = 8 * YZ_MAXWIN;  // per-warp global overflow arena
static_assert(OR_MAXHITS_CHAM <= 256, "a chamber plane's hit index fits a byte");
// survivors of the first cut wait in a per-warp queue in global memory and
// are evaluated in a batch when it fills or the range ends, so that the two
// phases do not alternate every 32 survivors (each switch refetches the
// other phase's instructions)
constexpr int YZ_QCAP_MIN = 64;     // queue entries per warp: the static (no-allocation) scratch
#ifndef OR_YZ_QCAP_CTX
#define OR_YZ_QCAP_CTX 2048
#endif
constexpr int YZ_QCAP_CTX = OR_YZ_QCAP_CTX;   // ... and a context's scratch

struct __align__(16) YzHit {
    float Y, eY, pos, drift;
    float tdc, z;  // z = the plane's z, read by every fit
    short det, el;
    int acc;  // calculate_y_uvhit accepted this hit for the tracklet
};
static_assert(sizeof(YzHit) == 32, "YzHit is two 16-byte words");

struct Stale {
    short det;
    float pos, drift;
};

// one queued unit: combinations [g0*C2, g1*C2) of heavy tracklet `heavy`,
// with the scratch entries 4..7 as they stand when the unit starts
struct YzUnit {
    int heavy;
    int g0, g1;
    int pad;
    Stale entry[4];
    // the unit's live outer iterations as the combination scorer's rows of
    // its tracklet: ranks [r0, r1)
    int r0, r1;
};
// a heavy tracklet
struct YzHeavy {
    int e, slot, k;
    int unit0, nunits;
    // outer-iteration scoring: the tracklet's first score row (-1: no rows,
    // nothing pruned), its row count (the live outer iterations), the inner
    // combinations per outer iteration, and the outer index of its best
    // combination (written with that combination by yz_finish; -1: none)
    int orow0, nrows, c2, best_g;
    // its window image in the image pool (16-byte words), -1: none
    int img;
};
// best combination of one unit
struct YzBest {
    unsigned long long key;
    int nuv;
    float chi2, ty, y0, ety, ey0;
    float det[8], el[8], pos[8], drift[8], sign[8], tdc[8], res[12];
    int pad;
};

// The first y fit of a combination (fit_2D_track over its accepted u/v hits,
// K:1602, AM:32-74) weighs every hit by its plane's error (calculate_y_uvhit,
// H:98: resolution * |dp_y / dp_x|) at its plane's z, so the normal matrix,
// its inverse and the parameter errors depend only on which of the eight
// planes (u3 u3' v3 v3' u2 u2' v2 v2', added in that order) gave a hit.  The
// fit needs at least one hit in each of the four projections: 3^4 = 81 plane
// sets per station-3 half.  yz_tab_kernel computes each entry with the same
// operations in the same order as the per-combination fit did (Fit2 then
// matinv_2x2 and sqrtf), so a combination's fit keeps only the right-hand
// side (B0, B1) and two dot products, bit for bit the same result.
constexpr int YZ_TAB_SETS = 81;
struct __align__(16) YzTab {
    float ai0, ai1, ai2, ai3;  // inverse of the normal matrix
    float thr_y0, thr_ty;      // Y0_MAX + 2 err_y0, TY_MAX + 2 err_ty (the first cut, K:1611)
    float ey0, ety;            // err_y0, err_ty
};
static_assert(sizeof(YzTab) == 32, "YzTab is two 16-byte words");
constexpr size_t YZ_TAB_BYTES = (2 * YZ_TAB_SETS * sizeof(YzTab) + 255) & ~size_t(255);

// index of a plane set: group values g = (second plane << 1 | first plane)
// in 1..3 for u3, v3, u2, v2
__device__ __forceinline__ int yz_tab_index(int gu3, int gv3, int gu2, int gv2) {
    return ((gu3 - 1) * 3 + (gv3 - 1)) * 9 + (gu2 - 1) * 3 + (gv2 - 1);
}

// Work counters of one YZ call (64-bit, in the counters area): combinations
// that reach the first y fit, the sum of their hit counts, and combinations
// that pass its 2-sigma cut (the survivors of the first cut).
constexpr int YZ_CTR_FITTED = 16, YZ_CTR_HITSUM = 18, YZ_CTR_SURVIVORS = 20;

struct YzScratch {
    const YzTab *tab;        // 2 x YZ_TAB_SETS entries: station-3 half 0 (D3p) then 1 (D3m)
    unsigned *list;          // planning units with tracklets; nullptr: every unit is visited
    YzUnit *units;
    YzHeavy *heavy;
    YzBest *best;
    unsigned int *counters;  // [0] units reserved, [1] heavy reserved, [2] queue head, [3] survivor-kernel
                             // head, [4..5] planning units taken, [6], [7] planning units listed (front, back), [8..9] pool entries, [10..11] image words,
                             // [16..21] work counters
    YzHit *garena;           // per-warp overflow arenas
    struct PassEntryStore *qbuf;  // per-warp survivor queues (qcap entries each)
    int cap_units, cap_heavy, garena_warps, qcap;
    // split first-cut / survivor kernels: each unit's survivors in order in
    // pool[useg[u].x .. + useg[u].y); useg[u].x < 0: the unit runs combined
    struct YzSurv *pool;
    int2 *useg;
    long long pool_cap;  // 0: no pool, the combined kernel runs
    // window images of the queued tracklets (YzImgHead, arena, pairs),
    // written by the planning pass; counter [10..11] allocates them
    uint4 *img;
    long long img_cap;   // 16-byte words; 0: no images, every unit windows its tracklet
    int count_work;      // nonzero: the kernels add up the work counters
};

// optional pruning: tracklet rows (row_off, as the scorer's) and keep flags
struct YzPrune {
    // tracklet keep flags of the tracklet scorer
    const int32_t *row_off;
    const uint8_t *keep;  // nullptr: plain
    long max_rows;
    // the combination scorer: one feature row per live (u3, v3) outer
    // iteration of every queued (heavy) tracklet, written by the planning
    // pass; scores filled before the first cut; an outer iteration scoring
    // below t_keep is skipped, unless its event is uncertain (unc[e])
    float *ofeat;          // [cap_orows * OR_NFEAT]; nullptr: no outer rows
    int32_t *og;           // [cap_orows] outer index g of each row
    float *oscore;         // [cap_orows]
    uint32_t *orows;       // row counter
    uint8_t *unc;          // [n_events] uncertain events
    const or_mlp_t *model; // nullptr: rows written, nothing scored or pruned
    long cap_orows;
    float t_keep, t_unc;
};


struct PassEntryStore {
    int c;
    float y0, ty, ey0, ety, stpos, stdrift;
    int stdet;
};

// A survivor as the first-cut kernel hands it to the survivor kernel: its
// four pairs (7 bits each: u3, v3, u2, v2), its first fit, and a code: bits
// 0-9 the arena offset of the scratch entry past its hit count, bits 10-11
// where that entry stands (YZ_ENT_*), bits 12-13 the unit's starting entry
// (4..7) when it stands there, bits 14-20 the plane set's table index, bits
// 22-29 the planes that give a hit (u3 u3' v3 v3' u2 u2' v2 v2'), bit 31
// whether the gates passed (a survivor that fails them is only kept for the
// station-3 signs it sets).
struct __align__(16) YzSurv {
    unsigned pairs;
    float y0, ty;
    unsigned code;
};
static_assert(YZ_MAXPAIR <= 128, "a pair index fits 7 bits");
constexpr unsigned YZ_ENT_HIT = 1u, YZ_ENT_UNIT = 2u;  // 0: no such entry

struct YzEvent {
    HitPlane hc[8];
    HitPlane p1y1, p1y2, p2y1, p2y2;
    HitPlane hod[3][2];
    short dl[8];
};

// What the lanes exchange while a chunk of survivors is evaluated
struct YzPhase2 {
    float term[16 * 12];      // chi2 terms
    signed char res[32 * 8];  // per survivor and hit: the pair's resolution or the hit's sign
    unsigned char item[32 * 8];
};

struct YzWarp {
    YzEvent ev;  // the event's plane views, the same for every lane
    Stale st[4];  // scratch entries 4..7 as the next combination finds them, the same for every lane
    YzHit arena[YZ_ARENA_HITS];
    short2 pair[4][YZ_MAXPAIR];  // windowed indices (or -1) in sides 0, 1 of list q
    union {
        struct {
            int start[8];
            float xmin[4], xmax[4];
            unsigned fl[(8 * YZ_MAXWIN + 31) / 32];  // windowed hits that are in a pair
            unsigned char widx[8 * YZ_MAXWIN];       // plane hit index of each windowed hit
        };                                           // while the windows are built
        YzPhase2 d;                                  // while survivors are evaluated
    } w;
    int np[4], nw[8], woff[8];
    float x0, tx, ex0, etx;
    int nhx;
    float xdd[4], xres[4], xp1x[4], xp1y[4], xp1z[4], xdpx[4], xdpy[4], xdpz[4];
    short xhs[4];
    // survivors this warp evaluated (work counter)
    unsigned long long nsurv;
    YzBest b;
};

// The event's plane views for a tracklet of station half st3, one plane per
// lane (every lane calls): u2 u2' v2 v2' u3 u3' v3 v3' (K:910-984), the
// prop-tube y planes and the x hodoscopes of stations 2-4.
// chambers: only the u and v planes.
__device__ __forceinline__ void yz_event_planes(YzEvent &E, const or_hits_view_t &hv, long e, int st3,
                                                bool chambers = false) {
    const int lane = lane_id();
    int det = 0;
    HitPlane *dst = nullptr;
    if (lane < 8) {
        const int u3 = det_u3(st3), v3 = det_v3(st3);
        det = lane == 0 ? DET_U2 : lane == 1 ? DET_UP2 : lane == 2 ? DET_V2 : lane == 3 ? DET_VP2
            : lane == 4 ? u3 : lane == 5 ? u3 - 1 : lane == 6 ? v3 : v3 - 1;
        E.dl[lane] = (short)det;
        dst = &E.hc[lane];
    } else if (chambers) {
    } else if (lane < 12) {
        det = lane == 8 ? DET_P1Y1 : lane == 9 ? DET_P1Y2 : lane == 10 ? DET_P2Y1 : DET_P2Y2;
        dst = lane == 8 ? &E.p1y1 : lane == 9 ? &E.p1y2 : lane == 10 ? &E.p2y1 : &E.p2y2;
    } else if (lane < 18) {
        const int q = (lane - 12) >> 1, c = (lane - 12) & 1;
        det = c_hodoplanesx[q + 1][c];
        dst = &E.hod[q][c];
    }
    if (dst) *dst = hits_of(hv, e, det);
}

// Build the tracklet's windows (make_hitpairs_in_station, H:464-549) with the
// per-hit y of this tracklet (calculate_y_uvhit, H:75-100).  Returns false
// when a window or a pair list exceeds the reference's 100-entry arrays.
//
// The hits of the eight planes are one index space in list order, and so are
// the hits in the windows, the candidate pairs of the four projections and
// the hits left unpaired: 32 entries of each at a time, whatever plane they
// belong to.  A plane holds some ten hits and a window some five, so plane
// by plane most lanes were idle and the loops' instructions were fetched
// eight times over (planning pass of 100,000 uneven events, with the changes
// to the unit states below: 12.1 -> 5.2 ms).
__device__ bool yz_build(YzWarp &S, const YzEvent &E, const float *T, const or_plane_t &P, int st3,
                         const YzHit *&base, YzHit *garena) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const float x0 = T[OR_TRK_X0], tx = T[OR_TRK_TX], ex0 = T[OR_TRK_ERR_X0], etx = T[OR_TRK_ERR_TX];
    // hits of the planes before plane `lane`, and the window of each projection
    int start, total;
    {
        const int n = lane < 8 ? E.hc[lane].n : 0;
        start = n;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, start, o);
            if (lane >= o) start += v;
        }
        total = __shfl_sync(0xffffffffu, start, 7);
        start -= n;
        if (lane < 8) S.w.start[lane] = start;
        if (lane < 4) {
            const float za = P.z[E.dl[2 * lane]], zb = P.z[E.dl[2 * lane + 1]];
            const float sp = P.spacing[E.dl[2 * lane]];
            S.w.xmin[lane] = fminf((tx - etx) * za, (tx - etx) * zb) + x0 - ex0 - sp;
            S.w.xmax[lane] = fmaxf((tx + etx) * za, (tx + etx) * zb) + x0 + ex0 + sp;
            S.np[lane] = 0;
        }
    }
    __syncwarp();
    // list of entry i of an index space whose lists start at s[0..7]
    auto list_of = [](const int *s, int i) {
        int l = 0;
#pragma unroll
        for (int k = 1; k < 8; ++k) l += i >= s[k];
        return l;
    };
    // windowed hits, in list order (H:480-511)
    int nwin = 0, wo = -1;
#pragma unroll 1
    for (int b0 = 0; b0 < total; b0 += 32) {
        const int f = b0 + lane;
        bool in = false;
        int i = 0;
        if (f < total) {
            const int l = list_of(S.w.start, f);
            i = f - S.w.start[l];
            in = wp_in_window(E.dl[l], E.hc[l].chan(i), S.w.xmin[l >> 1], S.w.xmax[l >> 1], P);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        const int k = nwin + __popc(m & lt);
        if (in && k < 8 * YZ_MAXWIN) S.w.widx[k] = (unsigned char)i;
        if (lane < 8 && start >= b0 && start < b0 + 32) wo = nwin + __popc(m & ((1u << (start - b0)) - 1u));
        nwin += __popc(m);
    }
    if (wo < 0) wo = nwin;
    const int next = __shfl_down_sync(0xffffffffu, wo, 1);
    const int nw = (lane == 7 ? nwin : next) - wo;
    if (__any_sync(0xffffffffu, lane < 8 && nw > YZ_MAXWIN)) return false;
    if (lane < 8) {
        S.nw[lane] = nw;
        S.woff[lane] = wo;
    }
    if (lane < (8 * YZ_MAXWIN + 31) / 32) S.w.fl[lane] = 0u;
    __syncwarp();
    // windowed hit records (K:1326-1355 computes these per combination)
    YzHit *dst = (nwin <= YZ_ARENA_HITS) ? S.arena : garena;
#pragma unroll 1
    for (int k = lane; k < nwin; k += 32) {
        const int l = list_of(S.woff, k);
        const HitPlane &h = E.hc[l];
        const int det = E.dl[l];
        const int hi = S.w.widx[k];
        YzHit r;
        r.det = (short)det;
        r.el = (short)h.chan(hi);
        r.tdc = h.tdc(hi);
        r.drift = h.drift(hi);
        r.pos = h.pos(hi);
        float yy = 0.f, ey = 0.f;
        r.acc = calculate_y_uvhit(det, r.el, r.drift, 0, x0, tx, P, yy, ey) ? 1 : 0;
        r.Y = yy;
        r.eY = ey;
        r.z = P.z[det];
        dst[k] = r;
    }
    __syncwarp();
    // append to projection q's pair list, in lane order
    auto append = [&](bool take, int q, short2 v) {
        const unsigned peers = __match_any_sync(0xffffffffu, take ? q : 4 + lane);
        int at = 0;
        if (take) {
            at = S.np[q];
            const int k = at + __popc(peers & lt);
            if (k < YZ_MAXPAIR) S.pair[q][k] = v;
        }
        __syncwarp();
        if (take && (peers & lt) == 0u) S.np[q] = at + __popc(peers);
        __syncwarp();
    };
    // pairs over each projection's two windowed lists (H:513-546)
    {
        const int n2 = __shfl_down_sync(0xffffffffu, nw, 1);
        const int c12 = lane < 8 && (lane & 1) == 0 ? nw * n2 : 0;  // lane 2q: projection q
        int incl = c12;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const int npair = __shfl_sync(0xffffffffu, incl, 7);
        if (lane < 8 && (lane & 1) == 0) S.w.start[lane >> 1] = incl - c12;
        __syncwarp();
#pragma unroll 1
        for (int b0 = 0; b0 < npair; b0 += 32) {
            const int f = b0 + lane;
            bool take = false;
            int q = 0;
            short2 v = make_short2(0, 0);
            if (f < npair) {
                q = (f >= S.w.start[1]) + (f >= S.w.start[2]) + (f >= S.w.start[3]);
                const int n2 = S.nw[2 * q + 1], c = f - S.w.start[q];
                const int ia = c / n2, ib = c - ia * n2;
                const float spacing = c_spacingplane[c_detsuperid[q < 2 ? 2 : st3][1 + (q & 1)]];
                const int oa = S.woff[2 * q] + ia, ob = S.woff[2 * q + 1] + ib;
                if (!(fabsf(dst[oa].pos - dst[ob].pos) > spacing)) {
                    take = true;
                    v = make_short2((short)ia, (short)ib);
                    atomicOr(&S.w.fl[oa >> 5], 1u << (oa & 31));
                    atomicOr(&S.w.fl[ob >> 5], 1u << (ob & 31));
                }
            }
            append(take, q, v);
        }
    }
    // then the hits without a partner, first plane's before second plane's
#pragma unroll 1
    for (int b0 = 0; b0 < nwin; b0 += 32) {
        const int k = b0 + lane;
        const bool take = k < nwin && !((S.w.fl[b0 >> 5] >> lane) & 1u);
        const int l = take ? list_of(S.woff, k) : 0;
        const short i = (short)(k - S.woff[l]);
        append(take, l >> 1, (l & 1) ? make_short2(-1, i) : make_short2(i, -1));
    }
    const bool ok = !__any_sync(0xffffffffu, lane < 4 && S.np[lane & 3] > YZ_MAXPAIR);
    base = dst;
    if (lane == 0) {
        S.x0 = x0;
        S.tx = tx;
        S.ex0 = ex0;
        S.etx = etx;
    }
    __syncwarp();
    return ok;
}

// A queued tracklet's windows as yz_build left them: the planning pass
// stores this image once, and the first-cut and survivor kernels load it
// for each of the tracklet's units instead of windowing the event's hits
// again.  Layout in 16-byte words: the head (7 words), the arena (2 words a
// hit), then the four pair lists back to back (4 pairs a word).
struct __align__(16) YzImgHead {
    int np[4];
    int nw[8], woff[8];
    float x0, tx, ex0, etx;
    int total, npair, pad[2];
};
static_assert(sizeof(YzImgHead) == 112, "YzImgHead is seven 16-byte words");
constexpr int YZ_IMG_HEAD_WORDS = sizeof(YzImgHead) / 16;

// Store the windows just built (base: their arena); returns the image's
// word offset, or -1 when the pool is full.
__device__ int yz_store_image(const YzWarp &S, const YzHit *base, const YzScratch &sc) {
    const int lane = lane_id();
    const int total = S.woff[7] + S.nw[7];
    const int npair = S.np[0] + S.np[1] + S.np[2] + S.np[3];
    const long long words = YZ_IMG_HEAD_WORDS + 2LL * total + (npair + 3) / 4;
    unsigned long long o = 0ull;
    if (lane == 0) o = atomicAdd(reinterpret_cast<unsigned long long *>(sc.counters + 10), (unsigned long long)words);
    o = __shfl_sync(0xffffffffu, o, 0);
    if ((long long)o + words > sc.img_cap) return -1;
    uint4 *dst = sc.img + o;
    if (lane == 0) {
        YzImgHead h;
#pragma unroll
        for (int q = 0; q < 4; ++q) h.np[q] = S.np[q];
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            h.nw[l] = S.nw[l];
            h.woff[l] = S.woff[l];
        }
        h.x0 = S.x0;
        h.tx = S.tx;
        h.ex0 = S.ex0;
        h.etx = S.etx;
        h.total = total;
        h.npair = npair;
        h.pad[0] = h.pad[1] = 0;
        *reinterpret_cast<YzImgHead *>(dst) = h;
    }
    const uint4 *src = reinterpret_cast<const uint4 *>(base);
    uint4 *da = dst + YZ_IMG_HEAD_WORDS;
#pragma unroll 1
    for (int i = lane; i < 2 * total; i += 32) da[i] = src[i];
    short2 *dp = reinterpret_cast<short2 *>(da + 2 * total);
    int off = 0;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
#pragma unroll 1
        for (int i = lane; i < S.np[q]; i += 32) dp[off + i] = S.pair[q][i];
        off += S.np[q];
    }
    return (int)o;
}

// Load a tracklet's windows from its image into the warp's state; returns
// the arena (in shared memory when it fits there, else the image itself).
__device__ const YzHit *yz_load_image(YzWarp &S, const uint4 *__restrict__ img) {
    const int lane = lane_id();
    const YzImgHead &h = *reinterpret_cast<const YzImgHead *>(img);
    const int total = h.total;
    if (lane < 4) S.np[lane] = h.np[lane];
    if (lane < 8) {
        S.nw[lane] = h.nw[lane];
        S.woff[lane] = h.woff[lane];
    }
    if (lane == 0) {
        S.x0 = h.x0;
        S.tx = h.tx;
        S.ex0 = h.ex0;
        S.etx = h.etx;
    }
    const uint4 *ia = img + YZ_IMG_HEAD_WORDS;
    const YzHit *base = reinterpret_cast<const YzHit *>(ia);
    if (total <= YZ_ARENA_HITS) {
        uint4 *da = reinterpret_cast<uint4 *>(S.arena);
#pragma unroll 1
        for (int i = lane; i < 2 * total; i += 32) da[i] = ia[i];
        base = S.arena;
    }
    const short2 *ip = reinterpret_cast<const short2 *>(ia + 2 * total);
    int off = 0;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const int n = h.np[q];
#pragma unroll 1
        for (int i = lane; i < n; i += 32) S.pair[q][i] = ip[off + i];
        off += n;
    }
    __syncwarp();
    return base;
}

// x hits of the tracklet (K:1300-1316)
__device__ __forceinline__ void yz_xhits(YzWarp &S, const float *T, const or_plane_t &P) {
    const int lane = lane_id();
    const int nhx = min((int)T[OR_TRK_NHITS], 4);  // XZ tracklets carry 2-4 hits
    if (lane < nhx) {
        const short d = (short)T[OR_TRK_HIT_DETID + lane];
        const short ch = (short)T[OR_TRK_HIT_CHAN + lane];
        S.xdd[lane] = T[OR_TRK_HIT_DRIFT + lane];
        S.xhs[lane] = (short)T[OR_TRK_HIT_SIGN + lane];
        S.xres[lane] = P.resolution[d];
        S.xp1x[lane] = x_bep(d, ch, P);
        S.xp1y[lane] = y_bep(d, ch, P);
        S.xp1z[lane] = z_bep(d, ch, P);
        S.xdpx[lane] = P.deltapx[d];
        S.xdpy[lane] = P.deltapy[d];
        S.xdpz[lane] = P.deltapz[d];
    }
    if (lane == 0) S.nhx = nhx;
    __syncwarp();
}

// A survivor's accepted u/v hits in the reference order (K:1326-1597), kept
// in registers: arena offsets, 16 bits each (hits 0-3 in lo, 4-7 in hi), and
// the left/right signs, 2 bits each in two's complement (0, 1 or -1).  The
// hits' fields are read from the arena where they are needed.
struct UvSet {
    unsigned long long lo, hi;
    unsigned sign;
};

__device__ __forceinline__ int uv_off(const UvSet &U, int k) {
    return (int)(((k < 4 ? U.lo : U.hi) >> (16 * (k & 3))) & 0xFFFFull);
}
__device__ __forceinline__ short uv_sign(const UvSet &U, int k) {
    return (short)((int)(U.sign << (30 - 2 * k)) >> 30);
}
__device__ __forceinline__ void uv_set_sign(UvSet &U, int k, int s) {
    U.sign = (U.sign & ~(3u << (2 * k))) | (((unsigned)s & 3u) << (2 * k));
}

// The pairs resolve_leftright_newhits walks over (H:714-780): hits i and i + 1
// (or the scratch entry past the end, plane `dst`) of neighbouring planes, not
// both with a sign; bit i set.  They depend on the planes and the starting
// signs alone, and no hit is in two of them.
__device__ __forceinline__ unsigned yz_walk_pairs(int n, const UvSet &U, const YzHit *base, short dst) {
    unsigned pm = 0u;
    if (n == 0) return pm;
    short di = base[uv_off(U, 0)].det;
    bool paired = false;  // hit i was the second of a pair
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const short dj = i + 1 < n ? base[uv_off(U, i + 1)].det : dst;
        if (!paired && abs(di - dj) == 1) {
            if (!uv_sign(U, i) || i + 1 >= n || !uv_sign(U, i + 1)) pm |= 1u << i;
            paired = true;
        } else {
            paired = false;
        }
        di = dj;
    }
    return pm;
}

__device__ __forceinline__ const YzHit *yz_list(const YzWarp &S, const YzHit *base, int l) { return base + S.woff[l]; }

// accepted station-3 hits of the outer iteration (iu3, iv3)
__device__ __forceinline__ int s3_count(const YzWarp &S, const YzHit *base, int iu3, int iv3, bool &valid) {
    const short2 pu = S.pair[2][iu3], pv = S.pair[3][iv3];
    int nu = 0, nv = 0;
    if (pu.x >= 0) nu += yz_list(S, base, 4)[pu.x].acc;
    if (pu.y >= 0) nu += yz_list(S, base, 5)[pu.y].acc;
    if (nu > 0) {
        if (pv.x >= 0) nv += yz_list(S, base, 6)[pv.x].acc;
        if (pv.y >= 0) nv += yz_list(S, base, 7)[pv.y].acc;
    }
    valid = nu > 0 && nv > 0;
    return nu + nv;
}

// Walk the outer iterations of the current tracklet in order and track the
// scratch entries 4..7 from the load pattern alone (no fits): entry k is set
// by the last inner combination writing offset k-4+... of the last valid
// outer iteration that reaches it.  When `units` is given, the state at the
// start of every unit (each `gper` outer iterations) is stored there.  `st`
// goes in as the state before the tracklet and comes out as the state after.
// live outer iterations (both pairs alive) before outer index g, g <= G:
// the scorer-row rank of g when g is live
__device__ __forceinline__ int live_before(const unsigned mu[4], const unsigned mv[4], int nu3, int g) {
    const int iu = g % nu3, iv = g / nu3;
    int below_v = 0, below_u = 0, au = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        au += __popc(mu[w]);
        if (w < (iv >> 5)) below_v += __popc(mv[w]);
        else if (w == (iv >> 5)) below_v += __popc(mv[w] & ((1u << (iv & 31)) - 1u));
        if (w < (iu >> 5)) below_u += __popc(mu[w]);
        else if (w == (iu >> 5)) below_u += __popc(mu[w] & ((1u << (iu & 31)) - 1u));
    }
    const bool v_live = iv < 128 && ((mv[iv >> 5] >> (iv & 31)) & 1u);
    return below_v * au + (v_live ? below_u : 0);
}

static_assert(8 * YZ_MAXWIN <= 1024, "arena offsets fit 10 bits");

// The station-2 record of the inner pair (iu2, iv2): its load attempts in
// the reference order (K:1467-1597) reduced to what the first cut needs, the
// same in every outer iteration.  16-bit field e (0..3) holds in bits 0-9 the
// arena offset of the last hit attempted when e of the pair's hits had been
// accepted -- for e below the accepted count, accepted hit e, in order -- so
// that after n3 station-3 hits the attempts write scratch entries e + n3 - 4;
// bits 10-13 which fields were written, bits 26-28 the accepted count, bits
// 42-45 the planes of the accepted hits (u2 u2' v2 v2'), bit 58 whether both
// the u2 and the v2 group gave a hit (the first fit is reached).
__device__ __forceinline__ unsigned long long yz_s2_record(const YzWarp &S, const YzHit *base, int iu2, int iv2) {
    const short2 pu = S.pair[0][iu2], pv = S.pair[1][iv2];
    const int offs[4] = {pu.x >= 0 ? S.woff[0] + pu.x : -1, pu.y >= 0 ? S.woff[1] + pu.y : -1,
                         pv.x >= 0 ? S.woff[2] + pv.x : -1, pv.y >= 0 ? S.woff[3] + pv.y : -1};
    unsigned long long rec = 0ull;
    unsigned pm = 0u, g2 = 0u;
    int nacc = 0, nu = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (a == 2) {
            nu = nacc;
            if (nu == 0) break;  // no u2 hit: v2 is not loaded
        }
        const int off = offs[a];
        if (off < 0) continue;
        const int sh = 16 * nacc;
        rec = (rec & ~(0x3FFull << sh)) | ((unsigned long long)off << sh);
        pm |= 1u << nacc;
        if (base[off].acc) {
            g2 |= 1u << a;
            ++nacc;
        }
    }
    const unsigned fit = (nu > 0 && nacc > nu) ? 1u : 0u;
    return rec | ((unsigned long long)pm << 10) | ((unsigned long long)nacc << 26) | ((unsigned long long)g2 << 42) |
           ((unsigned long long)fit << 58);
}

// The station-2 load attempts of an outer iteration do not depend on the
// iteration (only on the inner pair, K:1467-1597): the last inner combination
// writing scratch offset m (past the station-3 hit count) is the same in
// every live outer iteration.  Returns those hits as arena offsets, 16 bits
// per offset m = 0..3, 0xFFFF where no combination writes m.
__device__ unsigned long long yz_last_writes(const YzWarp &S, const YzHit *base) {
    const int nu2 = S.np[0];
    const int C2 = S.np[0] * S.np[1];
    unsigned long long lasto = ~0ull;
#pragma unroll 1
    for (int b0 = 0; b0 < C2; b0 += 32) {
        const int c = b0 + lane_id();
        const unsigned long long rec = c < C2 ? yz_s2_record(S, base, c % nu2, c / nu2) : 0ull;
        const unsigned pm = (unsigned)(rec >> 10) & 0xFu;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int l = last_lane(__ballot_sync(0xffffffffu, (pm >> m) & 1u));
            if (l >= 0) {
                const unsigned long long o =
                    (unsigned)__shfl_sync(0xffffffffu, (unsigned)((rec >> (16 * m)) & 0x3FFull), l);
                lasto = (lasto & ~(0xFFFFull << (16 * m))) | (o << (16 * m));
            }
        }
    }
    return lasto;
}

__device__ void yz_unit_states(const YzWarp &S, const YzHit *base, int G, int gper, Stale st[4], YzUnit *units,
                               int heavy, const unsigned *alive_u = nullptr, const unsigned *alive_v = nullptr) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const int nu3 = S.np[2];
    // the last inner combination's write of each offset m, as arena offsets
    const unsigned long long lasto = yz_last_writes(S, base);
    const Stale st_in[4] = {st[0], st[1], st[2], st[3]};
    // per entry k the arena offset of its last write so far (0xFFFF: st_in[k])
    unsigned long long carry = ~0ull;
    auto resolve = [&](int k, unsigned o) -> Stale {
        if (o == 0xFFFFu) return st_in[k];
        const YzHit &r = base[o];
        return Stale{r.det, r.pos, r.drift};
    };
#pragma unroll 1
    for (int b0 = 0; b0 < G; b0 += 32) {
        const int g = b0 + lane;
        unsigned long long mk = ~0ull;  // this outer iteration's writes of entries 4..7
        if (g < G) {
            bool valid;
            const int n3 = s3_count(S, base, g % nu3, g / nu3, valid);
            if (valid) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int mm = k + 4 - n3;
                    if (mm >= 0 && mm < 4)
                        mk = (mk & ~(0xFFFFull << (16 * k))) | (((lasto >> (16 * mm)) & 0xFFFFull) << (16 * k));
                }
            }
        }
        unsigned long long ent = 0ull;  // the entries as this outer iteration finds them
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned wk = (unsigned)((mk >> (16 * k)) & 0xFFFFull);
            const unsigned wm = __ballot_sync(0xffffffffu, wk != 0xFFFFu);
            const int src = last_lane(wm & lt);
            const unsigned v = __shfl_sync(0xffffffffu, wk, src < 0 ? 0 : src);
            const unsigned e = src >= 0 ? v : (unsigned)((carry >> (16 * k)) & 0xFFFFull);
            ent |= (unsigned long long)e << (16 * k);
            const int l = last_lane(wm);
            if (l >= 0) {
                const unsigned long long c = __shfl_sync(0xffffffffu, wk, l);
                carry = (carry & ~(0xFFFFull << (16 * k))) | (c << (16 * k));
            }
        }
        if (units && g < G && (g % gper) == 0) {
            YzUnit &u = units[g / gper];
            u.heavy = heavy;
            u.g0 = g;
            u.g1 = min(G, g + gper);
            u.pad = 0;
            u.r0 = alive_u ? live_before(alive_u, alive_v, nu3, u.g0) : 0;
            u.r1 = alive_u ? live_before(alive_u, alive_v, nu3, u.g1) : 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) u.entry[k] = resolve(k, (unsigned)((ent >> (16 * k)) & 0xFFFFull));
        }
    }
    __syncwarp();  // every lane has read the entry states
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const Stale v = resolve(k, (unsigned)((carry >> (16 * k)) & 0xFFFFull));
        if (lane == 0) st[k] = v;
    }
    __syncwarp();
}

// Accepted hits of a pair of projection q (bit 0: first plane, bit 1: second).
__device__ __forceinline__ int yz_pair_group(const YzWarp &S, const YzHit *base, int q, int i) {
    const short2 p = S.pair[q][i];
    return (p.x >= 0 && base[S.woff[2 * q] + p.x].acc ? 1 : 0) | (p.y >= 0 && base[S.woff[2 * q + 1] + p.y].acc ? 2 : 0);
}

// Which pairs of a projection come last, by their accepted hits.
struct YzLast {
    int one, two, r1;  // one hit; two hits; a second attempt after an accepted first one; -1: no such pair
};
__device__ __forceinline__ YzLast yz_last_pairs(const YzWarp &S, const YzHit *base, int q) {
    YzLast o{-1, -1, -1};
#pragma unroll 1
    for (int b0 = 0; b0 < S.np[q]; b0 += 32) {
        const int i = b0 + lane_id();
        int g = 0;
        bool r1 = false;
        if (i < S.np[q]) {
            g = yz_pair_group(S, base, q, i);
            r1 = (g & 1) && S.pair[q][i].y >= 0;
        }
        const unsigned m1 = __ballot_sync(0xffffffffu, g == 1 || g == 2);
        const unsigned m2 = __ballot_sync(0xffffffffu, g == 3);
        const unsigned mr = __ballot_sync(0xffffffffu, r1);
        if (m1) o.one = b0 + last_lane(m1);
        if (m2) o.two = b0 + last_lane(m2);
        if (mr) o.r1 = b0 + last_lane(mr);
    }
    return o;
}

// The last write of offset m = 0..3 past the station-3 hits over the inner
// pairs of an outer iteration (what yz_last_writes finds by walking them),
// from which u2 and v2 pairs come last: a combination tries its u2 pair, and
// after an accepted u2 hit its v2 pair, each hit at the count so far.  `first`
// / `second` give a pair's hits as arena offsets (-1: none) and the offset its
// first attempt's place ends with.
template <class First, class Rel0>
__device__ __forceinline__ unsigned long long yz_lasto(int nu2, int nv2, const YzLast &u, const YzLast &v, First second,
                                                       Rel0 rel0) {
    unsigned o1 = 0xFFFFu, o2 = 0xFFFFu, o3 = 0xFFFFu;
    const unsigned o0 = rel0(0, nu2 - 1);
    if (u.one > u.two) o1 = rel0(1, nv2 - 1);
    else if (u.two >= 0) o1 = second(0, u.two);
    if (u.two >= 0) o2 = u.one > u.two && v.r1 == nv2 - 1 ? second(1, v.r1) : rel0(1, nv2 - 1);
    else if (u.one >= 0 && v.r1 >= 0) o2 = second(1, v.r1);
    if (u.two >= 0 && v.r1 >= 0) o3 = second(1, v.r1);
    return (unsigned long long)o0 | ((unsigned long long)o1 << 16) | ((unsigned long long)o2 << 32) |
           ((unsigned long long)o3 << 48);
}

// The scratch entries 4..7 after a whole tracklet: for each entry, the last
// live outer iteration whose station-3 hit count puts one of the inner pairs'
// writes there.  The last iteration of n3 hits is the last v3 pair of one
// kind with the last u3 pair of another.
__device__ void yz_final_state(const YzWarp &S, const YzHit *base, Stale st[4]) {
    const YzLast u2 = yz_last_pairs(S, base, 0), v2 = yz_last_pairs(S, base, 1);
    const YzLast u3 = yz_last_pairs(S, base, 2), v3 = yz_last_pairs(S, base, 3);
    auto second = [&](int q, int i) { return (unsigned)(S.woff[2 * q + 1] + S.pair[q][i].y); };
    auto rel0 = [&](int q, int i) {
        const short2 p = S.pair[q][i];
        const bool sec = p.x < 0 || (!base[S.woff[2 * q] + p.x].acc && p.y >= 0);
        return (unsigned)(sec ? S.woff[2 * q + 1] + p.y : S.woff[2 * q] + p.x);
    };
    const unsigned long long lasto = yz_lasto(S.np[0], S.np[1], u2, v2, second, rel0);
    const int nu3 = S.np[2];
    auto g_of = [&](int iu, int iv) { return iu >= 0 && iv >= 0 ? iv * nu3 + iu : -1; };
    const int lastg[3] = {g_of(u3.one, v3.one), max(g_of(u3.one, v3.two), g_of(u3.two, v3.one)), g_of(u3.two, v3.two)};
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int best = -1;
        unsigned off = 0xFFFFu;
#pragma unroll
        for (int n3 = 2; n3 <= 4; ++n3) {
            const int mm = k + 4 - n3;
            if (mm > 3) continue;
            const unsigned o = (unsigned)(lasto >> (16 * mm)) & 0xFFFFu;
            if (o != 0xFFFFu && lastg[n3 - 2] > best) {
                best = lastg[n3 - 2];
                off = o;
            }
        }
        if (off != 0xFFFFu && lane_id() == 0) {
            const YzHit &r = base[off];
            st[k] = Stale{r.det, r.pos, r.drift};
        }
    }
    __syncwarp();
}

// A combination that passed the first y cut, queued for the full evaluation:
// index inside the tracklet, first fit, scratch entry past its hit count.
using PassEntry = PassEntryStore;

// Gather the accepted hits of combination c in the reference order
// (K:1326-1597), station 3 first; returns nuv, sets n3.
__device__ __forceinline__ int yz_gather(const YzWarp &S, const YzHit *base, int c, int C2, UvSet &U, int &n3) {
    const int iuv3 = c / C2, iuv2 = c - iuv3 * C2;
    const int nu2 = S.np[0], nu3 = S.np[2];
    const short2 p3u = S.pair[2][iuv3 % nu3], p3v = S.pair[3][iuv3 / nu3];
    const short2 p2u = S.pair[0][iuv2 % nu2], p2v = S.pair[1][iuv2 / nu2];
    U.lo = U.hi = 0ull;
    U.sign = 0u;
    int nuv = 0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        if (a == 4) n3 = nuv;
        const short2 p = a < 2 ? p3u : a < 4 ? p3v : a < 6 ? p2u : p2v;
        const int wi = (a & 1) ? p.y : p.x;
        if (wi < 0) continue;
        const int l = (a + 4) & 7;  // lists u3 u3' v3 v3' u2 u2' v2 v2'
        const int off = S.woff[l] + wi;
        if (!base[off].acc) continue;
        const unsigned long long f = (unsigned long long)off << (16 * (nuv & 3));
        if (nuv < 4) U.lo |= f;
        else U.hi |= f;
        ++nuv;
    }
    return nuv;
}

// The same from the pairs and the planes that give a hit (bits u3 u3' v3 v3'
// u2 u2' v2 v2').
__device__ __forceinline__ int yz_gather_planes(const YzWarp &S, int iu3, int iv3, int iu2, int iv2, unsigned planes,
                                                UvSet &U, int &n3) {
    const short2 p3u = S.pair[2][iu3], p3v = S.pair[3][iv3], p2u = S.pair[0][iu2], p2v = S.pair[1][iv2];
    int nuv = 0;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        if (a == 4) n3 = nuv;
        if (!((planes >> a) & 1u)) continue;
        const short2 p = a < 2 ? p3u : a < 4 ? p3v : a < 6 ? p2u : p2v;
        const unsigned long long f = (unsigned long long)(S.woff[(a + 4) & 7] + ((a & 1) ? p.y : p.x))
                                     << (16 * (nuv & 3));
        if (nuv < 4) U.lo |= f;
        else U.hi |= f;
        ++nuv;
    }
    return nuv;
}

// gates of a candidate after the refit: the hard cut (K:1638), the prop-tube
// y segments (K:1640-1702) and the hodoscopes with y (H:1002-1087)
__device__ __noinline__ bool yz_gates(const YzEvent &E, const or_plane_t &P, float x0, float y0, float tx, float ty,
                                      float ex0, float ey0, float etx, float ety) {
    if (fabsf(y0) > Y0_MAX || fabsf(ty) > TY_MAX) return false;
    const int nprop = prop_hits(E.p1y1, P.z[DET_P1Y1], E.p1y2, P.z[DET_P1Y2], 5.08f, y0, ty) +
                      prop_hits(E.p2y1, P.z[DET_P2Y1], E.p2y2, P.z[DET_P2Y2], 10.16f, y0, ty);
    if (nprop < NPROP_MIN) return false;
#pragma unroll 1
    for (int qq = 0; qq < 3; ++qq) {
        bool ok = false;
#pragma unroll 1
        for (int c = 0; c < 2 && !ok; ++c)
            ok = match_tracklet_to_hodo(qq + 1, c_hodoplanesx[qq + 1][c], E.hod[qq][c], x0, y0, tx, ty, ex0, ey0, etx,
                                        ety, P);
        if (!ok) return false;
    }
    return true;
}

// One residual of chi2_track (H:1149-1165): x hit m < nhx, else u/v hit
// m - nhx of U.
__device__ __forceinline__ float yz_residual(const YzWarp &S, const UvSet &U, const YzHit *base, int m, int nhx,
                                             const or_plane_t &P, float x0, float y0, float tx, float ty, float &res) {
    if (m < nhx) {
        res = S.xres[m];
        return residual_line(S.xp1x[m], S.xp1y[m], S.xp1z[m], S.xdpx[m], S.xdpy[m], S.xdpz[m], S.xdd[m], S.xhs[m], x0,
                             y0, tx, ty);
    }
    const int k = m - nhx;
    const YzHit &h = base[uv_off(U, k)];
    const short d = h.det;
    res = P.resolution[d];
    return residual_line(x_bep(d, h.el, P), y_bep(d, h.el, P), z_bep(d, h.el, P), P.deltapx[d], P.deltapy[d],
                         P.deltapz[d], h.drift, uv_sign(U, k), x0, y0, tx, ty);
}

// Sign state carried from one survivor chunk to the next (the first
// combination of an outer iteration fixes the station-3 signs), and the best
// key so far.
struct Phase2Carry {
    int g = -1;
    bool hasf = false, hascross = false;
    short sig[4] = {0, 0, 0, 0};
    short cross = 0;
    unsigned long long best = ~0ull;
};

// The full evaluation of n (<= 32) queued survivors Qc[0..n), in order: sign
// state, left/right walk, prop and hodoscope gates, chi2, best key
// (K:1613-1799).  The pairs to resolve, the single hits and the chi2 terms of
// all survivors are dealt to the lanes one by one: a chunk holds 8 (dimuon
// events) or 20 (uneven ones) survivors on average, and a lane per survivor
// left the others idle and the walks diverging (survivor kernel, 10,000
// dimuon events 317 -> 214 us, 100,000 uneven 8.2 -> 6.2 ms).  Out of line: it
// runs once per 32 survivors, and inlined it would sit in the middle of the
// first-cut loop's instructions.  GATED: the
// survivors come from the first-cut kernel (YzSurv), which has evaluated the
// gates; `tab` is the station half's table, S.st the unit's starting entries.
template <bool GATED>
__device__ __noinline__ void yz_phase2(YzWarp &S, const YzEvent &E, const YzHit *base, int C2, const or_plane_t &P,
                                       const std::conditional_t<GATED, YzSurv, PassEntryStore> *Qc, int n,
                                       const YzTab *__restrict__ tab, Phase2Carry &cs) {
    const int lane = lane_id();
    const float x0 = S.x0, tx = S.tx, ex0 = S.ex0, etx = S.etx;
    const int nhx = S.nhx;
    if (!GATED && lane == 0) S.nsurv += (unsigned long long)n;
    // --- one chunk of survivors ------------------------------------------
    const bool valid = lane < n;
    PassEntry q;
    bool gated = false;
    UvSet U{0ull, 0ull, 0u};
    int n3 = 0, nuv = 0, g = -1 - lane;
    if constexpr (GATED) {
        if (valid) {
            const uint4 v = *reinterpret_cast<const uint4 *>(Qc + lane);
            const int iu3 = (int)(v.x & 127u), iv3 = (int)(v.x >> 7) & 127;
            const int iu2 = (int)(v.x >> 14) & 127, iv2 = (int)(v.x >> 21) & 127;
            g = iu3 + iv3 * S.np[2];
            q.c = g * C2 + iu2 + iv2 * S.np[0];
            nuv = yz_gather_planes(S, iu3, iv3, iu2, iv2, v.w >> 22, U, n3);
            q.y0 = __uint_as_float(v.y);
            q.ty = __uint_as_float(v.z);
            gated = (v.w >> 31) != 0u;
            const float2 er = __ldg(reinterpret_cast<const float2 *>(&tab[(v.w >> 14) & 0x7Fu].ey0));
            q.ey0 = er.x;
            q.ety = er.y;
            const unsigned src = (v.w >> 10) & 3u;
            Stale e3{DET_SENTINEL, 0.f, 0.f};
            if (src == YZ_ENT_HIT) {
                const YzHit &r = base[v.w & 0x3FFu];
                e3 = Stale{r.det, r.pos, r.drift};
            } else if (src == YZ_ENT_UNIT) {
                e3 = S.st[(v.w >> 12) & 3u];
            }
            q.stdet = e3.det;
            q.stpos = e3.pos;
            q.stdrift = e3.drift;
        }
    } else if (valid) {
        q = Qc[lane];
    }
    const int c = valid ? q.c : 0;
    if constexpr (!GATED) g = valid ? c / C2 : -1 - lane;
    if constexpr (!GATED) {
        if (valid) nuv = yz_gather(S, base, c, C2, U, n3);
    }
    const Stale stj{(short)(valid ? q.stdet : DET_SENTINEL), valid ? q.stpos : 0.f, valid ? q.stdrift : 0.f};
    const float y0 = valid ? q.y0 : 0.f, ty = valid ? q.ty : 0.f;
    const float ey0 = valid ? q.ey0 : 0.f, ety = valid ? q.ety : 0.f;
    const unsigned seg = __match_any_sync(0xffffffffu, g);
    const unsigned vm = __ballot_sync(0xffffffffu, valid);
    const bool carried_f = (g == cs.g) && cs.hasf;
    const int fl = __ffs(vm & seg) - 1;
    const bool is_first = valid && !carried_f && fl == lane;
    // Every survivor walks at once.  A first survivor of its outer iteration
    // starts from unset signs; the others start with placeholder station-3
    // signs: the walk only asks whether a sign is set, so it passes over the
    // station-3 pairs and singles and resolves the station-2 hits and the
    // cross pair exactly as it does after their real signs, which are put in
    // below (the first survivor's, or the cross pair's where it resolved).
    // The pairs and then the single hits of all survivors are dealt to the
    // lanes (item: survivor << 3 | hit): a chunk holds a few survivors more
    // often than 32.
    YzPhase2 &D = S.w.d;
    auto deal = [&](unsigned m) {
        int tot = 0;
        for (unsigned b; (b = __ballot_sync(0xffffffffu, m != 0u)) != 0u;) {
            if (m) D.item[tot + __popc(b & lanemask_lt())] = (unsigned char)(lane << 3 | (__ffs(m) - 1));
            tot += __popc(b);
            m &= m - 1;
        }
        __syncwarp();
        return tot;
    };
    // survivor o's hits
    auto shfl_set = [&](int o) {
        const unsigned l0 = __shfl_sync(0xffffffffu, (unsigned)U.lo, o), l1 = __shfl_sync(0xffffffffu, (unsigned)(U.lo >> 32), o);
        const unsigned h0 = __shfl_sync(0xffffffffu, (unsigned)U.hi, o), h1 = __shfl_sync(0xffffffffu, (unsigned)(U.hi >> 32), o);
        UvSet V{(unsigned long long)l1 << 32 | l0, (unsigned long long)h1 << 32 | h0, 0u};
        return V;
    };
    unsigned pm = 0u;
    if (valid) {
        if (!is_first) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < n3) uv_set_sign(U, k, 1);
        }
        pm = yz_walk_pairs(nuv, U, base, stj.det);
    }
    {
        const int tot = deal(pm);
#pragma unroll 1
        for (int t0 = 0; t0 < tot; t0 += 32) {
            const bool in = t0 + lane < tot;
            const int it = in ? D.item[t0 + lane] : 0, o = it >> 3, i = it & 7;
            const UvSet V = shfl_set(o);
            const float oy = __shfl_sync(0xffffffffu, y0, o), ot = __shfl_sync(0xffffffffu, ty, o);
            const float oey = __shfl_sync(0xffffffffu, ey0, o), oet = __shfl_sync(0xffffffffu, ety, o);
            const int on = __shfl_sync(0xffffffffu, nuv, o);
            short dj = (short)__shfl_sync(0xffffffffu, (int)stj.det, o);
            float pj = __shfl_sync(0xffffffffu, stj.pos, o), drj = __shfl_sync(0xffffffffu, stj.drift, o);
            if (in) {
                const YzHit &hi = base[uv_off(V, i)];
                if (i + 1 < on) {
                    const YzHit &hj = base[uv_off(V, i + 1)];
                    dj = hj.det;
                    pj = hj.pos;
                    drj = hj.drift;
                }
                D.res[it] = (signed char)lr_pair_newhits(x0, tx, oy, ot, ex0, etx, oey, oet, hi.det, dj, hi.pos,
                                                         hi.drift, pj, drj, P, 150.f);
            }
        }
        __syncwarp();
    }
    bool xok = false;
    short xval = 0;
    for (unsigned m = pm; m; m &= m - 1) {
        const int i = __ffs(m) - 1, k = D.res[lane << 3 | i];
        if (k < 0) continue;
        uv_set_sign(U, i, c_lrpossibility[k][0]);
        if (i + 1 < nuv) uv_set_sign(U, i + 1, c_lrpossibility[k][1]);
        // the cross pair: the last station-3 hit with the first station-2 hit
        if (!is_first && i == n3 - 1 && i + 1 < nuv) {
            xok = true;
            xval = c_lrpossibility[k][0];
        }
    }
    {
        unsigned single = 0u;
        if (valid)
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < nuv && !uv_sign(U, k)) single |= 1u << k;
        __syncwarp();  // every lane has read its results
        const int tot = deal(single);
#pragma unroll 1
        for (int t0 = 0; t0 < tot; t0 += 32) {
            const bool in = t0 + lane < tot;
            const int it = in ? D.item[t0 + lane] : 0, o = it >> 3, i = it & 7;
            const UvSet V = shfl_set(o);
            const float oy = __shfl_sync(0xffffffffu, y0, o), ot = __shfl_sync(0xffffffffu, ty, o);
            if (in) {
                const YzHit &h = base[uv_off(V, i)];
                D.res[it] = (signed char)single_sign_newhits(x0, tx, oy, ot, h.det, h.pos, P);
            }
        }
        __syncwarp();
        for (; single; single &= single - 1) {
            const int k = __ffs(single) - 1;
            uv_set_sign(U, k, D.res[lane << 3 | k]);
        }
    }
    short sig[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const short mine = (k < n3) ? uv_sign(U, k) : (short)0;
        const short v = (short)__shfl_sync(0xffffffffu, (int)mine, fl < 0 ? 0 : fl);
        sig[k] = carried_f ? cs.sig[k] : v;
    }
    const unsigned xm = __ballot_sync(0xffffffffu, xok);
    const int xs = last_lane(xm & seg & lanemask_lt());
    const short xprev = (short)__shfl_sync(0xffffffffu, (int)xval, xs < 0 ? 0 : xs);
    bool pass = false;
    float chi2 = 0.f;
    if (valid && !is_first) {
        // the station-3 signs this survivor's walk would have started from:
        // the first survivor's, the last hit's re-set by an earlier survivor's
        // cross pair; its own cross pair, where resolved, already set the last
        // station-3 hit in the walk above
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < n3 && !(xok && k == n3 - 1)) uv_set_sign(U, k, sig[k]);
        if (n3 > 0 && !xok) {
            if (xs >= 0) uv_set_sign(U, n3 - 1, xprev);
            else if (g == cs.g && cs.hascross) uv_set_sign(U, n3 - 1, cs.cross);
        }
    }
    if (valid) {
        pass = GATED ? gated : yz_gates(E, P, x0, y0, tx, ty, ex0, ey0, etx, ety);
    }
    // chi2_track over the x hits and the uv hits (H:1182-1204): the terms of
    // the passing survivors dealt to the lanes, 16 survivors at a time; each
    // survivor adds its own in order
    {
        const unsigned passm = __ballot_sync(0xffffffffu, pass);
        const int rank = __popc(passm & lanemask_lt()), np = __popc(passm);
        if (pass) D.item[rank] = (unsigned char)lane;
        __syncwarp();
#pragma unroll 1
        for (int g0 = 0; g0 < np; g0 += 16) {
            const int tot = min(16, np - g0) * 12;
#pragma unroll 1
            for (int t0 = 0; t0 < tot; t0 += 32) {
                const int t = t0 + lane;
                const int o = t < tot ? D.item[g0 + t / 12] : 0, m = t % 12;
                UvSet V = shfl_set(o);
                V.sign = __shfl_sync(0xffffffffu, U.sign, o);
                const float oy = __shfl_sync(0xffffffffu, y0, o), ot = __shfl_sync(0xffffffffu, ty, o);
                const int on = __shfl_sync(0xffffffffu, nuv, o);
                if (t < tot && m < nhx + on) {
                    float res;
                    const float r = yz_residual(S, V, base, m, nhx, P, x0, oy, tx, ot, res);
                    D.term[t] = r * r / res / res;
                }
            }
            __syncwarp();
            if (pass && rank >= g0 && rank < g0 + 16)
#pragma unroll 1
                for (int m = 0; m < nhx + nuv; ++m) chi2 += D.term[(rank - g0) * 12 + m];
            __syncwarp();
        }
    }
    // carry of the sign state to the next survivor chunk
    {
        const int last = last_lane(vm);
        const int gl = __shfl_sync(0xffffffffu, g, last < 0 ? 0 : last);
        const unsigned segl = __ballot_sync(0xffffffffu, valid && g == gl);
        const int fnew = __ffs(__ballot_sync(0xffffffffu, is_first) & segl) - 1;
        short ns[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) ns[k] = (short)__shfl_sync(0xffffffffu, (int)sig[k], fnew < 0 ? 0 : fnew);
        const int xl = last_lane(xm & segl);
        const short nx = (short)__shfl_sync(0xffffffffu, (int)xval, xl < 0 ? 0 : xl);
        const bool cont = (gl == cs.g);
        if (fnew >= 0) {
            cs.hasf = true;
#pragma unroll 1
            for (int k = 0; k < 4; ++k) cs.sig[k] = ns[k];
        } else if (!cont) {
            cs.hasf = false;
        }
        if (xl >= 0) {
            cs.hascross = true;
            cs.cross = nx;
        } else if (!cont) {
            cs.hascross = false;
        }
        cs.g = gl;
    }
    // best: min (chi2, index) over chi2 < 10000.1 (K:1778)
    const bool elig = pass && chi2 < 10000.1f;
    const unsigned key = elig ? __float_as_uint(chi2) : 0xffffffffu;
    const unsigned kmin = __reduce_min_sync(0xffffffffu, key);
    if (kmin != 0xffffffffu) {
        const int win = __ffs(__ballot_sync(0xffffffffu, key == kmin)) - 1;
        const int cw = __shfl_sync(0xffffffffu, c, win);
        const unsigned long long full = ((unsigned long long)kmin << 32) | (unsigned long long)(unsigned)cw;
        if (full < cs.best) {
            cs.best = full;
            if (lane == win) {
                S.b.key = full;
                S.b.nuv = nuv;
                S.b.chi2 = chi2;
                S.b.ty = ty;
                S.b.y0 = y0;
                S.b.ety = ety;
                S.b.ey0 = ey0;
            }
            UvSet V = shfl_set(win);
            V.sign = __shfl_sync(0xffffffffu, U.sign, win);
            const float wy = __shfl_sync(0xffffffffu, y0, win), wt = __shfl_sync(0xffffffffu, ty, win);
            const int wn = __shfl_sync(0xffffffffu, nuv, win);
            if (lane < wn) {
                const int n = lane;
                const YzHit &h = base[uv_off(V, n)];
                S.b.det[n] = h.det;
                S.b.el[n] = h.el;
                S.b.pos[n] = h.pos;
                S.b.drift[n] = h.drift;
                S.b.sign[n] = uv_sign(V, n);
                S.b.tdc[n] = h.tdc;
            }
            // the winner's residuals, recomputed as chi2 formed them
            if (lane < nhx + wn) {
                float res;
                S.b.res[lane] = yz_residual(S, V, base, lane, nhx, P, x0, wy, tx, wt, res);
            }
        }
    }
    __syncwarp();
}

// Evaluate combinations [c0, c1) (whole outer iterations) of the current
// tracklet.  `st` is advanced to the scratch state after the range.  Returns
// the best key (chi2 bits << 32 | combination index) or ~0, with that
// combination's record in S.b.
//
// Phase 1 (every combination, registers only): station-3/2 load attempts in
// the reference order, the first y fit, its 2-sigma cut (K:1602-1611) and the
// scratch-entry scan.  Survivors (about 6% on the uneven batch) go to the
// warp's queue in global memory, in order.  Phase 2 (yz_phase2, 32 at a time,
// when the queue fills or the range ends): sign state, left/right walk, prop
// and hodoscope gates, chi2 (K:1613-1799).  This combined walk serves the
// planning kernel's light tracklets and the units whose survivors do not fit
// the pool; the first-cut kernel walks listed outer iterations with the
// inner pairs' lists instead (yz_first_walk).
//
// Outer iterations (iu3, iv3) whose u3 pair or v3 pair gives no accepted hit
// are skipped whole: the reference leaves such an iteration before any
// station-2 load (K:1326-1390), so it neither writes a scratch entry past a
// count of 4 nor yields a candidate, and jumping over it changes nothing.

// Pairs of lists 2 (u3) and 3 (v3) with an accepted hit, as 128-bit masks
// (at most YZ_MAXPAIR = 100 pairs per list).
struct YzAlive {
    unsigned u[4], v[4];
};

__device__ __forceinline__ YzAlive yz_alive(const YzWarp &S, const YzHit *base) {
    const int lane = lane_id();
    const YzHit *l4 = yz_list(S, base, 4), *l5 = yz_list(S, base, 5);
    const YzHit *l6 = yz_list(S, base, 6), *l7 = yz_list(S, base, 7);
    YzAlive m;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int i = w * 32 + lane;
        bool a = false, b = false;
        if (i < S.np[2]) {
            const short2 p = S.pair[2][i];
            a = (p.x >= 0 && l4[p.x].acc) || (p.y >= 0 && l5[p.y].acc);
        }
        if (i < S.np[3]) {
            const short2 p = S.pair[3][i];
            b = (p.x >= 0 && l6[p.x].acc) || (p.y >= 0 && l7[p.y].acc);
        }
        m.u[w] = __ballot_sync(0xffffffffu, a);
        m.v[w] = __ballot_sync(0xffffffffu, b);
    }
    return m;
}

__device__ __forceinline__ int bits128(const unsigned m[4]) {
    return __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
}

__device__ __forceinline__ bool bit128(const unsigned m[4], int i) {
    const unsigned w = i < 32 ? m[0] : (i < 64 ? m[1] : (i < 96 ? m[2] : m[3]));
    return (w >> (i & 31)) & 1u;
}

// first set bit at index >= p (0 <= p), or -1
__device__ __forceinline__ int next_bit128(const unsigned m[4], int p) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        if (w < (p >> 5)) continue;
        unsigned v = m[w];
        if (w == (p >> 5)) v &= ~0u << (p & 31);
        if (v) return w * 32 + __ffs(v) - 1;
    }
    return -1;
}

// first outer iteration after (iu, iv), u fastest, with both pairs alive; -1 if none
__device__ __forceinline__ int next_alive_outer(const YzAlive &m, int nu3, int iu, int iv) {
    if (bit128(m.v, iv)) {
        const int u = next_bit128(m.u, iu + 1);
        if (u >= 0) return u + iv * nu3;
    }
    const int v = next_bit128(m.v, iv + 1);
    const int u = next_bit128(m.u, 0);
    return (v < 0 || u < 0) ? -1 : u + v * nu3;
}

// index of the k-th set bit (k from 0) of a 128-bit mask, or -1
__device__ __forceinline__ int nth_bit128(const unsigned m[4], int k) {
#pragma unroll 1
    for (int w = 0; w < 4; ++w) {
        const int c = __popc(m[w]);
        if (k < c) {
            unsigned v = m[w];
#pragma unroll 1
            for (int i = 0; i < k; ++i) v &= v - 1u;
            return w * 32 + __ffs(v) - 1;
        }
        k -= c;
    }
    return -1;
}

// set bits of a 128-bit mask below index i
__device__ __forceinline__ int bits_below128(const unsigned m[4], int i) {
    int c = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        if (w < (i >> 5)) c += __popc(m[w]);
        else if (w == (i >> 5)) c += __popc(m[w] & ((1u << (i & 31)) - 1u));
    }
    return c;
}

// Distance from the hits of a prop-tube y plane at z = zp to the window of
// y the track can have there: through y3 at z3 with |ty| <= TY_MAX and
// |y0| <= Y0_MAX (the bounds the YZ hard cut enforces, K:1638), widened by
// the prop-tube match tolerance (K:1640-1702); 30 cm when there is no hit or
// no such line.
__device__ __forceinline__ float prop_gap(const HitPlane &h, float zp, float y3, float z3, float lo_t, float hi_t,
                                          float tol) {
    float d = 30.f;
    if (lo_t > hi_t) return d;
    const float ya = y3 + lo_t * (zp - z3), yb = y3 + hi_t * (zp - z3);
    const float lo = fminf(ya, yb) - tol, hi = fmaxf(ya, yb) + tol;
#pragma unroll 1
    for (int i = 0; i < h.n; ++i) {
        const float p = h.pos(i);
        d = fminf(d, fmaxf(fmaxf(lo - p, p - hi), 0.f));
    }
    return d;
}

// The combination scorer's 16 features of live outer iteration (iu, iv) of
// the current tracklet: the tracklet's x fit, the y of its u3 and v3 hits
// (mean of the accepted hits of each pair) and their difference against the
// x fit's error at station 3 -- the x error moves the two stereo estimates
// of y apart -- the distance of the P1 and P2 y-tube hits from the window
// the track's y can reach there, hit counts, the inner and outer loop sizes,
// the station-3 half and the tracklet's x-hit count.
__device__ void yz_outer_features(const YzWarp &S, const YzEvent &E, const YzHit *base, const or_plane_t &P, int iu,
                                  int iv, int st3, long C2, long Ga, float *f) {
    const short2 pu = S.pair[2][iu], pv = S.pair[3][iv];
    const YzHit *l4 = yz_list(S, base, 4), *l5 = yz_list(S, base, 5);
    const YzHit *l6 = yz_list(S, base, 6), *l7 = yz_list(S, base, 7);
    float su = 0.f, sv = 0.f;
    int nu = 0, nv = 0;
    if (pu.x >= 0 && l4[pu.x].acc) { su += l4[pu.x].Y; ++nu; }
    if (pu.y >= 0 && l5[pu.y].acc) { su += l5[pu.y].Y; ++nu; }
    if (pv.x >= 0 && l6[pv.x].acc) { sv += l6[pv.x].Y; ++nv; }
    if (pv.y >= 0 && l7[pv.y].acc) { sv += l7[pv.y].Y; ++nv; }
    const float yu = su / (float)max(nu, 1), yv = sv / (float)max(nv, 1);
    const float z3 = P.z[E.dl[4]];
    const float sig = fmaxf(S.ex0 + S.etx * z3, 1e-3f);
    const float y3 = 0.5f * (yu + yv);
    const float lo_t = fmaxf(-TY_MAX, (y3 - Y0_MAX) / z3), hi_t = fminf(TY_MAX, (y3 + Y0_MAX) / z3);
    const float d1 = fminf(prop_gap(E.p1y1, P.z[DET_P1Y1], y3, z3, lo_t, hi_t, 5.08f),
                           prop_gap(E.p1y2, P.z[DET_P1Y2], y3, z3, lo_t, hi_t, 5.08f));
    const float d2 = fminf(prop_gap(E.p2y1, P.z[DET_P2Y1], y3, z3, lo_t, hi_t, 10.16f),
                           prop_gap(E.p2y2, P.z[DET_P2Y2], y3, z3, lo_t, hi_t, 10.16f));
    f[0] = S.x0 * 0.01f;
    f[1] = S.tx * 10.f;
    f[2] = S.ex0;
    f[3] = S.etx * 100.f;
    f[4] = yu * 0.02f;
    f[5] = yv * 0.02f;
    f[6] = fminf(fmaxf((yu - yv) / sig, -20.f), 20.f) * 0.1f;
    f[7] = log1pf(fabsf(yu - yv));
    f[8] = d1 * 0.1f;
    f[9] = d2 * 0.1f;
    f[10] = (float)nu;
    f[11] = (float)nv;
    f[12] = log1pf((float)C2);
    f[13] = log1pf((float)Ga);
    f[14] = (float)(st3 - 3);
    f[15] = (float)S.nhx;
}


// Skip the pruned live outer iterations from rank r (the scorer's rows of
// the tracklet are its live outer iterations in loop order): returns the
// rank of the next kept one (nrows when none) and, when one follows, sets
// the scratch entries 4..7 as the skipped iterations' load attempts leave
// them in the reference -- for each entry, the last skipped iteration whose
// station-3 hit count puts one of its writes there -- so that the kept
// combinations read the same stale entries as in the plain run.
__device__ __noinline__ int yz_skip_pruned(const YzWarp &S, const YzHit *base, const YzAlive &al, int Au, int nrows,
                                           const float *__restrict__ osc, float t_keep, unsigned long long lasto,
                                           int r, int r_end, Stale st[4]) {
    const int lane = lane_id();
    int rk = nrows;  // no kept iteration before the range's end rank r_end
#pragma unroll 1
    for (int b = r; b < r_end; b += 32) {
        const int j = b + lane;
        const unsigned m = __ballot_sync(0xffffffffu, j < r_end && osc[j] >= t_keep);
        if (m) {
            rk = b + __ffs(m) - 1;
            break;
        }
    }
    if (rk >= nrows) return rk;
    unsigned done = 0u;
#pragma unroll 1
    for (int b = rk - 1; b >= r && done != 0xFu; b -= 32) {
        const int j = b - lane;  // lane 0 holds the latest rank of the chunk
        int n3 = 0;
        if (j >= r) {
            bool v;
            n3 = s3_count(S, base, nth_bit128(al.u, j % Au), nth_bit128(al.v, j / Au), v);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (done & (1u << k)) continue;
            const int mm = k + 4 - n3;
            const bool ok = j >= r && mm >= 0 && mm < 4 && ((lasto >> (16 * mm)) & 0xFFFFull) != 0xFFFFull;
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (m) {
                const int src = __shfl_sync(0xffffffffu, mm, __ffs(m) - 1);
                const YzHit &h = base[(int)((lasto >> (16 * src)) & 0xFFFFull)];
                const Stale v{h.det, h.pos, h.drift};
                __syncwarp();
                st[k] = v;
                done |= 1u << k;
            }
        }
    }
    __syncwarp();
    return rk;
}

// Station-3 part of the outer iteration (iu3, iv3) (K:1326-1390): the first
// y fit's right-hand side over its accepted hits in the reference order,
// their count and the table offset of the plane set.  False when the u3 or
// the v3 pair gives no accepted hit (the iteration ends before station 2).
struct Yz3 {
    float b0, b1;
    int n3, tab3;
};

__device__ __forceinline__ bool yz_station3(const YzWarp &S, const YzHit *base, int iu3, int iv3, Yz3 &o) {
    const short2 pu = S.pair[2][iu3], pv = S.pair[3][iv3];
    const unsigned long long offs = (unsigned long long)(pu.x >= 0 ? S.woff[4] + pu.x : 0xFFFF) |
                                    ((unsigned long long)(pu.y >= 0 ? S.woff[5] + pu.y : 0xFFFF) << 16) |
                                    ((unsigned long long)(pv.x >= 0 ? S.woff[6] + pv.x : 0xFFFF) << 32) |
                                    ((unsigned long long)(pv.y >= 0 ? S.woff[7] + pv.y : 0xFFFF) << 48);
    // B0 += w*y, B1 += w*y*z per accepted hit, as Fit2::add
    float b0 = 0.f, b1 = 0.f;
    int nu = 0, nv = 0, gu = 0, gv = 0;
#pragma unroll 1
    for (int a = 0; a < 4; ++a) {
        if (a == 2 && nu == 0) break;  // no u3 hit: v3 is not loaded
        const int off = (int)((offs >> (16 * a)) & 0xFFFFull);
        if (off == 0xFFFF) continue;
        const YzHit &r = base[off];
        if (!r.acc) continue;
        const float t = r.eY * r.Y;
        b0 += t;
        b1 += t * r.z;
        if (a < 2) {
            ++nu;
            gu |= 1 << a;
        } else {
            ++nv;
            gv |= 1 << (a - 2);
        }
    }
    const bool alive3 = nu > 0 && nv > 0;
    o.b0 = b0;
    o.b1 = b1;
    o.n3 = nu + nv;
    o.tab3 = alive3 ? yz_tab_index(gu, gv, 1, 1) : 0;
    return alive3;
}

// Station-2 load attempts of the inner pair (iu2, iv2) in the reference order
// (K:1467-1597) after the station-3 part s3: every attempted hit writes the
// scratch entry at the running count (4..7 at most: n3 <= 4, four attempts;
// `own` holds those writes as arena offsets, 16 bits per entry, `wmask` which
// entries), accepted ones enter the fit.  When the v2 group gives a hit and
// `fit` is set, the first y fit with the plane set's tabulated inverse and
// its 2-sigma cut (K:1602-1611).  Returns the accepted hit count.
__device__ __forceinline__ int yz_station2_fit(const YzWarp &S, const YzHit *base, int iu2, int iv2, const Yz3 &s3,
                                               bool fit, const YzTab *__restrict__ tab, unsigned long long &own,
                                               unsigned &wmask, bool &pass1, float &y0, float &ty, float &ey0,
                                               float &ety) {
    float b0 = s3.b0, b1 = s3.b1;
    int g2 = 0;  // plane bits u2 u2' v2 v2' of the accepted hits
    int nuv = s3.n3;
    const short2 pu = S.pair[0][iu2];
    auto attempt = [&](int off, int a) {
        const YzHit &r = base[off];
        const int k = nuv - 4;
        if (k >= 0) {
            const int sh = k << 4;
            own = (own & ~(0xFFFFull << sh)) | ((unsigned long long)off << sh);
            wmask |= 1u << k;
        }
        if (r.acc) {
            const float t = r.eY * r.Y;
            b0 += t;
            b1 += t * r.z;
            g2 |= 1 << a;
            ++nuv;
        }
    };
    // the four attempts as one loop body: arena offsets (0xFFFF = no hit) of
    // u2, u2', v2, v2' packed in 64 bits
    const short2 pv = S.pair[1][iv2];
    const unsigned long long offs = (unsigned long long)(pu.x >= 0 ? S.woff[0] + pu.x : 0xFFFF) |
                                    ((unsigned long long)(pu.y >= 0 ? S.woff[1] + pu.y : 0xFFFF) << 16) |
                                    ((unsigned long long)(pv.x >= 0 ? S.woff[2] + pv.x : 0xFFFF) << 32) |
                                    ((unsigned long long)(pv.y >= 0 ? S.woff[3] + pv.y : 0xFFFF) << 48);
    int nu2hits = s3.n3;
#pragma unroll 1
    for (int a = 0; a < 4; ++a) {
        if (a == 2) {
            nu2hits = nuv;
            if (nu2hits == s3.n3) break;  // the u2 group gave no hit
        }
        const int off = (int)((offs >> (16 * a)) & 0xFFFFull);
        if (off != 0xFFFF) attempt(off, a);
    }
    if (nu2hits > s3.n3 && nuv > nu2hits && fit) {  // the v2 group gave a hit: the fit is reached
        // Fit2::solve with the plane set's tabulated inverse
        const YzTab *te = tab + s3.tab3 + (g2 & 3) * 3 - 4 + (g2 >> 2);
        const float4 ai = __ldg(reinterpret_cast<const float4 *>(te));
        const float2 thr = __ldg(reinterpret_cast<const float2 *>(&te->thr_y0));
        y0 = 0.0f;
        y0 += ai.x * b0;
        y0 += ai.y * b1;
        ty = 0.0f;
        ty += ai.z * b0;
        ty += ai.w * b1;
        pass1 = !(fabsf(y0) > thr.x || fabsf(ty) > thr.y);
        if (pass1) {
            const float2 er = __ldg(reinterpret_cast<const float2 *>(&te->ey0));
            ey0 = er.x;
            ety = er.y;
        }
    }
    return nuv;
}

// One chunk's scratch entries and survivors.  Entry k+4 as the lane's
// combination c reads it: its own write, else the last earlier lane's write
// in this chunk, else the state st[] before the chunk; the chunk's last
// write becomes the new state.  `own` holds the lane's writes as arena
// offsets in the low 10 bits of 16-bit fields (entry k in field k; bits above
// them are ignored), `wmask` which entries it writes.  The survivors (pass1) go to Q[qn..] in lane
// order with the entry past their hit count; returns the new queue length.
__device__ __forceinline__ int yz_scan_queue(const YzHit *base, Stale st[4], unsigned long long own, unsigned wmask,
                                             int nuv, bool pass1, int c, float y0, float ty, float ey0, float ety,
                                             PassEntryStore *Q, int qn) {
    Stale stj{DET_SENTINEL, 0.f, 0.f};
    int stj_off = -1;
    {
        const int j = nuv;
        const unsigned lt = lanemask_lt();
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            const bool mine = (wmask >> k) & 1u;
            const int ok = (int)((own >> (16 * k)) & 0x3FFull);  // arena offsets are below 1,024
            const unsigned m = __ballot_sync(0xffffffffu, mine);
            const int src = last_lane(m & lt);
            const int so = __shfl_sync(0xffffffffu, ok, src < 0 ? 0 : src);
            if (j == k + 4) {
                if (mine) stj_off = ok;
                else if (src >= 0) stj_off = so;
                else stj = st[k];
            }
            const int lw = last_lane(m);
            if (lw >= 0) {
                const YzHit &r = base[__shfl_sync(0xffffffffu, ok, lw)];
                __syncwarp();  // every lane has read entry k
                st[k] = Stale{r.det, r.pos, r.drift};
            }
        }
    }
    if (pass1 && stj_off >= 0) {
        const YzHit &r = base[stj_off];
        stj = Stale{r.det, r.pos, r.drift};
    }
    // --- queue the survivors in order ----------------------------------
    const unsigned pm = __ballot_sync(0xffffffffu, pass1);
    if (pass1) {
        PassEntryStore e;
        e.c = c;
        e.y0 = y0;
        e.ty = ty;
        e.ey0 = ey0;
        e.ety = ety;
        e.stdet = stj.det;
        e.stpos = stj.pos;
        e.stdrift = stj.drift;
        Q[qn + __popc(pm & lanemask_lt())] = e;
    }
    qn += __popc(pm);
    __syncwarp();
    return qn;
}

template <bool PRUNE = false>
__device__ unsigned long long yz_range_t(YzWarp &S, const YzEvent &E, const YzHit *base, long c0l, long c1l,
                                         Stale st[4], const or_plane_t &P, const YzTab *__restrict__ tab,
                                         PassEntryStore *Q, int qcap, const float *__restrict__ osc = nullptr,
                                         float t_keep = 0.f) {
    const int lane = lane_id();
    const int nu2 = S.np[0], nu3 = S.np[2];
    const int C2 = S.np[0] * S.np[1];
    const int c0 = (int)c0l, c1 = (int)c1l;  // at most 100^4 combinations
    Phase2Carry cs;
    int qh = 0, qn = 0;  // survivors Q[qh..qn) wait for the full evaluation
    const int nv2 = S.np[1];
    // Lane's combination as digits (iu2, iv2, iu3, iv3) in radices (nu2, nv2,
    // nu3, nv3) -- the reference's index order (u2 fastest) -- advanced by 32
    // per chunk with carries instead of divisions.
    int d0, d1, d2, d3, s0, s1, s2, s3;
    auto set_digits = [&](int cb) {
        const int c = cb + lane;
        const int g = c / C2, r = c - g * C2;
        d0 = r % nu2;
        d1 = r / nu2;
        d2 = g % nu3;
        d3 = g / nu3;
    };
    set_digits(c0);
    {
        const int sg = 32 / C2, sr = 32 - sg * C2;
        s0 = sr % nu2;
        s1 = sr / nu2;
        s2 = sg % nu3;
        s3 = sg / nu3;
    }
    const YzAlive alive = yz_alive(S, base);
    // the combination scorer (PRUNE): live outer iterations scoring below
    // t_keep are skipped; `osc` holds the tracklet's scores in loop order
    int Au = 0, nrows = 0, r_end = 0;
    unsigned long long lasto = ~0ull;
    if constexpr (PRUNE) {
        if (osc) {
            Au = bits128(alive.u);
            nrows = Au * bits128(alive.v);
            r_end = live_before(alive.u, alive.v, nu3, (c1 + C2 - 1) / C2);  // rows of the range's outer iterations
            lasto = yz_last_writes(S, base);
        }
    }
    bool pruned3 = false;
    // station-3 part of the lane's current outer iteration (iu3, iv3): the
    // fit's right-hand side over its accepted hits in the reference order,
    // their count, the table offset of its plane set, and whether both u3
    // and v3 gave one (K:1326-1390); recomputed only when the outer digits
    // move.
    float b0_3 = 0.f, b1_3 = 0.f;
    int tab3 = 0;
    int n3 = 0;
    bool alive3 = false, need3 = true;
    int basec = c0;
    for (;;) {
        if (basec < c1) {
            // the chunk's first combination in a dead outer iteration: jump
            // to the next live one (every combination in between is dead);
            // lane 0 holds that combination's digits
            const int iu = __shfl_sync(0xffffffffu, d2, 0), iv = __shfl_sync(0xffffffffu, d3, 0);
            if (!(bit128(alive.u, iu) && bit128(alive.v, iv))) {
                const int gn = next_alive_outer(alive, nu3, iu, iv);
                basec = gn < 0 ? c1 : min(gn * C2, c1);
                if (basec < c1) set_digits(basec);
                need3 = true;
            }
        }
        if constexpr (PRUNE) {
            // the chunk's first combination in a pruned live outer
            // iteration: jump to the next kept one, with the scratch entries
            // the skipped ones write
            if (osc && basec < c1) {
                const int iu = __shfl_sync(0xffffffffu, d2, 0), iv = __shfl_sync(0xffffffffu, d3, 0);
                const int r = bits_below128(alive.v, iv) * Au + bits_below128(alive.u, iu);
                if (osc[r] < t_keep) {
                    const int rk = yz_skip_pruned(S, base, alive, Au, nrows, osc, t_keep, lasto, r, r_end, st);
                    if (rk >= nrows) {
                        basec = c1;
                    } else {
                        const int gk = nth_bit128(alive.u, rk % Au) + nth_bit128(alive.v, rk / Au) * nu3;
                        basec = min(gk * C2, c1);
                        if (basec < c1) set_digits(basec);
                    }
                    need3 = true;
                }
            }
        }
        const bool more = basec < c1;
        if (!more && qn == qh) break;
        if (more) {
            const int c = basec + lane;
            const bool valid = c < c1;
            int nuv = 0;
            // scratch entries this combination writes (offsets 4..7 past the
            // hit count): arena offsets of the hits, 16 bits each
            unsigned long long own = 0ull;
            unsigned wmask = 0u;
            float y0 = 0.f, ty = 0.f, ey0 = 0.f, ety = 0.f;
            bool pass1 = false;
            if (valid) {
                if (need3) {
                    Yz3 t3;
                    alive3 = yz_station3(S, base, d2, d3, t3);
                    b0_3 = t3.b0;
                    b1_3 = t3.b1;
                    n3 = t3.n3;
                    tab3 = t3.tab3;
                    if constexpr (PRUNE) {
                        pruned3 = osc && alive3 &&
                                  osc[bits_below128(alive.v, d3) * Au + bits_below128(alive.u, d2)] < t_keep;
                    }
                    need3 = false;
                }
                if (alive3)
                    nuv = yz_station2_fit(S, base, d0, d1, Yz3{b0_3, b1_3, n3, tab3}, !pruned3, tab, own, wmask, pass1,
                                          y0, ty, ey0, ety);
            }
            qn = yz_scan_queue(base, st, own, wmask, nuv, pass1, c, y0, ty, ey0, ety, Q, qn);
            // --- next chunk: digits + 32 -----------------------------------------
            basec += 32;
            d0 += s0;
            int cy = d0 >= nu2;
            d0 -= cy ? nu2 : 0;
            d1 += s1 + cy;
            cy = d1 >= nv2;
            d1 -= cy ? nv2 : 0;
            if (cy || s2 || s3) need3 = true;
            d2 += s2 + cy;
            cy = d2 >= nu3;
            d2 -= cy ? nu3 : 0;
            d3 += s3 + cy;
        }
        if (qn > qcap - 32 || (!more && qn > qh)) {
            // a full queue (the next chunk could add 32) or the end of the
            // range: evaluate every waiting survivor, 32 at a time, in order
            while (qh < qn) {
                const int n = min(qn - qh, 32);
                yz_phase2<false>(S, E, base, C2, P, Q + qh, n, nullptr, cs);
                qh += n;
                __syncwarp();
            }
            qh = qn = 0;
        }
    }
    return cs.best;
}


// ---------------------------------------------------------------------------
// First cut (split path)
// ---------------------------------------------------------------------------
//
// A combination is an outer iteration (u3, v3) with an inner pair (u2, v2).
// Of each projection only the pairs with an accepted hit matter; they are
// listed once per unit with their terms of the fit's right-hand side, and the
// combinations are walked over those lists, so each costs its additions, two
// dot products and two compares.
//   - Per outer iteration, 32 at a time: the sums over its station-3 hits,
//     its hit count and plane set, and the scratch entries 4..7 as the
//     iteration finds them (a last-writer scan over the live iterations
//     before it; which entries an iteration leaves depends on its hit count
//     alone, the inner pairs being the same in every one).
//   - The scratch entry past a combination's hit count is only read by the
//     left/right walk when its last hit is a v2 hit without its partner
//     plane's, and only pairs with a hit of that plane; the last writer of
//     that entry follows from the lists (yz_stale_code).
// Combinations that pass wait in a ring in shared memory; 32 at a time they
// go through the prop-tube and hodoscope gates, all lanes in use.  Only those
// that pass reach the survivor kernel, with the two kinds that set station-3
// signs for them: the first survivor of their outer iteration, and the
// survivors whose walk pairs the last station-3 hit with the first station-2
// hit (planes 19, 18).
//
// Bound: instruction issue.  Rebuilding each combination's station-3 part and
// attempts, scanning the scratch entries over every chunk of 32 and passing
// every survivor on took 22.9 ms of the 100,000-event uneven batch with 19.5
// ms in the survivor kernel; this takes 8.9 ms with 6.2 ms.
constexpr int YZ_KEPT_BATCH = 32;  // outer iterations listed at a time
constexpr int YZ_LIST_SMEM = 48;   // pairs per projection listed in shared memory; a unit with more uses the
                                   // warp's overflow arena
constexpr int YZ_PROP_SMEM = 40;   // hits per prop-tube y plane kept in shared memory
static_assert(4 * YZ_MAXPAIR * (sizeof(float4) + 4) <= YZ_GARENA_HITS * sizeof(YzHit), "the lists fit the arena");

// hodoscope x planes of stations 2-4 and the prop-tube y planes
struct YzGate {
    float hz[6], ymin[6], ymax[6];
    float pz[4];
};

struct YzFirstWarp {
    uint4 ring[64];  // survivors waiting for the gates (YzSurv; code bit 21: may pair planes 19 and 18)
    float4 term[4][YZ_LIST_SMEM];   // u2 v2 u3 v3 pairs with an accepted hit: (eY Y, eY Y z) of each hit, 0 if refused
    unsigned info[4][YZ_LIST_SMEM]; // pair | planes << 7; v2: | latest earlier pair with two attempts << 16
    unsigned long long kent[YZ_KEPT_BATCH];  // scratch entries 4..7, 16 bits each: arena offset, 0xFFFF = the unit's
    float2 kb[YZ_KEPT_BATCH];
    unsigned kt[YZ_KEPT_BATCH];  // pairs u3, v3 | table offset << 14 | planes << 21 | n3 << 25
    uint4 pend;                  // the current outer iteration's first survivor, not passed on yet
    float prop[4][YZ_PROP_SMEM];
    HitPlane pp[4];
    int np[4], woff[8];
};

// What the scratch entries need to know of a unit's u2 and v2 pairs.
struct YzInner {
    const uint4 *hits;    // the image's arena
    const short2 *pu, *pv;
    int ou, ov, ova;      // arena offsets of the lists u2', v2' and v2
    YzLast u, v;
    int first_two;        // first u2 pair with two accepted hits
};

__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

__device__ __forceinline__ bool yz_img_acc(const uint4 *hits, int off) { return hits[2 * off + 1].w != 0u; }

// List the pairs of projection q with an accepted hit, in order; returns
// their number.
__device__ __forceinline__ int yz_first_list(const YzFirstWarp &S, int q, const short2 *__restrict__ pair,
                                             const uint4 *__restrict__ hits, float4 *term, unsigned *info, YzLast &last,
                                             int &first_two) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const int n = S.np[q], oa = S.woff[2 * q], ob = S.woff[2 * q + 1];
    last = YzLast{-1, -1, -1};
    first_two = 1 << 20;
    int count = 0;
#pragma unroll 1
    for (int b0 = 0; b0 < n; b0 += 32) {
        const int i = b0 + lane;
        int g = 0;
        bool r1 = false;
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) {
            const short2 p = pair[i];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const int k = a == 0 ? p.x : p.y;
                if (k < 0) continue;
                const int off = (a == 0 ? oa : ob) + k;
                const uint4 v = hits[2 * off + 1];  // tdc, z, det | el, acc
                if (v.w == 0u) continue;
                const float2 ye = *reinterpret_cast<const float2 *>(hits + 2 * off);
                const float s = ye.y * ye.x, sz = s * __uint_as_float(v.y);
                g |= 1 << a;
                if (a == 0) {
                    t.x = s;
                    t.y = sz;
                } else {
                    t.z = s;
                    t.w = sz;
                }
            }
            r1 = (g & 1) && p.y >= 0;
        }
        const unsigned m1 = __ballot_sync(0xffffffffu, g == 1 || g == 2);
        const unsigned m2 = __ballot_sync(0xffffffffu, g == 3);
        const unsigned mr = __ballot_sync(0xffffffffu, r1);
        if (g) {
            const int k = count + __popc((m1 | m2) & lt);
            const int pr = last_lane(mr & lt);
            term[k] = t;
            info[k] = (unsigned)(i | g << 7) | (unsigned)(pr >= 0 ? b0 + pr : (last.r1 >= 0 ? last.r1 : 255)) << 16;
        }
        count += __popc(m1 | m2);
        if (m2 && last.two < 0) first_two = b0 + __ffs(m2) - 1;
        if (m1) last.one = b0 + last_lane(m1);
        if (m2) last.two = b0 + last_lane(m2);
        if (mr) last.r1 = b0 + last_lane(mr);
    }
    return count;
}

// Code of the scratch entry past the hits of the combination of u2 pair ui
// and v2 pair vi (info words), in an outer iteration of n3 hits that finds
// the entries `ent`: the latest attempt at that offset, by this combination,
// an earlier one of the iteration, or before the iteration.
__device__ __forceinline__ unsigned yz_stale_code(const YzInner &I, unsigned ui, unsigned vi, int n3,
                                                  unsigned long long ent) {
    const int iu = (int)(ui & 127u), gu = (int)(ui >> 7) & 3, iv = (int)(vi & 127u), gv = (int)(vi >> 7) & 3;
    const int prev = (int)(vi >> 16);
    if (gv == 3) return 0u;  // v2 and v2' pair with each other
    const int cu = gu == 3 ? 2 : 1;
    int off = -1;
    bool before = false;
    if (gv == 1 && I.pv[iv].y >= 0) {
        off = I.ov + I.pv[iv].y;  // its own refused v2' hit
    } else if (cu == 1 && I.first_two < iu) {
        return 0u;  // this v2 pair's own hit, tried after two u2 hits
    } else if (cu == 1 && I.u.two >= 0) {
        if (iv == 0) {
            before = true;
        } else if (I.u.one > I.u.two && prev == iv - 1) {
            off = I.ov + I.pv[prev].y;
        } else {
            const short2 p = I.pv[iv - 1];
            const bool sec = p.x < 0 || (!yz_img_acc(I.hits, I.ova + p.x) && p.y >= 0);
            off = sec ? I.ov + p.y : I.ova + p.x;
        }
    } else if (prev != 255) {
        off = I.ov + I.pv[prev].y;
    } else {
        before = true;
    }
    if (before) {
        const int e = n3 + cu + 1 - 4;  // entry 4 + e
        if (e > 3) return 0u;
        const unsigned o = (unsigned)(ent >> (16 * e)) & 0xFFFFu;
        return o == 0xFFFFu ? (YZ_ENT_UNIT << 10) | ((unsigned)e << 12) : o | (YZ_ENT_HIT << 10);
    }
    return (unsigned)off | (YZ_ENT_HIT << 10);
}

// The event's prop-tube y planes and, for the tracklet's x fit, which of the
// six hodoscope x planes (bit 2q + c) hold a hit in its x window: that part
// of match_tracklet_to_hodo (H:1002-1087) does not depend on the y fit, and
// its y window is the same for every hit of a plane.
__device__ __forceinline__ unsigned yz_first_event(YzFirstWarp &S, const or_hits_view_t &hv, long e,
                                                   const YzGate &G, const or_plane_t *__restrict__ P, float x0,
                                                   float tx, float ex0, float etx) {
    const int lane = lane_id();
    bool has = false;
    if (lane < 4) {
        S.pp[lane] = hits_of(hv, e, lane == 0 ? DET_P1Y1 : lane == 1 ? DET_P1Y2 : lane == 2 ? DET_P2Y1 : DET_P2Y2);
    } else if (lane < 10) {
        const int i = lane - 4;
        int stid = (i >> 1) + 1;
        const int det = c_hodoplanesx[stid][i & 1];
        const HitPlane h = hits_of(hv, e, det);
        if (det > 40) stid = 3;
        const float fudgefac = c_hodofudgefac[stid];
        const float cellwidth = __ldg(&P->cellwidth[det]);
        const float xhodo = G.hz[i] * tx + x0;
        float err_x = 3.f * (fabsf(G.hz[i] * etx) + ex0);
#pragma unroll 4
        for (int k = 0; k < h.n; ++k) {
            const float p = h.pos(k);
            float xmin = p - cellwidth * 0.5f;
            float xmax = p + cellwidth * 0.5f;
            xmin -= (xmax - xmin) * fudgefac;
            xmax += (xmax - xmin) * fudgefac;
            err_x += (xmax - xmin) * 0.15f;
            xmin -= err_x;
            xmax += err_x;
            has |= xmin <= xhodo && xhodo <= xmax;
        }
    }
    __syncwarp();
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = lane < min(S.pp[q].n, YZ_PROP_SMEM) ? S.pp[q].pos(lane) : 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int n = min(S.pp[q].n, YZ_PROP_SMEM);
        if (lane < n) S.prop[q][lane] = v[q];
#pragma unroll 1
        for (int i = lane + 32; i < n; i += 32) S.prop[q][i] = S.pp[q].pos(i);
    }
    return __ballot_sync(0xffffffffu, has) >> 4;
}

// a hit of prop-tube plane q within tol of e (prop_hits, K:1640-1701), for
// the lanes with `want`
__device__ __forceinline__ bool yz_prop_plane(const YzFirstWarp &S, int q, float e, float tol, bool want) {
    const int n = S.pp[q].n;
    bool ok = false;
    const int m = min(n, YZ_PROP_SMEM);
#pragma unroll 4
    for (int i = 0; i < m; ++i) ok |= fabsf(S.prop[q][i] - e) < tol;
#pragma unroll 1
    for (int i = m; i < n && __any_sync(0xffffffffu, want && !ok); ++i) ok |= fabsf(S.pp[q].pos(i) - e) < tol;
    return ok && want;
}

// the gates of a survivor (yz_gates), every lane of the warp
__device__ __forceinline__ bool yz_first_gates(const YzFirstWarp &S, const YzGate &G, unsigned hasx, bool valid, float y0,
                                               float ty, float ey0, float ety) {
    bool ok = valid && !(fabsf(y0) > Y0_MAX || fabsf(ty) > TY_MAX);
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {
        bool m = false;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int i = 2 * q + c;
            const float yhodo = G.hz[i] * ty + y0;
            const float err_y = 3.f * (fabsf(G.hz[i] * ety) + ey0);
            m |= ((hasx >> i) & 1u) && G.ymin[i] - err_y <= yhodo && yhodo <= G.ymax[i] + err_y;
        }
        ok = ok && m;
    }
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
        if (!__any_sync(0xffffffffu, ok)) return false;
        bool found = false;
#pragma unroll 1
        for (int q = 2 * s; q < 2 * s + 2 && __any_sync(0xffffffffu, ok && !found); ++q)
            found |= yz_prop_plane(S, q, ty * G.pz[q] + y0, s ? 10.16f : 5.08f, ok && !found);
        ok = found;
    }
    return ok;
}

// State of the survivors' order from one ring chunk to the next.
struct YzOrder {
    unsigned g = ~0u;   // outer iteration (its pairs) of the last survivor
    bool pend = false;  // its first survivor waits in S.pend
};

// Up to 32 survivors from the ring, in order: the gates, then those the
// survivor kernel needs go to Q; returns the new queue length.  Out of line:
// it runs once per 32 survivors.
__device__ __noinline__ int yz_first_pass(YzFirstWarp &S, const YzGate &G, unsigned hasx, int head, int n,
                                          const YzTab *__restrict__ tab, YzOrder &od, YzSurv *Q, int qn) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const bool valid = lane < n;
    const uint4 v = S.ring[(head + lane) & 63];
    const float y0 = __uint_as_float(v.y), ty = __uint_as_float(v.z);
    float2 er = make_float2(0.f, 0.f);
    if (valid) er = __ldg(reinterpret_cast<const float2 *>(&tab[(v.w >> 14) & 0x7Fu].ey0));
    const bool pass = yz_first_gates(S, G, hasx, valid, y0, ty, er.x, er.y);
    const unsigned g = valid ? v.x & 0x3FFFu : 0x10000u + lane;
    const unsigned gp = __shfl_up_sync(0xffffffffu, g, 1);
    const bool first = valid && g != (lane == 0 ? od.g : gp);
    const bool keep = valid && (pass || ((v.w >> 21) & 1u));
    const unsigned seg = __match_any_sync(0xffffffffu, g);
    const unsigned km = __ballot_sync(0xffffffffu, keep);
    const bool emit = keep || (first && (km & seg) != 0u);
    const unsigned em = __ballot_sync(0xffffffffu, emit);
    auto put = [&](int at, uint4 w, bool gate) {
        w.w = (w.w & 0x3FDFFFFFu) | (gate ? 0x80000000u : 0u);
        *reinterpret_cast<uint4 *>(Q + at) = w;
    };
    // the iteration carried from the last chunk: its first survivor goes
    // before the first one kept here
    const unsigned cont = __ballot_sync(0xffffffffu, valid && g == od.g);
    if (od.pend && (km & cont)) {
        if (lane == 0) put(qn, S.pend, false);
        ++qn;
        od.pend = false;
    }
    if (emit) put(qn + __popc(em & lt), v, pass);
    qn += __popc(em);
    // the chunk's last iteration may go on
    const int last = n - 1;
    const unsigned gl = __shfl_sync(0xffffffffu, g, last);
    if (gl != od.g) {
        const unsigned segl = __shfl_sync(0xffffffffu, seg, last);
        od.pend = (km & segl) == 0u;
        od.g = gl;
        __syncwarp();
        if (od.pend && lane == __ffs(segl) - 1) S.pend = v;
    }
    __syncwarp();
    return qn;
}

// The first cut of one unit, ranks [r0, r1) of the tracklet's live outer
// iterations.  `term` / `info`: the four lists (stride `cap`), of na[q]
// entries.  Returns the survivors passed on in Q, or -1 when the queue could
// overflow (the unit then runs on the combined path); *count = the
// combinations that passed the cut.
template <bool PRUNE>
__device__ __forceinline__ int yz_first_walk(YzFirstWarp &S, const YzGate &G, unsigned hasx, const float4 *term,
                                             const unsigned *info, int cap, const int na[4], const YzInner &I,
                                             unsigned long long lasto, int r0, int r1, bool half_p,
                                             const YzTab *__restrict__ tab, YzSurv *Q, int qcap,
                                             const float *__restrict__ osc, float t_keep, int *count) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    const int nu2 = na[0], nf = na[0] * na[1], nu3 = na[2];
    const float4 *tu = term, *tv = term + cap, *tu3 = term + 2 * cap, *tv3 = term + 3 * cap;
    const unsigned *iu = info, *iv = info + cap, *iu3 = info + 2 * cap, *iv3 = info + 3 * cap;
    // a chunk's step in the digits (u2, v2, outer)
    const int s2 = 32 / nf, sr = 32 - s2 * nf, s1 = sr / nu2, s0 = sr - s1 * nu2;
    const int l2 = lane / nf, lr = lane - l2 * nf, l1 = lr / nu2, l0 = lr - l1 * nu2;
    int qn = 0, nsurv = 0;
    int head = 0, waiting = 0;
    YzOrder od;
    unsigned long long carry = ~0ull;  // scratch entries as the next iteration finds them
#pragma unroll 1
    for (int b = r0; b < r1; b += 32) {
        // --- list the outer iterations of ranks b .. b+31 ------------------
        const int j = b + lane;
        const bool in = j < r1;
        bool kept = false;
        unsigned long long w = ~0ull;  // the entries this iteration writes
        float b0 = 0.f, b1 = 0.f;
        unsigned kt = 0u;
        if (in) {
            kept = !(PRUNE && osc) || osc[j] >= t_keep;
            const int jv = j / nu3, ju = j - jv * nu3;
            const float4 a = tu3[ju], c = tv3[jv];
            const unsigned ia = iu3[ju], ic = iv3[jv];
            const int gu = (int)(ia >> 7) & 3, gv = (int)(ic >> 7) & 3;
            // the hits in order; a refused one adds 0
            b0 = a.x;
            b1 = a.y;
            b0 += a.z;
            b1 += a.w;
            b0 += c.x;
            b1 += c.y;
            b0 += c.z;
            b1 += c.w;
            const int n3 = __popc(gu) + __popc(gv);
            kt = (ia & 127u) | (ic & 127u) << 7 | (unsigned)yz_tab_index(gu, gv, 1, 1) << 14 |
                 (unsigned)(gu | gv << 2) << 21 | (unsigned)n3 << 25;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int mm = k + 4 - n3;
                if (mm < 4) w = (w & ~(0xFFFFull << (16 * k))) | (((lasto >> (16 * mm)) & 0xFFFFull) << (16 * k));
            }
        }
        unsigned long long ent = 0ull;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned wk = (unsigned)(w >> (16 * k)) & 0xFFFFu;
            const unsigned wm = __ballot_sync(0xffffffffu, wk != 0xFFFFu);
            const int src = last_lane(wm & lt);
            const unsigned v = __shfl_sync(0xffffffffu, wk, src < 0 ? 0 : src);
            const unsigned c = (unsigned)(carry >> (16 * k)) & 0xFFFFu;
            ent |= (unsigned long long)(src >= 0 ? v : c) << (16 * k);
            if (wm) {
                const unsigned long long l = __shfl_sync(0xffffffffu, wk, last_lane(wm));
                carry = (carry & ~(0xFFFFull << (16 * k))) | (l << (16 * k));
            }
        }
        const unsigned km = __ballot_sync(0xffffffffu, kept);
        __syncwarp();  // every lane is done with the previous list
        if (kept) {
            const int pos = __popc(km & lt);
            S.kb[pos] = make_float2(b0, b1);
            S.kt[pos] = kt;
            S.kent[pos] = ent;
        }
        __syncwarp();
        // --- their combinations, 32 a chunk ----------------------------------
        const int ctot = __popc(km) * nf;
        int d0 = l0, d1 = l1, d2 = l2;
#pragma unroll 1
        for (int cb = 0; cb < ctot; cb += 32) {
            bool pass = false;
            float y0 = 0.f, ty = 0.f;
            unsigned t3 = 0u, ui = 0u, vi = 0u, ti = 0u;
            if (cb + lane < ctot) {
                t3 = S.kt[d2];
                const float2 s = S.kb[d2];
                ui = iu[d0];
                vi = iv[d1];
                const float4 a = tu[d0], c = tv[d1];
                // the station-2 hits in order; a refused one adds 0
                float f0 = s.x + a.x, f1 = s.y + a.y;
                f0 += a.z;
                f1 += a.w;
                f0 += c.x;
                f1 += c.y;
                f0 += c.z;
                f1 += c.w;
                // Fit2::solve with the plane set's tabulated inverse
                ti = ((t3 >> 14) & 0x7Fu) + ((ui >> 7) & 3u) * 3u - 4u + ((vi >> 7) & 3u);
                const YzTab *te = tab + ti;
                const float4 ai = __ldg(reinterpret_cast<const float4 *>(te));
                const float2 thr = __ldg(reinterpret_cast<const float2 *>(&te->thr_y0));
                y0 = 0.0f;
                y0 += ai.x * f0;
                y0 += ai.y * f1;
                ty = 0.0f;
                ty += ai.z * f0;
                ty += ai.w * f1;
                pass = !(fabsf(y0) > thr.x || fabsf(ty) > thr.y);
            }
            const unsigned pm = __ballot_sync(0xffffffffu, pass);
            if (pm) {
                if (pass) {
                    const unsigned g3 = (t3 >> 21) & 15u, g2 = ((ui >> 7) & 3u) | ((vi >> 7) & 3u) << 2;
                    unsigned code = yz_stale_code(I, ui, vi, (int)(t3 >> 25), S.kent[d2]) | ti << 14 | (g3 | g2 << 4) << 22;
                    // only v3' of the v3 pair, and a hit of plane 18
                    if (half_p && (g3 >> 2) == 2u && (g2 & 1u)) code |= 1u << 21;
                    S.ring[(head + waiting + __popc(pm & lt)) & 63] =
                        make_uint4((t3 & 0x3FFFu) | (ui & 127u) << 14 | (vi & 127u) << 21, __float_as_uint(y0),
                                   __float_as_uint(ty), code);
                }
                waiting += __popc(pm);
                nsurv += __popc(pm);
                __syncwarp();
                if (waiting >= 32) {
                    qn = yz_first_pass(S, G, hasx, head, 32, tab, od, Q, qn);
                    head = (head + 32) & 63;
                    waiting -= 32;
                    if (qn > qcap - 34) return -1;
                }
            }
            d0 += s0;
            int cy = d0 >= nu2;
            d0 -= cy ? nu2 : 0;
            d1 += s1 + cy;
            cy = d1 >= na[1];
            d1 -= cy ? na[1] : 0;
            d2 += s2 + cy;
        }
    }
    if (waiting) qn = yz_first_pass(S, G, hasx, head, waiting, tab, od, Q, qn);
    *count = nsurv;
    return qn;
}

// The combined evaluation of a range, out of line: the survivor kernel runs
// it only for units whose survivors did not fit the pool, the planning
// kernel for light tracklets, and inlined its registers would weigh on the
// rest of those kernels.
template <bool PRUNE>
__device__ __noinline__ unsigned long long yz_range_ool(YzWarp &S, const YzEvent &E, const YzHit *base, long c0l,
                                                        long c1l, Stale *st, const or_plane_t &P, const YzTab *tab,
                                                        PassEntryStore *Q, int qcap, const float *osc, float t_keep) {
    return yz_range_t<PRUNE>(S, E, base, c0l, c1l, st, P, tab, Q, qcap, osc, t_keep);
}

// write the best combination into the track record (K:1804-1825)
__device__ __forceinline__ void yz_store(float *T, const YzBest &b, int nhx) {
    const int lane = lane_id();
    const int nuv = b.nuv;
    if (lane == 0) {
        T[OR_TRK_STID] = 5.f;
        T[OR_TRK_NHITS] = (float)nhx + (float)nuv;
        T[OR_TRK_CHI2] = b.chi2;
        T[OR_TRK_TY] = b.ty;
        T[OR_TRK_Y0] = b.y0;
        T[OR_TRK_ERR_TY] = b.ety;
        T[OR_TRK_ERR_Y0] = b.ey0;
    }
    if (lane < nuv) {
        const int n = lane;
        T[OR_TRK_HIT_DETID + nhx + n] = b.det[n];
        T[OR_TRK_HIT_CHAN + nhx + n] = b.el[n];
        T[OR_TRK_HIT_POS + nhx + n] = b.pos[n];
        T[OR_TRK_HIT_DRIFT + nhx + n] = b.drift[n];
        T[OR_TRK_HIT_SIGN + nhx + n] = b.sign[n];
        T[OR_TRK_HIT_TDC + nhx + n] = b.tdc[n];
        if (n < nhx) T[OR_TRK_HIT_RESID + n] = b.res[n];
        T[OR_TRK_HIT_RESID + nhx + n] = b.res[nhx + n];
    }
}

// the result of a heavy tracklet: its best combination (K:1804-1825) and,
// for the scorer's labels, that combination's outer index
__device__ __forceinline__ void yz_finish(const YzScratch &sc, int heavy, int c2, float *T, unsigned long long key,
                                          const YzBest &b, int nhx) {
    if (key == ~0ull) return;  // best_g stays -1
    if (lane_id() == 0) sc.heavy[heavy].best_g = (int)((unsigned)key / (unsigned)max(c2, 1));
    yz_store(T, b, nhx);
}

__device__ __forceinline__ YzHit *yz_garena(const YzScratch &sc, int gwarp) {
    return sc.garena + (long)(gwarp % sc.garena_warps) * YZ_GARENA_HITS;
}

// Work of a tracklet's first cut, from its pair lists: a combination reaches
// the first y fit when each of the u3, v3, u2 and v2 pairs gives an accepted
// hit, so the fitted combinations are the product of the four counts of such
// pairs, and the sum of their hit counts follows from each projection's
// accepted hits.  Returned on every lane.
__device__ void yz_fit_counts(const YzWarp &S, const YzHit *base, unsigned long long &fitted,
                              unsigned long long &hitsum) {
    const int lane = lane_id();
    unsigned long long A[4], H[4];
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const YzHit *la = yz_list(S, base, 2 * q), *lb = yz_list(S, base, 2 * q + 1);
        unsigned a = 0, h = 0;
#pragma unroll 1
        for (int i = lane; i < S.np[q]; i += 32) {
            const short2 p = S.pair[q][i];
            const unsigned k = (p.x >= 0 && la[p.x].acc ? 1u : 0u) + (p.y >= 0 && lb[p.y].acc ? 1u : 0u);
            a += k > 0;
            h += k;
        }
        A[q] = __reduce_add_sync(0xffffffffu, a);
        H[q] = __reduce_add_sync(0xffffffffu, h);
    }
    fitted = A[0] * A[1] * A[2] * A[3];
    hitsum = H[0] * A[1] * A[2] * A[3] + A[0] * H[1] * A[2] * A[3] + A[0] * A[1] * H[2] * A[3] +
             A[0] * A[1] * A[2] * H[3];
}

__device__ __forceinline__ void yz_flush_counts(const YzScratch &sc, unsigned long long fitted,
                                                unsigned long long hitsum, unsigned long long nsurv) {
    unsigned long long *c = reinterpret_cast<unsigned long long *>(sc.counters);
    if (fitted) atomicAdd(c + YZ_CTR_FITTED / 2, fitted);
    if (hitsum) atomicAdd(c + YZ_CTR_HITSUM / 2, hitsum);
    if (nsurv) atomicAdd(c + YZ_CTR_SURVIVORS / 2, nsurv);
}

template <int W>
__global__ void __launch_bounds__(W * 32, (OR_YZ_PLAN_WARPS_SM / W > 0 ? OR_YZ_PLAN_WARPS_SM / W : 1))
    yz_plan_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv,
                   const uint8_t *__restrict__ toomany, int n_events, int chunk, YzScratch sc,
                   uint32_t *__restrict__ errw, YzPrune prune) {
    extern __shared__ __align__(16) unsigned char yz_smem[];
    or_plane_t &P = *reinterpret_cast<or_plane_t *>(yz_smem);
    YzWarp *warps = reinterpret_cast<YzWarp *>(yz_smem + ((sizeof(or_plane_t) + 15) & ~size_t(15)));
    load_plane_smem(&P, gplane);
    __syncthreads();
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    YzWarp &S = warps[w];
    YzHit *garena = yz_garena(sc, blockIdx.x * W + w);
    PassEntryStore *Q = sc.qbuf + (long)((blockIdx.x * W + w) % sc.garena_warps) * sc.qcap;
    if (lane == 0) S.nsurv = 0ull;
    unsigned long long n_fitted = 0ull, n_hitsum = 0ull;  // lane 0's work counters

    // planning units (event, `chunk` slots) from a device counter: slots are
    // independent (one reference thread each), events very uneven
    const int per_event = OR_NSLOTS / chunk;
    const unsigned long long nall = (unsigned long long)n_events * per_event;
    const unsigned nlarge = sc.list ? sc.counters[6] : 0u;
    const unsigned long long nplan = sc.list ? (unsigned long long)nlarge + sc.counters[7] : nall;
    unsigned long long *plan_ctr = reinterpret_cast<unsigned long long *>(sc.counters + 4);
    // the next unit is taken while the current one is worked on; with no more
    // units than warps each warp has its own
    const bool own = nplan <= (unsigned long long)gridDim.x * W;
    unsigned long long nxt = own ? (unsigned long long)w * gridDim.x + blockIdx.x : 0ull;
    if (!own && lane == 0) nxt = atomicAdd(plan_ctr, 1ull);
    for (;;) {
        const unsigned long long pt = __shfl_sync(0xffffffffu, nxt, 0);
        if (pt >= nplan) break;
        nxt = nplan;
        if (!own && lane == 0) nxt = atomicAdd(plan_ctr, 1ull);
        const unsigned long long pu =
            sc.list ? (unsigned long long)sc.list[pt < nlarge ? pt : nall - 1 - (pt - nlarge)] : pt;
        const long e = (long)(pu / per_event);
        const int slot0 = (int)(pu % per_event) * chunk;
        if (toomany[e]) continue;  // K:873-878
        long budget = YZ_CHUNK_INLINE;
        long row = 0;  // scorer row of the next tracklet (slots in order, tracklets in slot order)
        if (prune.keep) {
            row = prune.row_off[e];
#pragma unroll 1
            for (int s = 0; s < slot0; ++s) row += min((int)tv.ntracks[e * OR_NSLOTS + s], OR_SLOTCAP);
        }
#pragma unroll 1
        for (int slot = slot0; slot < slot0 + chunk; ++slot) {
            const int ntr = min((int)tv.ntracks[e * OR_NSLOTS + slot], OR_SLOTCAP);
            const long slot_row = row;
            row += ntr;
            if (ntr == 0) continue;
            const int st3 = 3 + (slot & 1);  // K:884
            YzEvent &E = S.ev;
            __syncwarp();  // every lane is done with the previous slot's views
            yz_event_planes(E, hv, e, st3, prune.ofeat == nullptr);
            Stale *st = S.st;
            if (lane < 4) st[lane] = Stale{DET_SENTINEL, 0.f, 0.f};
            __syncwarp();
#pragma unroll 1
            for (int it = 0; it < ntr; ++it) {
                float *T = trk_rec(tv, e, slot, it);
                const YzHit *base;
                const bool fits = yz_build(S, E, T, P, st3, base, garena);
                if (lane == 0) T[OR_TRK_STID] = 3.f;  // K:1285
                if (!fits) {
                    if (lane == 0) atomicOr(errw, ERRW_CAPACITY);
                    continue;
                }
                const int nu2 = S.np[0], nv2 = S.np[1], nu3 = S.np[2], nv3 = S.np[3];
                if (nu2 == 0 || nu3 == 0 || nv2 == 0 || nv3 == 0) continue;
                const long C2 = (long)nu2 * nv2;
                const long G = (long)nu3 * nv3;
                if (prune.keep) {
                    const long r = slot_row + it;
                    if (r < prune.max_rows && !prune.keep[r]) {
                        // pruned: no combination is evaluated, as when none
                        // passes; the scratch entries still advance over its
                        // load pattern so later tracklets of the slot see the
                        // plain state
                        yz_unit_states(S, base, (int)G, 1, st, nullptr, 0);
                        __syncwarp();
                        continue;
                    }
                }
                const YzAlive al = yz_alive(S, base);
                const long Ga = (long)bits128(al.u) * bits128(al.v);  // live outer iterations
                if (Ga == 0) continue;  // no candidate and no scratch entry past 3 written
                if (sc.count_work) {
                    unsigned long long f, h;
                    yz_fit_counts(S, base, f, h);
                    n_fitted += f;
                    n_hitsum += h;
                }
                const long C = G * C2;
                const long Cl = Ga * C2 + G;  // live combinations, plus one step per outer iteration
                // Light tracklets are evaluated here only with score rows
                // (which ones have rows follows from it); without, queueing
                // them too is faster (planning pass of 10,000 one-dimuon
                // events 729 -> 548 us, both unit kernels 543 -> 580 us).
                bool inline_it = prune.ofeat && Cl <= YZ_LIGHT && Cl <= budget;
                if (!inline_it) {
                    // whole outer iterations per unit, about YZ_UNIT live combinations each
                    const long gper = max(1L, min(G, (YZ_UNIT * G) / (Ga * C2)));
                    const int nunits = (int)((G + gper - 1) / gper);
                    int hid = 0, u0 = 0;
                    if (lane == 0) {
                        hid = (int)atomicAdd(&sc.counters[1], 1u);
                        u0 = (int)atomicAdd(&sc.counters[0], (unsigned)nunits);
                    }
                    hid = __shfl_sync(0xffffffffu, hid, 0);
                    u0 = __shfl_sync(0xffffffffu, u0, 0);
                    if (hid >= sc.cap_heavy || (long)u0 + nunits > sc.cap_units) {
                        // no room on the queue: evaluate here; void the reserved units
#pragma unroll 1
                        for (int u = lane; u < nunits; u += 32)
                            if (u0 + u < sc.cap_units) sc.units[u0 + u].heavy = -1;
                        if (lane == 0 && hid < sc.cap_heavy) sc.heavy[hid].nunits = 0;
                        inline_it = true;
                    } else {
                        // the combination scorer's rows: one per live outer iteration
                        int orow0 = -1;
                        if (prune.ofeat) {
                            yz_xhits(S, T, P);
                            unsigned r0 = 0u;
                            if (lane == 0) r0 = atomicAdd(prune.orows, (unsigned)Ga);
                            r0 = __shfl_sync(0xffffffffu, r0, 0);
                            if ((long)r0 + Ga <= prune.cap_orows) {
                                orow0 = (int)r0;
                                const int Au = bits128(al.u);
#pragma unroll 1
                                for (long r = lane; r < Ga; r += 32) {
                                    const int iu = nth_bit128(al.u, (int)(r % Au)), iv = nth_bit128(al.v, (int)(r / Au));
                                    float f[OR_NFEAT];
                                    yz_outer_features(S, E, base, P, iu, iv, st3, C2, Ga, f);
                                    float4 *dst = reinterpret_cast<float4 *>(prune.ofeat + (r0 + r) * OR_NFEAT);
#pragma unroll
                                    for (int q = 0; q < OR_NFEAT / 4; ++q)
                                        dst[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
                                    prune.og[r0 + r] = iu + iv * nu3;
                                }
                            }
                        }
                        const int img = sc.img_cap > 0 ? yz_store_image(S, base, sc) : -1;
                        if (lane == 0) {
                            YzHeavy hv2;
                            hv2.img = img;
                            hv2.e = (int)e;
                            hv2.slot = slot;
                            hv2.k = it;
                            hv2.unit0 = u0;
                            hv2.nunits = nunits;
                            hv2.orow0 = orow0;
                            hv2.nrows = (int)Ga;
                            hv2.c2 = (int)C2;
                            hv2.best_g = -1;
                            sc.heavy[hid] = hv2;
                        }
                        if (nunits == 1) {
                            if (lane < 4) sc.units[u0].entry[lane] = st[lane];
                            if (lane == 4) {
                                YzUnit &un = sc.units[u0];
                                un.heavy = hid;
                                un.g0 = 0;
                                un.g1 = (int)G;
                                un.pad = 0;
                                un.r0 = 0;
                                un.r1 = (int)Ga;
                            }
                            __syncwarp();
                            // the entries the slot's next tracklet finds
                            if (it + 1 < ntr) yz_final_state(S, base, st);
                        } else {
                            yz_unit_states(S, base, (int)G, (int)gper, st, sc.units + u0, hid, al.u, al.v);
                        }
                    }
                }
                if (inline_it) {
                    budget -= Cl;
                    yz_xhits(S, T, P);
                    if (!prune.ofeat) {  // the gates' planes were not loaded
                        yz_event_planes(E, hv, e, st3);
                        __syncwarp();
                    }
                    const unsigned long long bk =
                        yz_range_ool<false>(S, E, base, 0, C, st, P, sc.tab + YZ_TAB_SETS * (st3 - 3), Q, sc.qcap,
                                            nullptr, 0.f);
                    __syncwarp();
                    if (bk != ~0ull) yz_store(T, S.b, S.nhx);
                }
                __syncwarp();
            }
        }
    }
    __syncwarp();
    if (lane == 0 && sc.count_work) yz_flush_counts(sc, n_fitted, n_hitsum, S.nsurv);
}

// the scores of a queued tracklet's live outer iterations, when the
// combination scorer prunes it (rows written, event not uncertain)
__device__ __forceinline__ const float *yz_tracklet_scores(const YzPrune &prune, const YzHeavy &h) {
    if (!prune.model || h.orow0 < 0 || (prune.unc && prune.unc[h.e])) return nullptr;
    return prune.oscore + h.orow0;
}

// persistent warps drain the unit queue
template <int W, bool PRUNE>
__global__ void __launch_bounds__(W * 32, (OR_YZ_WARPS_SM / W > 0 ? OR_YZ_WARPS_SM / W : 1))
    yz_work_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv, YzScratch sc,
                   YzPrune prune) {
    extern __shared__ __align__(16) unsigned char yz_smem[];
    or_plane_t &P = *reinterpret_cast<or_plane_t *>(yz_smem);
    YzWarp *warps = reinterpret_cast<YzWarp *>(yz_smem + ((sizeof(or_plane_t) + 15) & ~size_t(15)));
    load_plane_smem(&P, gplane);
    __syncthreads();
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    YzWarp &S = warps[w];
    YzHit *garena = yz_garena(sc, blockIdx.x * W + w);
    PassEntryStore *Q = sc.qbuf + (long)((blockIdx.x * W + w) % sc.garena_warps) * sc.qcap;
    if (lane == 0) S.nsurv = 0ull;
    __syncwarp();
    const int nunits = min((int)sc.counters[0], sc.cap_units);
    for (;;) {
        int u = 0;
        if (lane == 0) u = (int)atomicAdd(&sc.counters[2], 1u);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= nunits) break;
        const YzUnit un = sc.units[u];
        if (un.heavy < 0) continue;
        const YzHeavy hv2 = sc.heavy[un.heavy];
        float *T = trk_rec(tv, hv2.e, hv2.slot, hv2.k);
        const int st3 = 3 + (hv2.slot & 1);
        YzEvent &E = S.ev;
        __syncwarp();  // every lane is done with the previous unit's views
        yz_event_planes(E, hv, hv2.e, st3);
        __syncwarp();
        const YzHit *base;
        if (hv2.img >= 0) base = yz_load_image(S, sc.img + hv2.img);
        else yz_build(S, E, T, P, st3, base, garena);
        yz_xhits(S, T, P);
        Stale *st = S.st;
        __syncwarp();  // every lane is done with the previous unit's states
#pragma unroll 1
        for (int k = 0; k < 4; ++k) st[k] = un.entry[k];
        __syncwarp();
        const long C2 = (long)S.np[0] * S.np[1];
        const float *osc = PRUNE ? yz_tracklet_scores(prune, hv2) : nullptr;
        const unsigned long long bk =
            yz_range_t<PRUNE>(S, E, base, (long)un.g0 * C2, (long)un.g1 * C2, st, P,
                              sc.tab + YZ_TAB_SETS * (st3 - 3), Q, sc.qcap, osc, prune.t_keep);
        __syncwarp();
        YzBest *dst = sc.best + u;
        if (hv2.nunits == 1) {  // the tracklet's only unit
            yz_finish(sc, un.heavy, hv2.c2, T, bk, S.b, S.nhx);
        } else if (bk == ~0ull) {
            if (lane == 0) dst->key = ~0ull;
        } else {
            const unsigned *src = reinterpret_cast<const unsigned *>(&S.b);
            unsigned *d = reinterpret_cast<unsigned *>(dst);
#pragma unroll 1
            for (int i = lane; i < (int)(sizeof(YzBest) / 4); i += 32) d[i] = src[i];
        }
        __syncwarp();
    }
    if (lane == 0 && sc.count_work) yz_flush_counts(sc, 0ull, 0ull, S.nsurv);
}


// Split path, first kernel: the first cut and the gates of every queued unit
// (no left/right walk, so it needs far fewer registers); what the survivor
// kernel needs of a unit goes, in order, to one contiguous piece of the pool.
template <int W, bool PRUNE>
__global__ void __launch_bounds__(W * 32, (OR_YZ_FIRST_WARPS_SM / W > 0 ? OR_YZ_FIRST_WARPS_SM / W : 1))
    yz_first_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv, YzScratch sc,
                    YzPrune prune) {
    extern __shared__ __align__(16) unsigned char yz_smem[];
    YzGate &G = *reinterpret_cast<YzGate *>(yz_smem);
    YzFirstWarp *warps = reinterpret_cast<YzFirstWarp *>(yz_smem + ((sizeof(YzGate) + 15) & ~size_t(15)));
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 6) {
        const int i = threadIdx.x;
        int stid = (i >> 1) + 1;
        const int det = c_hodoplanesx[stid][i & 1];
        if (det > 40) stid = 3;
        const float fudgefac = c_hodofudgefac[stid];
        float ymin = gplane->y1[det], ymax = gplane->y2[det];
        ymin -= (ymax - ymin) * fudgefac;
        ymax += (ymax - ymin) * fudgefac;
        G.hz[i] = gplane->z[det];
        G.ymin[i] = ymin;
        G.ymax[i] = ymax;
    } else if (threadIdx.x < 10) {
        const int q = threadIdx.x - 6;
        G.pz[q] = gplane->z[q == 0 ? DET_P1Y1 : q == 1 ? DET_P1Y2 : q == 2 ? DET_P2Y1 : DET_P2Y2];
    }
    __syncthreads();
    YzFirstWarp &S = warps[w];
    const int gw = blockIdx.x * W + w;
    if (gw >= sc.garena_warps) return;  // queues and arenas exist for garena_warps warps
    float4 *garena = reinterpret_cast<float4 *>(yz_garena(sc, gw));
    YzSurv *Q = reinterpret_cast<YzSurv *>(sc.qbuf + (long)gw * sc.qcap);
    const int qcap = sc.qcap * (int)(sizeof(PassEntryStore) / sizeof(YzSurv));
    unsigned long long *pool_ctr = reinterpret_cast<unsigned long long *>(sc.counters + 8);
    const int nunits = min((int)sc.counters[0], sc.cap_units);
    unsigned long long n_surv = 0ull;
    // The next unit is taken while the current one is worked on, and read
    // before that is done; with no more units than warps each warp has its
    // own (a unit taken ahead would wait while other warps are idle).
    const bool own = nunits <= (int)gridDim.x * W;
    int nxt = own ? w * (int)gridDim.x + (int)blockIdx.x : 0;
    if (!own && lane == 0) nxt = (int)atomicAdd(&sc.counters[2], 1u);
    int u = __shfl_sync(0xffffffffu, nxt, 0);
    int heavy = -1, r0 = 0, r1 = 0;
    auto read_unit = [&](int i) {
        if (i >= nunits) return;
        heavy = sc.units[i].heavy;
        r0 = sc.units[i].r0;
        r1 = sc.units[i].r1;
    };
    read_unit(u);
    while (u < nunits) {
        const int cu = u, cheavy = heavy, c0 = r0, c1 = r1;
        nxt = nunits;
        if (!own && lane == 0) nxt = (int)atomicAdd(&sc.counters[2], 1u);
        if (cheavy < 0) {
            u = __shfl_sync(0xffffffffu, nxt, 0);
            read_unit(u);
            continue;
        }
        const YzHeavy hv2 = sc.heavy[cheavy];
        const int st3 = 3 + (hv2.slot & 1);
        const YzTab *tab = sc.tab + YZ_TAB_SETS * (st3 - 3);
        int ns = -1, count = 0;  // -1: the unit runs on the combined path (survivor kernel)
        __syncwarp();            // every lane is done with the previous unit's state
        if (hv2.img < 0) {
            u = __shfl_sync(0xffffffffu, nxt, 0);
            read_unit(u);
        } else {
            const uint4 *img = sc.img + hv2.img;
            const YzImgHead &h = *reinterpret_cast<const YzImgHead *>(img);
            const int total = h.total;
            if (lane < 4) S.np[lane] = h.np[lane];
            if (lane < 8) S.woff[lane] = h.woff[lane];
            const unsigned hasx = yz_first_event(S, hv, hv2.e, G, gplane, h.x0, h.tx, h.ex0, h.etx);
            u = __shfl_sync(0xffffffffu, nxt, 0);
            read_unit(u);
            __syncwarp();
            // a station without a hodoscope hit in the x window closes the
            // gates for every combination
            const bool closed = !(hasx & 3u) || !(hasx & 12u) || !(hasx & 48u);
            if (closed && !sc.count_work) {
                ns = 0;
            } else if (!closed) {
                YzInner I;
                I.hits = img + YZ_IMG_HEAD_WORDS;
                const short2 *pair = reinterpret_cast<const short2 *>(I.hits + 2 * total);
                int most = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) most = max(most, S.np[q]);
                const bool small = most <= YZ_LIST_SMEM;
                const int cap = small ? YZ_LIST_SMEM : YZ_MAXPAIR;
                float4 *term = small ? &S.term[0][0] : garena;
                unsigned *info = small ? &S.info[0][0] : reinterpret_cast<unsigned *>(garena + 4 * YZ_MAXPAIR);
                int na[4];
                YzLast last;
                int first_two;
                const short2 *pq = pair;
                {
                    // the hits of all four lists' first pairs are on their way
                    // to L1 before the first list is made
                    short2 pp[4];
                    int at = 0;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        pp[q] = lane < S.np[q] ? pair[at + lane] : make_short2(-1, -1);
                        at += S.np[q];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (pp[q].x >= 0) prefetch_l1(I.hits + 2 * (S.woff[2 * q] + pp[q].x));
                        if (pp[q].y >= 0) prefetch_l1(I.hits + 2 * (S.woff[2 * q + 1] + pp[q].y));
                    }
                }
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    const int n = yz_first_list(S, q, pq, I.hits, term + q * cap, info + q * cap, last, first_two);
                    if (q == 0) {
                        na[0] = n;
                        I.pu = pq;
                        I.u = last;
                        I.first_two = first_two;
                    } else if (q == 1) {
                        na[1] = n;
                        I.pv = pq;
                        I.v = last;
                    } else if (q == 2) {
                        na[2] = n;
                    } else {
                        na[3] = n;
                    }
                    pq += S.np[q];
                }
                I.ou = S.woff[1];
                I.ov = S.woff[3];
                I.ova = S.woff[2];
                __syncwarp();
                auto second = [&](int q, int i) {
                    return (unsigned)(q == 0 ? I.ou + I.pu[i].y : I.ov + I.pv[i].y);
                };
                auto rel0 = [&](int q, int i) {
                    const short2 p = q == 0 ? I.pu[i] : I.pv[i];
                    const int oa = q == 0 ? S.woff[0] : I.ova, ob = q == 0 ? I.ou : I.ov;
                    const bool sec = p.x < 0 || (!yz_img_acc(I.hits, oa + p.x) && p.y >= 0);
                    return (unsigned)(sec ? ob + p.y : oa + p.x);
                };
                if (na[0] * na[1] == 0) {
                    ns = 0;
                } else {
                    const unsigned long long lasto = yz_lasto(S.np[0], S.np[1], I.u, I.v, second, rel0);
                    const float *osc = PRUNE ? yz_tracklet_scores(prune, hv2) : nullptr;
                    ns = yz_first_walk<PRUNE>(S, G, hasx, term, info, cap, na, I, lasto, c0, c1, st3 == 3, tab, Q, qcap,
                                              osc, prune.t_keep, &count);
                }
            }
        }
        __syncwarp();
        long long off = -1;
        if (lane == 0 && ns >= 0) {
            const unsigned long long o = ns ? atomicAdd(pool_ctr, (unsigned long long)ns) : 0ull;
            if (o + (unsigned long long)ns <= (unsigned long long)sc.pool_cap) off = (long long)o;
        }
        off = __shfl_sync(0xffffffffu, off, 0);
        if (off >= 0) {
            n_surv += (unsigned long long)count;
            const uint4 *src = reinterpret_cast<const uint4 *>(Q);
            uint4 *dst = reinterpret_cast<uint4 *>(sc.pool + off);
#pragma unroll 1
            for (int i = lane; i < ns; i += 32) dst[i] = src[i];
        }
        if (lane == 0) sc.useg[cu] = make_int2(off >= 0 ? (int)off : -1, off >= 0 ? ns : 0);
        __syncwarp();
    }
    if (lane == 0 && sc.count_work) yz_flush_counts(sc, 0ull, 0ull, n_surv);
}

// Split path, second kernel: per unit, the tracklet's windows from their image
// and then its survivors replayed in order with the sign carry (or the whole
// unit on the combined path when its survivors or its image did not fit);
// writes the unit's best.
#ifndef OR_YZ_SECOND_WARPS_SM
#define OR_YZ_SECOND_WARPS_SM 28
#endif
template <int W, bool PRUNE>
__global__ void __launch_bounds__(W * 32, (OR_YZ_SECOND_WARPS_SM / W > 0 ? OR_YZ_SECOND_WARPS_SM / W : 1))
    yz_second_kernel(const or_plane_t *__restrict__ gplane, or_hits_view_t hv, or_tracks_view_t tv, YzScratch sc,
                     YzPrune prune) {
    extern __shared__ __align__(16) unsigned char yz_smem[];
    or_plane_t &P = *reinterpret_cast<or_plane_t *>(yz_smem);
    YzWarp *warps = reinterpret_cast<YzWarp *>(yz_smem + ((sizeof(or_plane_t) + 15) & ~size_t(15)));
    load_plane_smem(&P, gplane);
    __syncthreads();
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    YzWarp &S = warps[w];
    const int gw = blockIdx.x * W + w;
    if (gw >= sc.garena_warps) return;
    YzHit *garena = yz_garena(sc, gw);
    PassEntryStore *Q = sc.qbuf + (long)gw * sc.qcap;
    if (lane == 0) S.nsurv = 0ull;
    __syncwarp();
    const int nunits = min((int)sc.counters[0], sc.cap_units);
    // with no more units than warps each warp has its own (taking one ahead,
    // as the first kernel does, is no gain here: 10,000 dimuon events 218 ->
    // 228 us)
    const bool own = nunits <= (int)gridDim.x * W;
    for (int mine = own ? w * (int)gridDim.x + (int)blockIdx.x : 0;; mine = nunits) {
        int u = mine;
        if (!own) {
            if (lane == 0) u = (int)atomicAdd(&sc.counters[3], 1u);
            u = __shfl_sync(0xffffffffu, u, 0);
        }
        if (u >= nunits) break;
        const YzUnit un = sc.units[u];
        if (un.heavy < 0) continue;
        const int2 seg = sc.useg[u];
        if (seg.x >= 0 && seg.y == 0) {  // no survivor: nothing to evaluate
            if (lane == 0) sc.best[u].key = ~0ull;
            continue;
        }
        const YzHeavy hv2 = sc.heavy[un.heavy];
        float *T = trk_rec(tv, hv2.e, hv2.slot, hv2.k);
        const int st3 = 3 + (hv2.slot & 1);
        YzEvent &E = S.ev;
        Stale *st = S.st;
        __syncwarp();
        if (seg.x < 0) yz_event_planes(E, hv, hv2.e, st3);  // the gates and the windows are evaluated here
        if (lane < 4) st[lane] = sc.units[u].entry[lane];
        __syncwarp();
        const YzHit *base;
        if (hv2.img >= 0) base = yz_load_image(S, sc.img + hv2.img);
        else yz_build(S, E, T, P, st3, base, garena);
        yz_xhits(S, T, P);
        const long C2 = (long)S.np[0] * S.np[1];
        const YzTab *tab = sc.tab + YZ_TAB_SETS * (st3 - 3);
        unsigned long long bk;
        if (seg.x < 0) {
            const float *osc = PRUNE ? yz_tracklet_scores(prune, hv2) : nullptr;
            bk = yz_range_ool<PRUNE>(S, E, base, (long)un.g0 * C2, (long)un.g1 * C2, st, P, tab, Q, sc.qcap, osc,
                                     prune.t_keep);
        } else {
            Phase2Carry cs;
#pragma unroll 1
            for (int i = 0; i < seg.y; i += 32) {
                yz_phase2<true>(S, E, base, (int)C2, P, sc.pool + seg.x + i, min(seg.y - i, 32), tab, cs);
                __syncwarp();
            }
            bk = cs.best;
        }
        __syncwarp();
        YzBest *dst = sc.best + u;
        if (hv2.nunits == 1) {  // the tracklet's only unit
            yz_finish(sc, un.heavy, hv2.c2, T, bk, S.b, S.nhx);
        } else if (bk == ~0ull) {
            if (lane == 0) dst->key = ~0ull;
        } else {
            const unsigned *src = reinterpret_cast<const unsigned *>(&S.b);
            unsigned *d = reinterpret_cast<unsigned *>(dst);
#pragma unroll 1
            for (int i = lane; i < (int)(sizeof(YzBest) / 4); i += 32) d[i] = src[i];
        }
        __syncwarp();
    }
    if (lane == 0 && sc.count_work) yz_flush_counts(sc, 0ull, 0ull, S.nsurv);
}


// Heavy tracklets of several units: the units' minimum key wins (those of
// one unit are written by the kernel that evaluates it).  A warp reads the
// unit counts of 32 tracklets at a time: few have more than one.  One warp
// per tracklet, whatever its units, took 1.18 ms of the 100,000-event batch.
__global__ void __launch_bounds__(128) yz_apply_kernel(or_tracks_view_t tv, YzScratch sc) {
    const int lane = threadIdx.x & 31;
    const int nheavy = min((int)sc.counters[1], sc.cap_heavy);
#pragma unroll 1
    for (int h0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; h0 < nheavy; h0 += gridDim.x * blockDim.x) {
        const int mine = h0 + lane < nheavy ? sc.heavy[h0 + lane].nunits : 0;
        for (unsigned m = __ballot_sync(0xffffffffu, mine > 1); m; m &= m - 1) {
            const int h = h0 + __ffs(m) - 1;
            const YzHeavy hv2 = sc.heavy[h];
            if ((long)hv2.unit0 + hv2.nunits > sc.cap_units) continue;
            unsigned long long best = ~0ull;
            int bu = -1;
#pragma unroll 1
            for (int u = lane; u < hv2.nunits; u += 32) {
                const unsigned long long k = sc.best[hv2.unit0 + u].key;
                if (k < best) {
                    best = k;
                    bu = hv2.unit0 + u;
                }
            }
#pragma unroll 1
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ok = __shfl_xor_sync(0xffffffffu, best, o);
                const int ou = __shfl_xor_sync(0xffffffffu, bu, o);
                if (ok < best) {
                    best = ok;
                    bu = ou;
                }
            }
            if (best == ~0ull) continue;
            float *T = trk_rec(tv, hv2.e, hv2.slot, hv2.k);
            const int nhx = min((int)T[OR_TRK_NHITS], 4);
            __syncwarp();  // every lane has read the count that yz_finish replaces
            yz_finish(sc, h, hv2.c2, T, best, sc.best[bu], nhx);
        }
    }
}

// Planning units (event, chunk of `chunk` slots) that hold tracklets, in
// event order within a block: those of many tracklets from the list's front
// (counters[6] of them), the others from its back (counters[7]), so that the
// long ones do not start last (planning pass of 10,000 uneven events 614 ->
// 586 us, with the combination scorer 1,860 -> 1,660 us).  The planning
// warps take them one by one from a counter, so units without tracklets (all
// of a rejected event's) would cost an atomic each: 0.4 ms for 20,000
// rejected events at one slot per unit.
constexpr int YZ_LIST_THREADS = 1024;
__device__ __forceinline__ void yz_list_units(const or_tracks_view_t &tv, const uint8_t *__restrict__ toomany,
                                              int n_events, int chunk, const YzScratch &sc, int block) {
    __shared__ int warp_n[YZ_LIST_THREADS / 32];
    __shared__ unsigned base[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long e = (long)block * (YZ_LIST_THREADS / 32) + w;
    const int ntr = e < n_events && !toomany[e] ? min((int)tv.ntracks[e * OR_NSLOTS + lane], OR_SLOTCAP) : 0;
    const bool have = ntr > 0;
    int sum = ntr;  // of the lane's chunk
    for (int o = 1; o < chunk; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const unsigned hm = __ballot_sync(0xffffffffu, have);
    // the first lane of each chunk with tracklets stands for it
    const int c0 = lane / chunk * chunk;
    const unsigned cm = (chunk == 32 ? ~0u : (1u << chunk) - 1u) << c0;
    const bool take = lane == c0 && (hm & cm) != 0u;
    const bool large = sum >= 2 + 5 * chunk / 4;
    const unsigned lm = __ballot_sync(0xffffffffu, take && large), sm = __ballot_sync(0xffffffffu, take && !large);
    if (lane == 0) warp_n[w] = __popc(lm) | __popc(sm) << 16;
    __syncthreads();
    if (w == 0) {
        const int v = warp_n[lane];
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        warp_n[lane] = incl - v;
        const int all = __shfl_sync(0xffffffffu, incl, 31);
        const unsigned mine = lane ? (unsigned)all >> 16 : (unsigned)all & 0xffffu;
        if (lane < 2) base[lane] = mine ? atomicAdd(&sc.counters[6 + lane], mine) : 0u;
    }
    __syncthreads();
    if (!take) return;
    const unsigned unit = (unsigned)(e * (OR_NSLOTS / chunk) + lane / chunk);
    if (large) sc.list[base[0] + (warp_n[w] & 0xffff) + __popc(lm & lanemask_lt())] = unit;
    else sc.list[(long)n_events * (OR_NSLOTS / chunk) - 1 - (base[1] + (warp_n[w] >> 16) + __popc(sm & lanemask_lt()))] = unit;
}

// The 2 x 81 plane-set entries of the first y fit (see YzTab): for every
// set, Fit2's normal matrix accumulated over the set's planes in the order
// u3 u3' v3 v3' u2 u2' v2 v2' with the plane's weight and z, then
// matinv_2x2 and the errors as in Fit2::solve, and the first cut's bounds.
// The blocks after the first list the planning units.
__global__ void __launch_bounds__(YZ_LIST_THREADS)
    yz_tab_kernel(const or_plane_t *__restrict__ gplane, YzTab *__restrict__ tab, or_tracks_view_t tv,
                  const uint8_t *__restrict__ toomany, int n_events, int chunk, YzScratch sc) {
    if (blockIdx.x > 0) {
        yz_list_units(tv, toomany, n_events, chunk, sc, (int)blockIdx.x - 1);
        return;
    }
    const int t = threadIdx.x;
    if (t >= 2 * YZ_TAB_SETS) return;
    const or_plane_t &P = *gplane;
    const int st3 = 3 + t / YZ_TAB_SETS;
    const int i = t % YZ_TAB_SETS;
    const int g[4] = {i / 27 + 1, (i / 9) % 3 + 1, (i / 3) % 3 + 1, i % 3 + 1};  // u3 v3 u2 v2
    const int det[8] = {det_u3(st3), det_u3(st3) - 1, det_v3(st3), det_v3(st3) - 1, DET_U2, DET_UP2, DET_V2, DET_VP2};
    Fit2 f;
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
        if (!((g[k >> 1] >> (k & 1)) & 1)) continue;
        const int d = det[k];
        const float w = P.resolution[d] * fabsf(P.deltapy[d] / P.deltapx[d]);  // calculate_y_uvhit's err_y, H:98
        f.add(0.f, P.z[d], w);
    }
    const float A[4] = {f.A0, f.A1, f.A2, f.A3};
    float Ai[4];
    matinv_2x2(A, Ai);
    YzTab e;
    e.ai0 = Ai[0];
    e.ai1 = Ai[1];
    e.ai2 = Ai[2];
    e.ai3 = Ai[3];
    e.ey0 = sqrtf(fabsf(Ai[0]));
    e.ety = sqrtf(fabsf(Ai[3]));
    e.thr_y0 = Y0_MAX + 2 * e.ey0;
    e.thr_ty = TY_MAX + 2 * e.ety;
    tab[t] = e;
}

// Events the combination scorer leaves to the plain method: a queued
// tracklet all of whose live outer iterations score below t_keep, the best
// of them at or above t_unc -- the scorer would drop the whole tracklet
// without a clear margin.  Such an event is evaluated without pruning.
__global__ void __launch_bounds__(128) yz_unc_kernel(YzScratch sc, YzPrune prune) {
    const int lane = threadIdx.x & 31;
    const int nheavy = min((int)sc.counters[1], sc.cap_heavy);
    const long ncap = min((long)*prune.orows, prune.cap_orows);
#pragma unroll 1
    for (int h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; h < nheavy; h += (gridDim.x * blockDim.x) >> 5) {
        const YzHeavy hv2 = sc.heavy[h];
        if (hv2.nunits <= 0 || hv2.orow0 < 0 || (long)hv2.orow0 + hv2.nrows > ncap) continue;
        float mx = -1.f;
#pragma unroll 1
        for (int r = lane; r < hv2.nrows; r += 32) mx = fmaxf(mx, prune.oscore[hv2.orow0 + r]);
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0 && mx < prune.t_keep && mx >= prune.t_unc) prune.unc[hv2.e] = 1;
    }
}

// Units of pruned tracklets with no kept row in their rank range are dropped
// before the first cut (their best key is "none"); everything they would
// have done is skipped anyway, including the window rebuild.
__global__ void __launch_bounds__(128) yz_kill_units_kernel(YzScratch sc, YzPrune prune) {
    const int lane = threadIdx.x & 31;
    const int nunits = min((int)sc.counters[0], sc.cap_units);
    const long ncap = min((long)*prune.orows, prune.cap_orows);
#pragma unroll 1
    for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < nunits; u += (gridDim.x * blockDim.x) >> 5) {
        const YzUnit un = sc.units[u];
        if (un.heavy < 0) continue;
        const YzHeavy hv2 = sc.heavy[un.heavy];
        if (hv2.orow0 < 0 || (long)hv2.orow0 + hv2.nrows > ncap || prune.unc[hv2.e]) continue;
        bool kept = false;
#pragma unroll 1
        for (int r = un.r0 + lane; r < un.r1 && !kept; r += 32) kept = prune.oscore[hv2.orow0 + r] >= prune.t_keep;
        if (!__any_sync(0xffffffffu, kept) && lane == 0) {
            sc.units[u].heavy = -1;
            sc.best[u].key = ~0ull;
        }
    }
}

// Labels of the scorer's rows after the plain chain: 1 for the row of the
// outer iteration that holds its tracklet's best combination when the
// tracklet ended as a global track (stationID 6 after global tracking), else
// 0.  The scratch still holds the last YZ call's heavy tracklets.
__global__ void __launch_bounds__(128) yz_outer_labels_kernel(YzScratch sc, or_tracks_view_t tv,
                                                              const uint8_t *__restrict__ toomany,
                                                              const int32_t *__restrict__ og, const uint32_t *orows,
                                                              long cap, uint8_t *__restrict__ labels) {
    const int lane = threadIdx.x & 31;
    const int nheavy = min((int)sc.counters[1], sc.cap_heavy);
    const long ncap = min((long)*orows, cap);
#pragma unroll 1
    for (int h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; h < nheavy; h += (gridDim.x * blockDim.x) >> 5) {
        const YzHeavy hv2 = sc.heavy[h];
        if (hv2.nunits <= 0 || hv2.orow0 < 0 || (long)hv2.orow0 + hv2.nrows > ncap) continue;
        const float *T = trk_rec(tv, hv2.e, hv2.slot, hv2.k);
        const bool global = !toomany[hv2.e] && T[OR_TRK_STID] == 6.f;
#pragma unroll 1
        for (int r = lane; r < hv2.nrows; r += 32)
            labels[hv2.orow0 + r] = (global && og[hv2.orow0 + r] == hv2.best_g) ? 1 : 0;
    }
}

size_t yz_first_smem_bytes(int warps) {
    return ((sizeof(YzGate) + 15) & ~size_t(15)) + sizeof(YzFirstWarp) * (size_t)warps;
}
size_t yz_smem_bytes(int warps) {
    return ((sizeof(or_plane_t) + 15) & ~size_t(15)) + sizeof(YzWarp) * (size_t)warps;
}

// Scratch the YZ stage needs: queue of units, per-unit best records, heavy
// tracklets, per-warp overflow arenas.
static long long yz_pool_cap(int qcap, int cap_units) {
    return (OR_YZ_SPLIT && qcap == YZ_QCAP_CTX) ? YZ_POOL_PER_UNIT * cap_units : 0;
}
static long long yz_img_cap(int qcap, int cap_units) {
    return (OR_YZ_SPLIT && qcap == YZ_QCAP_CTX) ? YZ_IMG_PER_UNIT * cap_units : 0;
}

size_t yz_scratch_bytes_q(int cap_units, int cap_heavy, int garena_warps, int qcap) {
    size_t b = 256 + YZ_TAB_BYTES + (sizeof(YzUnit) + sizeof(YzBest)) * (size_t)cap_units +
               sizeof(YzHeavy) * (size_t)cap_heavy;
    b = (b + 255) & ~size_t(255);
    b += sizeof(YzHit) * YZ_GARENA_HITS * (size_t)garena_warps;
    b += sizeof(PassEntryStore) * (size_t)qcap * (size_t)garena_warps;
    if (yz_pool_cap(qcap, cap_units) > 0) {
        b = (b + 255) & ~size_t(255);
        b += sizeof(int2) * (size_t)cap_units;
        b = (b + 255) & ~size_t(255);
        b += sizeof(YzSurv) * (size_t)yz_pool_cap(qcap, cap_units);
    }
    if (yz_img_cap(qcap, cap_units) > 0) {
        b = (b + 255) & ~size_t(255);
        b += 16 * (size_t)yz_img_cap(qcap, cap_units);
    }
    return b;
}

// the static (no-allocation) scratch: survivor queues of YZ_QCAP_MIN entries
size_t yz_scratch_bytes(int cap_units, int cap_heavy, int garena_warps) {
    return yz_scratch_bytes_q(cap_units, cap_heavy, garena_warps, YZ_QCAP_MIN);
}

// a context's scratch
size_t yz_scratch_bytes_ctx(int cap_units, int cap_heavy, int garena_warps) {
    return yz_scratch_bytes_q(cap_units, cap_heavy, garena_warps, YZ_QCAP_CTX);
}

// the work counters of the last YZ call on `scratch` (synchronous copy)
cudaError_t yz_read_counts(const void *scratch, long long out[3]) {
    unsigned long long c[32];
    const cudaError_t e = cudaMemcpy(c, scratch, sizeof(c), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    out[0] = (long long)c[YZ_CTR_FITTED / 2];
    out[1] = (long long)c[YZ_CTR_HITSUM / 2];
    out[2] = (long long)c[YZ_CTR_SURVIVORS / 2];
    return cudaSuccess;
}

// The pointers into a YZ scratch area (the layout yz_scratch_bytes_q sizes).
static YzScratch yz_scratch_layout(void *scratch, int cap_units, int cap_heavy, int garena_warps, int qcap,
                                   long long pool_limit) {
    char *p = static_cast<char *>(scratch);
    YzScratch sc;
    sc.counters = reinterpret_cast<unsigned int *>(p);
    p += 256;
    sc.tab = reinterpret_cast<YzTab *>(p);
    p += YZ_TAB_BYTES;
    sc.units = reinterpret_cast<YzUnit *>(p);
    p += sizeof(YzUnit) * (size_t)cap_units;
    sc.best = reinterpret_cast<YzBest *>(p);
    p += sizeof(YzBest) * (size_t)cap_units;
    sc.heavy = reinterpret_cast<YzHeavy *>(p);
    p += sizeof(YzHeavy) * (size_t)cap_heavy;
    p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255));
    sc.garena = reinterpret_cast<YzHit *>(p);
    p += sizeof(YzHit) * YZ_GARENA_HITS * (size_t)garena_warps;
    sc.qbuf = reinterpret_cast<PassEntryStore *>(p);
    p += sizeof(PassEntryStore) * (size_t)qcap * (size_t)garena_warps;
    sc.pool_cap = yz_pool_cap(qcap, cap_units);
    if (pool_limit >= 0 && pool_limit < sc.pool_cap) sc.pool_cap = pool_limit;  // the rest of the pool goes unused
    sc.useg = nullptr;
    sc.pool = nullptr;
    if (sc.pool_cap > 0) {
        p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255));
        sc.useg = reinterpret_cast<int2 *>(p);
        p += sizeof(int2) * (size_t)cap_units;
        p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255));
        sc.pool = reinterpret_cast<YzSurv *>(p);
    }
    // the images follow the whole pool (pool_limit only narrows its use)
    p = reinterpret_cast<char *>(scratch) + yz_scratch_bytes_q(cap_units, cap_heavy, garena_warps, qcap) -
        16 * (size_t)yz_img_cap(qcap, cap_units);
    sc.img = yz_img_cap(qcap, cap_units) > 0 ? reinterpret_cast<uint4 *>(p) : nullptr;
    sc.img_cap = yz_img_cap(qcap, cap_units);
    sc.cap_units = cap_units;
    sc.cap_heavy = cap_heavy;
    sc.garena_warps = garena_warps;
    sc.qcap = qcap;
    sc.count_work = 0;
    sc.list = nullptr;
    return sc;
}

cudaError_t launch_mlp_score(const or_mlp_t *, const float *, long, const int32_t *, float *, uint32_t *, cudaStream_t,
                             int);

template <int W>
static cudaError_t launch_yz_impl(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv,
                                  const uint8_t *toomany, int n_events, uint32_t *errw, void *scratch, int cap_units,
                                  int cap_heavy, int garena_warps, cudaStream_t stream, int sm_count, YzPrune prune,
                                  int qcap, long long pool_limit, int count_work, bool cleared) {
    if (n_events <= 0) return cudaSuccess;
    const size_t smem = yz_smem_bytes(W);
    cudaError_t err;
    if (prune.ofeat) {
        if ((err = cudaMemsetAsync(prune.orows, 0, sizeof(uint32_t), stream))) return err;
        if (prune.unc && (err = cudaMemsetAsync(prune.unc, 0, (size_t)n_events, stream))) return err;
    } else {
        prune.model = nullptr;  // no rows: nothing to score or prune
    }
    if ((err = smem_attr_once((const void *)yz_plan_kernel<W>, (int)smem)))
        return err;
    YzScratch sc = yz_scratch_layout(scratch, cap_units, cap_heavy, garena_warps, qcap, pool_limit);
    YzTab *tab = const_cast<YzTab *>(sc.tab);
    sc.count_work = count_work;
    if (!cleared && (err = cudaMemsetAsync(sc.counters, 0, 256, stream))) return err;
    // One slot per planning unit: a heavy event's tracklets spread over 32
    // warps (a single uneven event's planning pass 442 -> 59 us, 333 of them
    // 619 -> 107 us, 100,000 12.6 -> 11.8 ms).  With the combination scorer
    // the unit stays at 8 slots: which light tracklets it evaluates itself,
    // and so which ones have score rows, depends on the unit's budget.
    const int chunk = prune.ofeat ? YZ_PLAN_CHUNK_SCORED : YZ_PLAN_CHUNK;
    const long nplan = (long)n_events * (OR_NSLOTS / chunk);
    // the list stands in the best records' area: it is read by the planning
    // pass alone, and nothing writes a best record before that is done
    const bool listed = nplan <= (long)(sizeof(YzBest) / 4) * cap_units;
    sc.list = listed ? reinterpret_cast<unsigned *>(sc.best) : nullptr;
    const unsigned list_blocks = listed ? (unsigned)(((long)n_events * 32 + YZ_LIST_THREADS - 1) / YZ_LIST_THREADS) : 0u;
    yz_tab_kernel<<<1 + list_blocks, YZ_LIST_THREADS, 0, stream>>>(d_plane, tab, tv, toomany, n_events, chunk, sc);
    if ((err = cudaGetLastError())) return err;
    const long blocks = garena_warps / W;
    const long blocks_plan = min((nplan + W - 1) / W, blocks);
    yz_plan_kernel<W><<<(unsigned)blocks_plan, W * 32, smem, stream>>>(d_plane, hv, tv, toomany, n_events, chunk, sc,
                                                                       errw, prune);
    if ((err = cudaGetLastError())) return err;
    if (prune.model) {
        // score the rows on the tensor cores (the row count stays on the
        // device), then the uncertain events
        if ((err = launch_mlp_score(prune.model, prune.ofeat, prune.cap_orows,
                                    reinterpret_cast<const int32_t *>(prune.orows), prune.oscore, errw, stream,
                                    sm_count)))
            return err;
        yz_unc_kernel<<<(unsigned)(sm_count * 4), 128, 0, stream>>>(sc, prune);
        if ((err = cudaGetLastError())) return err;
        yz_kill_units_kernel<<<(unsigned)(sm_count * 8), 128, 0, stream>>>(sc, prune);
        if ((err = cudaGetLastError())) return err;
    }
    if (sc.pool_cap > 0) {
        const size_t smem1 = yz_first_smem_bytes(W);
        const long res1 = (long)sm_count * (OR_YZ_FIRST_WARPS_SM / W > 0 ? OR_YZ_FIRST_WARPS_SM / W : 1);
        const long res = (long)sm_count * (OR_YZ_SECOND_WARPS_SM / W > 0 ? OR_YZ_SECOND_WARPS_SM / W : 1);
        if (prune.model) {
            if ((err = smem_attr_once((const void *)yz_first_kernel<W, true>, (int)smem1))) return err;
            if ((err = smem_attr_once((const void *)yz_second_kernel<W, true>, (int)smem))) return err;
            yz_first_kernel<W, true><<<(unsigned)min(blocks, res1), W * 32, smem1, stream>>>(d_plane, hv, tv, sc, prune);
            if ((err = cudaGetLastError())) return err;
            yz_second_kernel<W, true><<<(unsigned)min(blocks, res), W * 32, smem, stream>>>(d_plane, hv, tv, sc, prune);
        } else {
            if ((err = smem_attr_once((const void *)yz_first_kernel<W, false>, (int)smem1))) return err;
            if ((err = smem_attr_once((const void *)yz_second_kernel<W, false>, (int)smem))) return err;
            yz_first_kernel<W, false><<<(unsigned)min(blocks, res1), W * 32, smem1, stream>>>(d_plane, hv, tv, sc, prune);
            if ((err = cudaGetLastError())) return err;
            yz_second_kernel<W, false><<<(unsigned)min(blocks, res), W * 32, smem, stream>>>(d_plane, hv, tv, sc,
                                                                                          prune);
        }
    } else if (prune.model) {
        if ((err = smem_attr_once((const void *)yz_work_kernel<W, true>, (int)smem))) return err;
        yz_work_kernel<W, true><<<(unsigned)blocks, W * 32, smem, stream>>>(d_plane, hv, tv, sc, prune);
    } else {
        if ((err = smem_attr_once((const void *)yz_work_kernel<W, false>, (int)smem))) return err;
        yz_work_kernel<W, false><<<(unsigned)blocks, W * 32, smem, stream>>>(d_plane, hv, tv, sc, prune);
    }
    if ((err = cudaGetLastError())) return err;
    yz_apply_kernel<<<(unsigned)(sm_count * 4), 128, 0, stream>>>(tv, sc);
    return cudaGetLastError();
}

static cudaError_t launch_yz_w(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv,
                               const uint8_t *toomany, int n_events, uint32_t *errw, void *scratch, int cap_units,
                               int cap_heavy, int garena_warps, cudaStream_t stream, int sm_count, YzPrune prune,
                               int warps, int qcap, long long pool_limit, int count_work, bool cleared = false) {
#define OR_YZ_LAUNCH(W)                                                                                         \
    launch_yz_impl<W>(d_plane, hv, tv, toomany, n_events, errw, scratch, cap_units, cap_heavy, garena_warps, stream, \
                      sm_count, prune, qcap, pool_limit, count_work, cleared)
    switch (warps) {
    case 1: return OR_YZ_LAUNCH(1);
    case 2: return OR_YZ_LAUNCH(2);
    case 8: return OR_YZ_LAUNCH(8);
    case 16: return OR_YZ_LAUNCH(16);
    default: return OR_YZ_LAUNCH(4);
    }
#undef OR_YZ_LAUNCH
}

cudaError_t launch_yz(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv, const uint8_t *toomany,
                      int n_events, uint32_t *errw, void *scratch, int cap_units, int cap_heavy, int garena_warps,
                      cudaStream_t stream, int sm_count) {
    return launch_yz_w(d_plane, hv, tv, toomany, n_events, errw, scratch, cap_units, cap_heavy, garena_warps, stream,
                       sm_count, YzPrune{}, 4, YZ_QCAP_MIN, -1, 0);
}

// with `warps` events (work units) per CTA: 1, 2, 4, 8 or 16
cudaError_t launch_yz_tuned(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv,
                            const uint8_t *toomany, int n_events, uint32_t *errw, void *scratch, int cap_units,
                            int cap_heavy, int garena_warps, cudaStream_t stream, int sm_count, int warps,
                            long long pool_limit, int count_work, bool cleared) {
    return launch_yz_w(d_plane, hv, tv, toomany, n_events, errw, scratch, cap_units, cap_heavy, garena_warps, stream,
                       sm_count, YzPrune{}, warps, YZ_QCAP_CTX, pool_limit, count_work, cleared);
}

// YZ with the scorer's keep flags: pruned tracklets are left as tracklets no
// combination extends; kept ones get the plain result
cudaError_t launch_yz_pruned(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv,
                             const uint8_t *toomany, int n_events, uint32_t *errw, void *scratch, int cap_units,
                             int cap_heavy, int garena_warps, cudaStream_t stream, int sm_count,
                             const int32_t *row_off, const uint8_t *keep, long max_rows, int warps,
                             long long pool_limit, int count_work) {
    YzPrune pr{};
    pr.row_off = row_off;
    pr.keep = keep;
    pr.max_rows = max_rows;
    return launch_yz_w(d_plane, hv, tv, toomany, n_events, errw, scratch, cap_units, cap_heavy, garena_warps, stream,
                       sm_count, pr, warps, YZ_QCAP_CTX, pool_limit, count_work);
}

// YZ with the combination scorer: rows of features for every live outer
// iteration of each queued tracklet, scored by `prune.model` (nullptr: rows
// only), outer iterations below t_keep skipped
cudaError_t launch_yz_scored(const or_plane_t *d_plane, or_hits_view_t hv, or_tracks_view_t tv,
                             const uint8_t *toomany, int n_events, uint32_t *errw, void *scratch, int cap_units,
                             int cap_heavy, int garena_warps, cudaStream_t stream, int sm_count, const or_mlp_t *model,
                             float t_keep, float t_unc, float *feat, int32_t *og, float *score, uint32_t *rows,
                             uint8_t *unc, long max_rows, int warps, long long pool_limit, int count_work) {
    YzPrune pr{};
    pr.ofeat = feat;
    pr.og = og;
    pr.oscore = score;
    pr.orows = rows;
    pr.unc = unc;
    pr.model = model;
    pr.cap_orows = max_rows;
    pr.t_keep = t_keep;
    pr.t_unc = t_unc;
    return launch_yz_w(d_plane, hv, tv, toomany, n_events, errw, scratch, cap_units, cap_heavy, garena_warps, stream,
                       sm_count, pr, warps, YZ_QCAP_CTX, pool_limit, count_work);
}

// labels of the last scored YZ call's rows (see yz_outer_labels_kernel)
cudaError_t launch_yz_outer_labels(void *scratch, int cap_units, int cap_heavy, int garena_warps, or_tracks_view_t tv,
                                   const uint8_t *toomany, const int32_t *og, const uint32_t *rows, long max_rows,
                                   uint8_t *labels, cudaStream_t stream, int sm_count) {
    const YzScratch sc = yz_scratch_layout(scratch, cap_units, cap_heavy, garena_warps, YZ_QCAP_CTX, -1);
    yz_outer_labels_kernel<<<(unsigned)(sm_count * 4), 128, 0, stream>>>(sc, tv, toomany, og, rows, max_rows, labels);
    return cudaGetLastError();
}

}  // namespace orgpu
