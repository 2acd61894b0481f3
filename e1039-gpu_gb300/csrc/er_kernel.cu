// er_kernel.cu -- event reducer (hit filtering, declustering, per-channel
// de-duplication, in-place compaction, station-multiplicity reject).
//
// Replaces gkernel_eR<<<N,8>>> (OnlineReconstruction/reconstruction_kernels
// .cuh:8-172) and event_reduction() (reconstruction_helper.cuh:168-361).
//
// Layout on the GPU: one warp per event.  The warp stages the
// occupied part of each plane slot (5*n floats, rounded up to 16 bytes --
// slot capacities are multiples of 16 bytes, so the round-up stays inside the
// slot) into shared memory with 1-D TMA bulk copies completing on an
// mbarrier; planes are taken in batches that fit the warp's buffer (a warp
// prefix sum over the planes' sizes), each lane issuing the copies of its
// planes.  The hits of a batch are then one index space, 32 at a time,
// whatever planes they belong to:
//   - the reference's cluster state after an in-time hit is "closed" when
//     the hit lies more than one channel from the one before and the run of
//     such hits has an odd length (a hit that closes a cluster does not start
//     the next one, so in a run every second hit opens one), else "open":
//     the run's length is a ballot and a carry;
//   - a hit that closes a cluster, or ends its plane inside one, lists the
//     cluster, whose first hit is the last cluster start before it (a ballot
//     and a carry); the 2-hit and the n-hit rule then take a lane per listed
//     cluster, in floats (pairs of floats where the reference rounds double
//     products);
//   - the first survivor of a channel: where every plane's channels ascend
//     (a sorted event) the hits of a channel follow one another, and it is the
//     first kept one of its run; else the lane that sets the channel's bit in
//     the plane's map, or the first of the lanes of a chunk that share it.
// Survivors are written back with the new SoA stride into the same slot,
// consecutive lanes to consecutive words; a plane that keeps all its hits is
// not written.  Bytes beyond the survivors are left as they were, as the
// reference leaves them.
//
// Bound: instruction issue, and shared-memory latency behind it (the SM's
// schedulers issue in 60 % of the cycles; more warps per SM changed nothing).
// For 100,000 uneven events, 20,000 of high occupancy, 333 uneven and 10,000
// dimuon ones, in us:
//   a lane per plane running the state machine          2,820  972  245   99
//   flat hits, each end walking back to its cluster's
//   start, channels by __match_any_sync                 1,600  564  144   64
//   clusters listed, runs of one channel by ballot      1,050  355   80   50
#include "or_device.cuh"

namespace orgpu {

// Staging buffer per warp: the smallest that holds a full chamber plane.  More
// batches per event, but more warps per SM (with the second form above 100,000
// uneven events took 1.60 ms; 1.88 at 6 KB, 2.01 at 8 KB).
constexpr int ER_BUF_FLOATS = 1024;
constexpr int ER_MAX_STAGED_HITS = ER_BUF_FLOATS / 5 + 8;
constexpr int ER_FIRST_WORDS = (ER_MAX_STAGED_HITS + 31) / 32;
constexpr int ER_NPLANES = 48, ER_NCHAMBERS = 24;
static_assert(ER_BUF_FLOATS >= 5 * OR_MAXHITS_CHAM + 3, "a full plane fits the buffer");
constexpr uint32_t ER_WAIT_LIMIT = 1u << 26;        // bounded mbarrier wait, unless or_set_wait_limit says otherwise
constexpr uint32_t ER_DRAIN_LIMIT = 1u << 28;       // ... and the wait for copies in flight after it gave up

// the 48 planes the reducer touches: the 24 chambers of the E1039 set
// (reconstruction_constants.h:60), 16 hodoscopes, 8 prop tubes (K:25-57)
__device__ __constant__ unsigned char c_er_det[ER_NPLANES] = {
    1,  2,  3,  4,  5,  6,  13, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30,
    31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 41, 42, 43, 44, 45, 46, 47, 48, 49, 50, 51, 52, 53, 54};

struct __align__(16) ErWarp {
    float buf[ER_BUF_FLOATS];
    uint64_t bar;
    int16_t n[ER_NPLANES];
    int16_t kept[ER_NPLANES];
    int16_t at[ER_NPLANES];     // survivors of the batch before each plane
    int16_t soff[ER_NPLANES];   // start of each plane's image in buf
    int16_t hoff[ER_NPLANES];   // hits of the batch before each plane
    uint16_t list[ER_MAX_STAGED_HITS];  // chamber hits in time, then the survivors: index in the batch
    uint8_t plane[ER_MAX_STAGED_HITS];  // plane of each hit of the batch
    uint8_t keep[ER_MAX_STAGED_HITS];
    uint8_t chan[ER_MAX_STAGED_HITS];   // its channel, 255 outside 0..201
    uint8_t cl[ER_MAX_STAGED_HITS / 2][2];  // clusters of two or more: first and last list entry
    uint32_t seen[ER_NPLANES][7];       // channels 0..201 of each plane's survivors
    uint32_t first[ER_FIRST_WORDS];     // bit per hit of the batch: the first of its plane
    float *slot[ER_NPLANES];
    uint8_t occupied[ER_NPLANES];       // the batch's planes with hits
};
static_assert(ER_MAX_STAGED_HITS <= 256, "a list entry fits a byte");
static_assert(7 * 32 >= 202, "channel bits");

struct PlaneRef {
    float *slot;
    uint32_t *count;
    int cap;
};

__device__ __forceinline__ PlaneRef er_plane(const or_hits_view_t &hv, long e, int det) {
    PlaneRef r;
    if (det <= OR_NCHAM) {
        r.slot = hv.hits_cham + e * OR_EVT_CHAM_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_CHAM * (det - 1);
        r.count = hv.nhits_cham + e * OR_NCHAM + det - 1;
        r.cap = OR_MAXHITS_CHAM;
    } else if (det <= OR_NCHAM + OR_NHODO) {
        const int k = det - OR_NCHAM - 1;
        r.slot = hv.hits_hodo + e * OR_EVT_HODO_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_HODO * k;
        r.count = hv.nhits_hodo + e * OR_NHODO + k;
        r.cap = OR_MAXHITS_HODO;
    } else {
        const int k = det - OR_NCHAM - OR_NHODO - 1;
        r.slot = hv.hits_prop + e * OR_EVT_PROP_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_PROP * k;
        r.count = hv.nhits_prop + e * OR_NPROP + k;
        r.cap = OR_MAXHITS_PROP;
    }
    return r;
}

// (float)(c * x); the double product's rounding of a float is its second, so
// pairs of floats decide it nearly always (an FP64 instruction takes 64 cycles)
__device__ __noinline__ float er_scale_double(double c, float x) { return (float)(c * (double)x); }
__device__ __forceinline__ float er_scale(double c, FF cf, float x) {
    const FF v = ff_mul(cf, x);
    if (x == 0.f) return x;
    return ff_sure(v) ? v.h : er_scale_double(c, x);
}

// The rules for a cluster of `cls` >= 2 in-time hits list[s..t] of one plane
// (reference H:267-318); h = the plane's image, n its hits, first the batch
// index of its first hit.
static __device__ __forceinline__ void er_cluster(ErWarp &S, int s, int t, const float *h, int n, int first, int det) {
    auto pos = [&](int i) { return h[n + i]; };
    auto tdc = [&](int i) { return h[2 * n + i]; };
    auto drift = [&](int i) { return h[4 * n + i]; };
    const int cls = t - s + 1;
    const int a = S.list[s] - first, b = S.list[t] - first;
    if (cls == 2) {  // H:267-295
        constexpr FF half = ff_const(0.9 * 0.5), ninths = ff_const(4.0 / 9.0);
        const float w_max = er_scale(0.9 * 0.5, half, pos(b) - pos(a));
        const float w_min = er_scale(4.0 / 9.0, ninths, w_max);
        if ((drift(a) > w_max && drift(b) > w_min) || (drift(a) > w_min && drift(b) > w_max)) {
            S.keep[first + (drift(a) > drift(b) ? a : b)] = 0;
        } else {
            const float dt = tdc(a) - tdc(b);
            if (((dt >= 0.f && dt < 8.f) || (dt <= 0.f && dt > -8.f)) &&
                (det >= 19 && det <= 24)) {
                S.keep[first + a] = 0;
                S.keep[first + b] = 0;
            }
        }
    } else if (cls >= 3) {  // H:297-318
        float dt_mean = 0.0f;
        int prev = a;
        for (int k = s + 1; k <= t; ++k) {
            const int m = S.list[k] - first;
            const float d = tdc(m) - tdc(prev);
            dt_mean += (d > 0.f ? d : (tdc(prev) - tdc(m)));
            prev = m;
        }
        dt_mean = dt_mean / (float)(cls - 1);
        const bool all = dt_mean < 10.f;
        for (int k = all ? s : s + 1; k <= t; ++k) S.keep[S.list[k]] = 0;
    }
}

// event_reduction() (reconstruction_helper.cuh:168-361) on the staged planes
// [p0, p1) of `hits` hits: S.kept, S.at and, per plane in order, the
// survivors' batch indices in S.list; returns their number.  The after-pulse branch (H:204-230) never changes a
// flag: uniqueID_curr is reset every hit.
static __device__ __forceinline__ int er_reduce(ErWarp &S, int p0, int p1, int hits) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    for (int i = lane; i < ER_FIRST_WORDS; i += 32) S.first[i] = 0u;
    __syncwarp();
    int nocc = 0;
    for (int q0 = p0; q0 < p1; q0 += 32) {
        const int p = q0 + lane;
        const bool occ = p < p1 && S.n[p] > 0;
        const unsigned m = __ballot_sync(0xffffffffu, occ);
        if (p < p1) S.kept[p] = 0;
        if (occ) {
            S.occupied[nocc + __popc(m & lt)] = (uint8_t)p;
            atomicOr(&S.first[S.hoff[p] >> 5], 1u << (S.hoff[p] & 31));
        }
        nocc += __popc(m);
    }
    __syncwarp();
    // in-time hits; those of chambers are listed.  `up`: the channels of
    // every plane are in ascending order, as a sorted event's are
    int nlist = 0, started = 0;
    bool up = true;
    float before = 0.f;  // the last chunk's last channel
#pragma unroll 1
    for (int b0 = 0; b0 < hits; b0 += 32) {
        const int f = b0 + lane;
        bool cham = false;
        float x = 0.f;
        if (f < hits) {
            // its plane: as many occupied planes start at or before it
            const int p = S.occupied[started + __popc(S.first[b0 >> 5] & (lt | (1u << lane))) - 1];
            const int n = S.n[p], i = f - S.hoff[p];
            const bool intime = (((int)S.buf[S.soff[p] + 3 * n + i]) & 2) != 0;  // H:198
            x = S.buf[S.soff[p] + i];
            const int c = (short)x;
            S.plane[f] = (uint8_t)p;
            S.chan[f] = (uint8_t)(c >= 0 && c < 202 ? c : 255);
            S.keep[f] = intime;
            cham = intime && p < ER_NCHAMBERS;
        }
        float y = __shfl_up_sync(0xffffffffu, x, 1);
        if (lane == 0) y = before;
        before = __shfl_sync(0xffffffffu, x, 31);
        up &= f >= hits || (x > -32768.f && x < 32768.f && (((S.first[b0 >> 5] >> lane) & 1u) || y <= x));
        started += __popc(S.first[b0 >> 5]);
        const unsigned m = __ballot_sync(0xffffffffu, cham);
        if (cham) S.list[nlist + __popc(m & lt)] = (uint16_t)f;
        nlist += __popc(m);
    }
    __syncwarp();
    // cluster state after each listed hit (H:241-258), and the clusters of two
    // or more, each at the hit that ends it: a cluster starts at its plane's
    // first listed hit or after a hit that closed one
    int run = 0;  // hits far from the one before, up to the last chunk's end
    int begin = 0, ncl = 0;
    unsigned after = 0u;  // the last chunk's last hit closed a cluster
#pragma unroll 1
    for (int b0 = 0; b0 < nlist; b0 += 32) {
        const int k = b0 + lane;
        bool first = true, far = false, last = false;
        if (k < nlist) {
            const int f = S.list[k], p = S.plane[f];
            last = f - S.hoff[p] == S.n[p] - 1;
            const int g = k > 0 ? S.list[k - 1] : f;
            if (k > 0 && S.plane[g] == p) {
                const float *h = S.buf + S.soff[p] - S.hoff[p];
                first = false;
                far = fabsf(h[f] - h[g]) > 1;
            }
        }
        const unsigned le = lt | (1u << lane);
        const unsigned near = ~__ballot_sync(0xffffffffu, far);
        const int l = last_lane(near & le);
        const int r = l >= 0 ? lane - l : run + lane + 1;
        const bool closes = far && (r & 1);
        const unsigned closed = __ballot_sync(0xffffffffu, closes);
        const unsigned starts = __ballot_sync(0xffffffffu, first && k < nlist) | (closed << 1) | after;
        // [s, t] ends here: before the hit that closes it, or with the plane
        const int m = last_lane(starts & (closes ? lt : le));
        const int s = m >= 0 ? b0 + m : begin;
        const int t = closes ? k - 1 : !first && !far && last ? k : -1;
        const unsigned cm = __ballot_sync(0xffffffffu, t > s);
        if (t > s) {
            uint8_t *c = S.cl[ncl + __popc(cm & lt)];
            c[0] = (uint8_t)s;
            c[1] = (uint8_t)t;
        }
        ncl += __popc(cm);
        const int mm = last_lane(starts);
        if (mm >= 0) begin = b0 + mm;
        after = closed >> 31;
        run = __shfl_sync(0xffffffffu, r, 31);
    }
    __syncwarp();
#pragma unroll 1
    for (int k = lane; k < ncl; k += 32) {
        const int s = S.cl[k][0], t = S.cl[k][1], p = S.plane[S.list[s]];
        er_cluster(S, s, t, S.buf + S.soff[p], S.n[p], S.hoff[p], c_er_det[p]);
    }
    __syncwarp();
    // H:334-349, first survivor per channel wins
    int ns = 0;
    up = __all_sync(0xffffffffu, up);
    if (!up) {
        for (int i = p0 * 7 + lane; i < p1 * 7; i += 32) S.seen[0][i] = 0u;
        __syncwarp();
    }
    int chan = -1;      // the last chunk's last channel, and
    bool taken = false;  // whether it has a survivor
#pragma unroll 1
    for (int b0 = 0; b0 < hits; b0 += 32) {
        const int f = b0 + lane;
        int p = 0, c = 255;
        bool k = false, first = true;
        if (f < hits) {
            p = S.plane[f];
            k = S.keep[f];
            c = S.chan[f];
            first = (S.first[b0 >> 5] >> lane) & 1u;
        }
        if (up) {
            // hits of one channel follow one another
            int d = __shfl_up_sync(0xffffffffu, c, 1);
            if (lane == 0) d = chan;
            const unsigned starts = __ballot_sync(0xffffffffu, first || c != d);
            const unsigned all = __ballot_sync(0xffffffffu, k);
            const int l = last_lane(starts & (lt | (1u << lane)));
            const unsigned same = lt & (l >= 0 ? ~0u << l : ~0u);  // its channel's hits before it
            bool had = (all & same) != 0u || (l < 0 && taken);
            if (c != 255) k = k && !had;
            chan = __shfl_sync(0xffffffffu, c, 31);
            taken = __shfl_sync(0xffffffffu, had || ((all >> lane) & 1u), 31);
        } else {
            if (!k) c = 255;
            // a lane that finds its channel's bit set is a later hit of the
            // channel, or shares it with lanes of this chunk: of those the
            // first survives, unless the bit was set before
            if (c != 255) k = !((atomicOr(&S.seen[p][c >> 5], 1u << (c & 31)) >> (c & 31)) & 1u);
            if (__any_sync(0xffffffffu, c != 255 && !k)) {
                const unsigned peers = __match_any_sync(0xffffffffu, c != 255 ? p * 256 + c : -1 - lane);
                const unsigned set = __ballot_sync(0xffffffffu, k) & peers;
                if (c != 255) k = set != 0u && (peers & lt) == 0u;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, k);
        const int j = ns + __popc(m & lt);
        if (k) S.list[j] = (uint16_t)f;
        if (f < hits && first) S.at[p] = (int16_t)j;
        ns += __popc(m);
        __syncwarp();
    }
    for (int o = lane; o < nocc; o += 32) {
        const int p = S.occupied[o];
        S.kept[p] = (int16_t)((o + 1 < nocc ? S.at[S.occupied[o + 1]] : ns) - S.at[p]);
    }
    __syncwarp();
    return ns;
}

template <int W>
__global__ void __launch_bounds__(W * 32) er_kernel(or_hits_view_t hv, uint8_t *__restrict__ toomany, int n_events,
                                                    uint32_t *__restrict__ errw, ChainClear clear,
                                                    uint32_t wait_limit) {
    extern __shared__ __align__(16) unsigned char er_smem[];
    ErWarp *sm = reinterpret_cast<ErWarp *>(er_smem);
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    ErWarp &S = sm[w];
    if (lane == 0) mbar_init(&S.bar, 1);
    __syncwarp();
    uint32_t phase = 0;
    if (blockIdx.x == 0 && w == 0)
        for (int i = lane; i < 64; i += 32)
#pragma unroll
            for (int b = 0; b < 2; ++b)
                if (clear.counters[b]) clear.counters[b][i] = 0u;

    for (long e = (long)blockIdx.x * W + w; e < n_events; e += (long)gridDim.x * W) {
        for (int p = lane; p < ER_NPLANES; p += 32) {
            const PlaneRef r = er_plane(hv, e, c_er_det[p]);
            const int n = (int)*r.count;
            S.n[p] = (int16_t)(n < r.cap ? n : r.cap);
            S.slot[p] = r.slot;
        }
        __syncwarp();
        int p0 = 0;
        while (p0 < ER_NPLANES) {
            // batch [p0, p1): planes whose staged images fit the buffer
            int p1 = p0, off = 0, hits = 0;
            // 32 planes at a time: prefix sums of the staged sizes and hit
            // counts over the lanes; the planes that fit form a prefix
            for (;;) {
                const int p = p1 + lane;
                const int n_l = p < ER_NPLANES ? S.n[p] : 0;
                const int sz_l = p < ER_NPLANES ? ((5 * n_l + 3) & ~3) : ER_BUF_FLOATS + 1;
                int csz = sz_l, cn = n_l;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int a = __shfl_up_sync(0xffffffffu, csz, d);
                    const int b = __shfl_up_sync(0xffffffffu, cn, d);
                    if (lane >= d) {
                        csz += a;
                        cn += b;
                    }
                }
                const bool fit = off + csz <= ER_BUF_FLOATS;
                const int nfit = __popc(__ballot_sync(0xffffffffu, fit));
                if (fit) {
                    S.soff[p] = (int16_t)(off + csz - sz_l);
                    S.hoff[p] = (int16_t)(hits + cn - n_l);
                }
                if (nfit == 0) break;
                off += __shfl_sync(0xffffffffu, csz, nfit - 1);
                hits += __shfl_sync(0xffffffffu, cn, nfit - 1);
                p1 += nfit;
                if (nfit < 32 || p1 >= ER_NPLANES) break;
            }
            __syncwarp();
            if (off > 0) {
                // lane 0 announces the batch's bytes before any copy is
                // issued; then every lane issues the copies of its planes
                if (lane == 0) mbar_arrive_expect_tx(&S.bar, (uint32_t)off * 4u);
                __syncwarp();
                fence_proxy_async_smem();  // buffer was read by the generic proxy
                for (int p = p0 + lane; p < p1; p += 32) {
                    const int sz = (5 * S.n[p] + 3) & ~3;
                    if (sz == 0) continue;
                    tma_load_1d(S.buf + S.soff[p], S.slot[p], (uint32_t)sz * 4u, &S.bar);
                }
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&S.bar, phase, wait_limit))) {
                    // the wait gave up: raise the error word, then wait (again
                    // bounded) for this batch's copies still in flight, so that
                    // the warp leaves no bulk copy writing into shared memory
                    if (lane == 0) atomicOr(errw, ERRW_TMA_TIMEOUT);
                    mbar_wait_bounded(&S.bar, phase, ER_DRAIN_LIMIT);
                    __syncwarp();
                    return;
                }
                phase ^= 1u;
            }
            const int ns = er_reduce(S, p0, p1, hits);
            for (int p = p0 + lane; p < p1; p += 32) *er_plane(hv, e, c_er_det[p]).count = (uint32_t)S.kept[p];
            // write back the planes that lost hits
#pragma unroll 1
            for (int j = lane; j < ns; j += 32) {
                const int f = S.list[j], p = S.plane[f], n = S.n[p], k = S.kept[p];
                if (k == n) continue;
                const float *src = S.buf + S.soff[p] - S.hoff[p] + f;
                float *dst = S.slot[p] + j - S.at[p];
#pragma unroll
                for (int q = 0; q < 5; ++q) dst[q * k] = src[q * n];
            }
            __syncwarp();
            p0 = p1;
        }
        // K:128-139: station sums of the reduced chamber counts, planes 0-5,
        // 6-11, 12-17 and 18-23 of the list
        {
            const int lim = lane < 6 ? MAXD0 : lane < 12 ? MAXD2 : MAXD3;
            int m = lane < ER_NCHAMBERS ? S.kept[lane] : 0;
            const int st = lane / 6;
            int sum = 0;
#pragma unroll
            for (int k = 0; k < 6; ++k) sum += __shfl_sync(0xffffffffu, m, min(31, st * 6 + k));
            const bool over = __any_sync(0xffffffffu, lane < ER_NCHAMBERS && sum > lim);
            if (lane == 0) toomany[e] = (uint8_t)over;
        }
        __syncwarp();
    }
}

// Host launcher.
template <int W>
static cudaError_t er_launch(or_hits_view_t hv, uint8_t *toomany, int n_events, uint32_t *errw, cudaStream_t stream,
                             int sm_count, ChainClear clear, uint32_t wait_limit) {
    const size_t smem = sizeof(ErWarp) * W;
    cudaError_t e = smem_attr_once((const void *)er_kernel<W>, (int)smem);
    if (e != cudaSuccess) return e;
    long blocks = (n_events + W - 1) / W;
    const long cap = (long)sm_count * (48 / W > 0 ? 48 / W : 1);  // up to 48 resident warps per SM
    if (blocks > cap) blocks = cap;
    er_kernel<W><<<(unsigned)blocks, W * 32, smem, stream>>>(hv, toomany, n_events, errw, clear, wait_limit);
    return cudaGetLastError();
}

// Self-test of the bounded wait: one warp waits on an mbarrier that nothing
// arrives at and no bulk copy targets, `polls` polls at most.  The wait runs
// out, the kernel raises ERRW_TMA_TIMEOUT as the reducer does, invalidates the
// barrier and returns; the context stays usable.
__global__ void __launch_bounds__(32) wait_selftest_kernel(uint32_t *__restrict__ errw, uint32_t polls) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncwarp();
    const bool done = __all_sync(0xffffffffu, mbar_wait_bounded(&bar, 0u, polls));
    if (!done && threadIdx.x == 0) atomicOr(errw, ERRW_TMA_TIMEOUT);
    __syncwarp();
    if (threadIdx.x == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar)) : "memory");
}

cudaError_t launch_wait_selftest(uint32_t *errw, uint32_t polls, cudaStream_t stream) {
    wait_selftest_kernel<<<1, 32, 0, stream>>>(errw, polls);
    return cudaGetLastError();
}

// Host launcher; `warps` = events per CTA (1, 2, 4, 8 or 16), `polls` = the
// wait's limit (< 0: ER_WAIT_LIMIT).
cudaError_t launch_event_reduce(or_hits_view_t hv, uint8_t *toomany, int n_events, uint32_t *errw,
                                cudaStream_t stream, int sm_count, int warps, ChainClear clear, long long polls) {
    if (n_events <= 0) return cudaSuccess;
    const uint32_t limit = polls < 0 || polls > ER_WAIT_LIMIT ? ER_WAIT_LIMIT : (uint32_t)polls;
    switch (warps) {
    case 1: return er_launch<1>(hv, toomany, n_events, errw, stream, sm_count, clear, limit);
    case 2: return er_launch<2>(hv, toomany, n_events, errw, stream, sm_count, clear, limit);
    case 8: return er_launch<8>(hv, toomany, n_events, errw, stream, sm_count, clear, limit);
    case 16: return er_launch<16>(hv, toomany, n_events, errw, stream, sm_count, clear, limit);
    default: return er_launch<4>(hv, toomany, n_events, errw, stream, sm_count, clear, limit);
    }
}

}  // namespace orgpu
