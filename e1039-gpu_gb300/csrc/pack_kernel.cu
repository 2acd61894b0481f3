// pack_kernel.cu -- device-side hit packer: compact hit records to the
// reference hit layout.
//
// Does on the GPU what the reference host loop does per event
// (OnlineReconstruction/online_reconstruction.cu:589-636): for every plane
// write the hit count and the five SoA fields [chan | pos | tdc | flag |
// drift] with stride = count, pos = (float)wire_position[det][elem].
// Records of an event must be sorted by (det, elem, tdc); hits beyond a
// plane's slot capacity are dropped (the reference host would write past the
// slot).  An event whose records are out of that order raises ERRW_INPUT
// (or_stream_sync reports it as an argument error); its slots are then
// undefined but every write stays inside them.  Records whose det is outside
// 1..54 (they sort first or last) are skipped.  One warp per event: the planes'
// runs are where the det changes from one record to the next (512 records'
// planes in flight), then the field writes (128 records in flight).
//
// Bound: the pieces of 100 to 600 bytes, off sector boundaries, that an
// event's planes are written in (3.5 of 6.9 TB/s; staging the records in
// shared memory by bulk copies, so that no read waits, changed nothing: 519
// us).  A histogram by shared-memory atomics (all lanes on one counter where
// records are sorted), a scan by one lane and one record in flight per lane
// took 685 us for 100,000 uneven events and, with the R-T spline, 166 us for
// 16,001; plane runs from neighbours and 128 records in flight 600 and 143
// us; whole-record loads, 512 planes in flight and a block per eight events
// 513 and 122 us (20,000 events of high occupancy 259 -> 236 us).
//
// With an R-T table the drift field is computed from the tdc as the
// reference host does while packing (online_reconstruction.cu:387-396); the
// same conversion also runs in place on hits packed elsewhere (rt_apply).
#include "or_device.cuh"

namespace orgpu {

constexpr int PK_WARPS = 8;
constexpr int PK_DETS = 16;  // chunks of 32 records whose plane is in flight per warp
constexpr int PK_AHEAD = 4;  // ... and whose fields are
constexpr int PK_BLOCKS = 4; // per SM: 64 registers

// Drift distance of a hit on plane det from the R-T calibration, or `drift`
// unchanged when the plane has no profile (hodoscopes never have one).
// Evaluation follows the spline's piece convention: piece k covers
// (t[k], t[k+1]]; x <= t[0] uses piece 0 and x >= t[n-1] piece n-2.  The
// cubic is evaluated in double in nested form and rounded to float once, as
// the reference's float drift_distance receives the double result (:332, :395).
static __device__ __forceinline__ float rt_drift(const or_rt_table_t *__restrict__ rt, int det, float tdc,
                                                 float drift) {
    const int n = rt->nknots[det];
    if (n <= 0) return drift;
    if (tdc < rt->tmin[det]) return (float)((double)rt->cellwidth[det] * 0.5);
    if (tdc > rt->tmax[det]) return 0.f;
    const double *t = rt->t[det];
    const double x = (double)tdc;
    int k = 0;
    if (n > 1) {
        if (x >= t[n - 1]) {
            k = n - 2;
        } else if (x > t[0]) {
            int lo = 0, hi = n - 1;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (x > t[mid]) lo = mid;
                else hi = mid;
            }
            k = lo;
        }
    }
    const double dx = x - t[k];
    const double v = rt->r[det][k] + dx * (rt->b[det][k] + dx * (rt->c[det][k] + dx * rt->d[det][k]));
    return (float)v;
}

static __device__ __forceinline__ bool rt_plane(int det) {
    return (det >= 1 && det <= OR_NCHAM) || (det > OR_NCHAM + OR_NHODO && det < OR_NDET);
}

// One record; `AL`: the records are 16-byte aligned, one load each
template <bool AL>
static __device__ __forceinline__ or_hit_record_t pk_record(const or_hit_record_t *R) {
    if (!AL) return *R;
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(R));
    or_hit_record_t h;
    h.det = (int16_t)(v.x & 0xffffu);
    h.elem = (int16_t)(v.x >> 16);
    h.tdc = __uint_as_float(v.y);
    h.drift = __uint_as_float(v.z);
    h.flag = (int32_t)v.w;
    return h;
}

template <bool RT, bool AL>
__global__ void __launch_bounds__(PK_WARPS * 32, PK_BLOCKS)
    pack_kernel(const or_hit_record_t *__restrict__ rec, const int64_t *__restrict__ off, int n_events,
                const float *__restrict__ wire_pos_f, const or_rt_table_t *__restrict__ rt, or_hits_view_t hv,
                uint32_t *__restrict__ errw) {
    // first record of each plane, and the one after its last
    __shared__ int first[PK_WARPS][64];
    __shared__ int past[PK_WARPS][64];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    for (long e = (long)blockIdx.x * PK_WARPS + w; e < n_events; e += (long)gridDim.x * PK_WARPS) {
        const int64_t r0 = off[e], r1 = off[e + 1];
        const int nrec = (int)(r1 - r0);
        const or_hit_record_t *R = rec + r0;
        first[w][lane] = past[w][lane] = 0;
        first[w][lane + 32] = past[w][lane + 32] = 0;
        __syncwarp();
        // Records are sorted by det: a plane's run starts where det changes.
        // Records with det out of range sort first or last and are skipped.
        int carry = -0x10000;  // det of the record before the chunk
#pragma unroll 1
        for (int b0 = 0; b0 < nrec; b0 += 32 * PK_DETS) {
            int d[PK_DETS];
#pragma unroll
            for (int i = 0; i < PK_DETS; ++i) {
                const int r = b0 + 32 * i + lane;
                d[i] = r < nrec ? (int)R[r].det : 0x10000;
            }
#pragma unroll
            for (int i = 0; i < PK_DETS; ++i) {
                const int r = b0 + 32 * i + lane;
                int prev = __shfl_up_sync(0xffffffffu, d[i], 1);
                if (lane == 0) prev = carry;
                carry = __shfl_sync(0xffffffffu, d[i], 31);
                if (d[i] != prev) {
                    if (d[i] >= 1 && d[i] < OR_NDET) first[w][d[i]] = r;
                    if (prev >= 1 && prev < OR_NDET) past[w][prev] = r;
                }
            }
        }
        if (lane == 0 && carry >= 1 && carry < OR_NDET) past[w][carry] = nrec;
        __syncwarp();
        // counts (capped) for all 54 planes; `past` is the count from here on
        for (int d = 1 + lane; d < OR_NDET; d += 32) {
            const int cap = d <= OR_NCHAM ? OR_MAXHITS_CHAM : d <= OR_NCHAM + OR_NHODO ? OR_MAXHITS_HODO : OR_MAXHITS_PROP;
            const int n = max(0, min(past[w][d] - first[w][d], cap));
            past[w][d] = n;
            if (d <= OR_NCHAM) hv.nhits_cham[e * OR_NCHAM + d - 1] = (uint32_t)n;
            else if (d <= OR_NCHAM + OR_NHODO) hv.nhits_hodo[e * OR_NHODO + d - OR_NCHAM - 1] = (uint32_t)n;
            else hv.nhits_prop[e * OR_NPROP + d - OR_NCHAM - OR_NHODO - 1] = (uint32_t)n;
        }
        __syncwarp();
        bool unsorted = false;
        int cd = -0x10000, ce = 0;  // the record before the chunk: det, elem, tdc
        float ct = 0.f;
#pragma unroll 1
        for (int b0 = 0; b0 < nrec; b0 += 32 * PK_AHEAD) {
            or_hit_record_t h[PK_AHEAD];
            float pos[PK_AHEAD];
#pragma unroll
            for (int i = 0; i < PK_AHEAD; ++i) {
                const int r = b0 + 32 * i + lane;
                h[i].det = (int16_t)0x7FFF;
                h[i].elem = 0;
                if (r < nrec) h[i] = pk_record<AL>(R + r);
            }
#pragma unroll
            for (int i = 0; i < PK_AHEAD; ++i) {
                const int d = h[i].det, el = h[i].elem;
                const bool in = d >= 1 && d < OR_NDET && el >= 0 && el < OR_WIREPOS_STRIDE;
                pos[i] = in ? __ldg(wire_pos_f + d * OR_WIREPOS_STRIDE + el) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < PK_AHEAD; ++i) {
                const int r = b0 + 32 * i + lane;
                const int d = h[i].det, el = h[i].elem;
                const float tdc = h[i].tdc;
                int pd = __shfl_up_sync(0xffffffffu, d, 1), pe = __shfl_up_sync(0xffffffffu, el, 1);
                float pt = __shfl_up_sync(0xffffffffu, tdc, 1);
                if (lane == 0) {
                    pd = cd;
                    pe = ce;
                    pt = ct;
                }
                cd = __shfl_sync(0xffffffffu, d, 31);
                ce = __shfl_sync(0xffffffffu, el, 31);
                ct = __shfl_sync(0xffffffffu, tdc, 31);
                if (r >= nrec) continue;
                unsorted |= d < pd || (d == pd && (el < pe || (el == pe && tdc < pt)));
                if (d < 1 || d >= OR_NDET) continue;
                const int k = r - first[w][d], n = past[w][d];
                if (k < 0 || k >= n) continue;  // beyond the slot, or out of order
                float *slot;
                if (d <= OR_NCHAM)
                    slot = hv.hits_cham + e * OR_EVT_CHAM_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_CHAM * (d - 1);
                else if (d <= OR_NCHAM + OR_NHODO)
                    slot = hv.hits_hodo + e * OR_EVT_HODO_FLOATS +
                           (long)OR_NHITSPARAM * OR_MAXHITS_HODO * (d - OR_NCHAM - 1);
                else
                    slot = hv.hits_prop + e * OR_EVT_PROP_FLOATS +
                           (long)OR_NHITSPARAM * OR_MAXHITS_PROP * (d - OR_NCHAM - OR_NHODO - 1);
                slot[k] = (float)el;
                slot[n + k] = pos[i];
                slot[2 * n + k] = tdc;
                slot[3 * n + k] = (float)h[i].flag;
                slot[4 * n + k] = (RT && rt_plane(d)) ? rt_drift(rt, d, tdc, h[i].drift) : h[i].drift;
            }
        }
        if (__any_sync(0xffffffffu, unsorted) && lane == 0) atomicOr(errw, ERRW_INPUT);
        __syncwarp();
    }
}

// In-place R-T conversion on the reference layout: one warp per event, the
// chamber and prop-tube planes in turn, lanes over a plane's hits.
__global__ void __launch_bounds__(PK_WARPS * 32)
    rt_apply_kernel(const or_rt_table_t *__restrict__ rt, or_hits_view_t hv, int n_events) {
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    for (long e = (long)blockIdx.x * PK_WARPS + w; e < n_events; e += (long)gridDim.x * PK_WARPS) {
        for (int p = 0; p < OR_NCHAM + OR_NPROP; ++p) {
            const bool cham = p < OR_NCHAM;
            const int d = cham ? 1 + p : OR_NCHAM + OR_NHODO + 1 + (p - OR_NCHAM);
            if (rt->nknots[d] <= 0) continue;
            float *slot;
            int n;
            if (cham) {
                n = min((int)hv.nhits_cham[e * OR_NCHAM + p], OR_MAXHITS_CHAM);
                slot = hv.hits_cham + e * OR_EVT_CHAM_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_CHAM * p;
            } else {
                n = min((int)hv.nhits_prop[e * OR_NPROP + p - OR_NCHAM], OR_MAXHITS_PROP);
                slot = hv.hits_prop + e * OR_EVT_PROP_FLOATS + (long)OR_NHITSPARAM * OR_MAXHITS_PROP * (p - OR_NCHAM);
            }
            for (int k = lane; k < n; k += 32) slot[4 * n + k] = rt_drift(rt, d, slot[2 * n + k], slot[4 * n + k]);
        }
    }
}

// Blocks beyond the resident ones even out events of different size (100,000
// uneven events: 8 blocks to an SM 582 us, 32: 542, one event per warp: 513).
static long pack_blocks(int n_events, int sm_count) {
    long blocks = (n_events + PK_WARPS - 1) / PK_WARPS;
    const long cap = (long)sm_count * 512;
    return blocks > cap ? cap : blocks;
}

cudaError_t launch_pack(const or_hit_record_t *rec, const int64_t *off, int n_events, const float *wire_pos_f,
                        const or_rt_table_t *rt, or_hits_view_t hv, uint32_t *errw, cudaStream_t stream,
                        int sm_count) {
    if (n_events <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)pack_blocks(n_events, sm_count);
    // records of an aligned table are read whole; those of any other (a record
    // is 16 bytes of 4-byte alignment) field by field (20,000 events of high
    // occupancy: 236 and 248 us)
    const bool al = (reinterpret_cast<uintptr_t>(rec) & 15u) == 0;
    auto *kernel = rt ? (al ? pack_kernel<true, true> : pack_kernel<true, false>)
                      : (al ? pack_kernel<false, true> : pack_kernel<false, false>);
    kernel<<<blocks, PK_WARPS * 32, 0, stream>>>(rec, off, n_events, wire_pos_f, rt, hv, errw);
    return cudaGetLastError();
}

cudaError_t launch_rt_apply(const or_rt_table_t *rt, or_hits_view_t hv, int n_events, cudaStream_t stream,
                            int sm_count) {
    if (n_events <= 0) return cudaSuccess;
    rt_apply_kernel<<<(unsigned)pack_blocks(n_events, sm_count), PK_WARPS * 32, 0, stream>>>(rt, hv, n_events);
    return cudaGetLastError();
}

}  // namespace orgpu
