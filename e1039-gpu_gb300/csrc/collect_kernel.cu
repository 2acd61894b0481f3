// collect_kernel.cu -- gather the final tracks of a batch into one dense
// buffer for the device-to-host copy.
//
// The reference copies whole collections back and walks them on the host to
// fill its output tree (OnlineReconstruction/online_reconstruction.cu
// :1023-1224, OROutput.h:25-102); a 10000-event track collection is 3 GB.
// Here the tracks with stationID == `stid` (6 = global tracks) are written as
// OR_COLLECT_STRIDE-float rows [event, slot*16+position, 148-float record],
// so only the tracks cross PCIe/C2C.  A cluster of blocks takes 256 events, a
// warp one or two of them: lane = slot, so an event's 32 counts are one
// 64-byte read and its stationIDs are read 32 slots at a time; scans over the
// warps of a block and the blocks of a cluster order the rows, one atomicAdd
// per cluster reserves them.  Within a cluster rows are in (event, slot,
// position) order; the order across clusters is not fixed; every row carries
// its event and slot.
//
// Bound: DRAM latency on small batches (three dependent reads), the reads of
// one 32-byte sector per track record on large ones.  One thread per event
// walking its slots in turn, and copying its rows alone, took 73 us for a
// single uneven event, 162 us for 10,000 one-dimuon events and 659 us for
// 100,000 uneven ones; a block per 256 events, eight to a warp, 15, 33 and
// 255 us, with 28 us for 256 dimuon events on its one SM; this takes 16 us
// for 10,000 dimuon events, 205 us for 100,000 uneven ones and 8 us for 256.
#include <cooperative_groups.h>

#include <algorithm>

#include "or_device.cuh"

namespace cg = cooperative_groups;

namespace orgpu {

constexpr int CO_THREADS = 1024;
constexpr int CO_WARPS = CO_THREADS / 32;
constexpr int CO_EVENTS = 256;  // whose rows are in order: a cluster's

// P events per warp, a cluster of CO_EVENTS / CO_WARPS / P blocks.
template <int P>
__global__ void __launch_bounds__(CO_THREADS)
    collect_kernel(or_tracks_view_t tv, const uint8_t *__restrict__ toomany, int n_events, float stid,
                   float *__restrict__ out, long long capacity, unsigned long long *__restrict__ cursor) {
    __shared__ unsigned long long base;
    __shared__ int block_tot;
    __shared__ int warp_tot[CO_WARPS];
    // tracks to gather: event in the warp * 512 + slot * 16 + position
    __shared__ uint16_t list[CO_WARPS][OR_TRKMAX];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long e0 = ((long)blockIdx.x * CO_WARPS + w) * P;
    int n[P];
    unsigned mask[P];  // the lane's slot: positions to gather
    int most = 0;
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const long e = e0 + i;
        mask[i] = 0u;
        n[i] = 0;
        if (e < n_events && !toomany[e]) n[i] = min((int)tv.ntracks[e * OR_NSLOTS + lane], OR_SLOTCAP);
        most = max(most, n[i]);
    }
    most = __reduce_max_sync(0xffffffffu, most);
#pragma unroll 1
    for (int k0 = 0; k0 < most; k0 += 4) {  // 4 P reads in flight per lane
        float v[P][4];
#pragma unroll
        for (int i = 0; i < P; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                v[i][k] = k0 + k < n[i] ? __ldg(trk_rec(tv, e0 + i, lane, k0 + k) + OR_TRK_STID) : 0.f;
#pragma unroll
        for (int i = 0; i < P; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k0 + k < n[i] && v[i][k] == stid) mask[i] |= 1u << (k0 + k);
    }
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < P; ++i) cnt += __popc(mask[i]);
    const int tot = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) warp_tot[w] = tot;
    __syncthreads();
    if (w == 0) {  // exclusive scan of the warps' counts
        const int v = warp_tot[lane];
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        warp_tot[lane] = incl - v;
        if (lane == 31) block_tot = incl;
    }
    // the blocks of a cluster reserve their rows together: the first one gives
    // each block its first row
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (cluster.block_rank() == 0 && w == 0) {
        const int nb = (int)cluster.num_blocks();
        const int v = lane < nb ? *cluster.map_shared_rank(&block_tot, lane) : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        const int all = __shfl_sync(0xffffffffu, incl, 31);
        unsigned long long b = 0ull;
        // a single cluster's count is the batch's
        if (lane == 0 && n_events <= CO_EVENTS) *cursor = (unsigned long long)all;
        else if (lane == 0 && all) b = atomicAdd(cursor, (unsigned long long)all);
        b = __shfl_sync(0xffffffffu, b, 0);
        if (lane < nb) *cluster.map_shared_rank(&base, lane) = b + (unsigned)(incl - v);
    }
    cluster.sync();
    if (tot == 0) return;
    long long row = (long long)base + warp_tot[w];
    // the warp's events go through the list together, as many as fit
    int i = 0;
    while (i < P) {
        int filled = 0;
        for (; i < P; ++i) {
            unsigned m = 0u;
#pragma unroll
            for (int k = 0; k < P; ++k)
                if (k == i) m = mask[k];
            const int c = __popc(m);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            const int rows = __shfl_sync(0xffffffffu, incl, 31);
            if (filled + rows > OR_TRKMAX) break;
            int at = filled + incl - c;
            for (; m; m &= m - 1) list[w][at++] = (uint16_t)(i * OR_TRKMAX + lane * OR_SLOTCAP + __ffs(m) - 1);
            filled += rows;
        }
        __syncwarp();
        const int nf = (int)min((long long)filled, max(capacity - row, 0ll)) * OR_COLLECT_STRIDE;
        const float *rec = trk_rec(tv, e0, 0, 0);
        float *dst = out + row * OR_COLLECT_STRIDE;
#pragma unroll 8
        for (int q = lane; q < nf; q += 32) {
            const int r = q / OR_COLLECT_STRIDE, f = q - r * OR_COLLECT_STRIDE;
            const int c = list[w][r];
            const int sk = c % OR_TRKMAX;
            dst[q] = f == 0 ? (float)(e0 + c / OR_TRKMAX) : (f == 1 ? (float)sk : __ldg(rec + (long)c * OR_NTRKPARAM + f - 2));
        }
        row += filled;
        __syncwarp();
    }
}

cudaError_t launch_collect(or_tracks_view_t tv, const uint8_t *toomany, int n_events, float stid, float *out,
                           long long capacity, unsigned long long *cursor, cudaStream_t stream, int sm_count) {
    if (n_events <= 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (n_events > CO_EVENTS && (e = cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), stream)) != cudaSuccess)
        return e;
    const long groups = ((long)n_events + CO_EVENTS - 1) / CO_EVENTS;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(CO_THREADS);
    cfg.stream = stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    auto launch = [&](auto *kernel, int per_warp) {
        const int per_block = CO_WARPS * per_warp;
        at.val.clusterDim.x = (std::min(n_events, CO_EVENTS) + per_block - 1) / per_block;
        cfg.gridDim = dim3((unsigned)(groups * at.val.clusterDim.x));
        return cudaLaunchKernelEx(&cfg, kernel, tv, toomany, n_events, stid, out, capacity, cursor);
    };
    // An event per warp while every block has an SM of its own, two beyond
    // (one / two / eight events a warp, us: 256 dimuon events 8 / 12 / 28,
    // 2,000 10 / 14 / 30, 10,000 19 / 16 / 33, 100,000 uneven 295 / 205 / 255)
    e = n_events <= CO_WARPS * sm_count ? launch(collect_kernel<1>, 1) : launch(collect_kernel<2>, 2);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace orgpu
