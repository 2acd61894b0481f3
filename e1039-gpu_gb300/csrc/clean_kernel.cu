// clean_kernel.cu -- duplicate removal among YZ tracks (back-track cleaning).
//
// Replaces gKernel_BackTrackCleaning (OnlineReconstruction/
// reconstruction_helper.cuh:1789-1843) and
// gKernel_BackTrackCleaning_crossthreads (:1846-1909).
//
// For two tracks with stationID >= 5 the one with the worse chi2/(nhits-4)
// is demoted to stationID 3 when the shared (detector, element) hits exceed a
// third of its hits; the shared-hit counter keeps accumulating over the
// partners of one track, as the reference's does.
//
// One warp per event, lane t = the reference's thread t = track slot t.
//  - The first pass touches only the lane's own slot, as in the reference.
//  - In the cross-slot pass the reference's 32 threads run the same loop
//    nest together: at step (i_trd, i, j) every thread t != i_trd compares
//    its track i with track j of slot i_trd, reading the stationIDs the
//    earlier steps left, and the demotions of the step land after it.  The
//    lanes follow that lockstep order exactly: read and decide, then demote.
//    All writes store the same value (3), so lanes demoting the same track do
//    not conflict.
#include "or_device.cuh"

namespace orgpu {

// shared (detector, element) hits of A's hits found among B's, H:1810-1817
__device__ __forceinline__ int common_hits(const float *A, int na, const float *B, int nb) {
    int acc = 0;
    for (int ih = 0; ih < na; ++ih) {
        const float d = A[OR_TRK_HIT_DETID + ih], c = A[OR_TRK_HIT_CHAN + ih];
        for (int jh = 0; jh < nb; ++jh) {
            if (B[OR_TRK_HIT_DETID + jh] == d && B[OR_TRK_HIT_CHAN + jh] == c) {
                ++acc;
                break;
            }
        }
    }
    return acc;
}

// the comparison of H:1819-1838 / H:1886-1904: 1 = demote j, 2 = demote i
__device__ __forceinline__ int clean_decide(const float *Ti, int ni, const float *Tj, int nj, int nc) {
    if (Ti[OR_TRK_CHI2] / (float)(ni - 4) < Tj[OR_TRK_CHI2] / (float)(nj - 4))
        return ((float)nc > (float)ni * 0.3333f) ? 1 : 0;
    return ((float)nc > (float)nj * 0.3333f) ? 2 : 0;
}

// The general form, on the records themselves: any detector ids and channels.
static __device__ __noinline__ void clean_event_general(const or_tracks_view_t &tv, long e, int n_own) {
    const int lane = threadIdx.x & 31;
    // --- pass 1: the lane's own slot (H:1789-1843) ------------------------
    for (int i = 0; i < n_own; ++i) {
        float *Ti = trk_rec(tv, e, lane, i);
        if (Ti[OR_TRK_STID] < 5) continue;
        const int ni = min((int)(short)Ti[OR_TRK_NHITS], OR_MAXHITS_PER_TRACK);
        int nc = 0;
        for (int j = i + 1; j < n_own; ++j) {
            float *Tj = trk_rec(tv, e, lane, j);
            if (Tj[OR_TRK_STID] < 5) continue;
            const int nj = min((int)(short)Tj[OR_TRK_NHITS], OR_MAXHITS_PER_TRACK);
            nc += common_hits(Ti, ni, Tj, nj);
            const int d = clean_decide(Ti, ni, Tj, nj, nc);
            if (d == 1) Tj[OR_TRK_STID] = 3.f;
            else if (d == 2) Ti[OR_TRK_STID] = 3.f;
        }
    }
    __syncwarp();
    // --- pass 2: across slots, in lockstep (H:1846-1909) ------------------
    const int maxn = __reduce_max_sync(0xffffffffu, (unsigned)n_own);
    for (int u = 0; u < OR_NSLOTS; ++u) {
        const int m = __shfl_sync(0xffffffffu, n_own, u);
        if (m == 0) continue;
        for (int i = 0; i < maxn; ++i) {
            float *Ti = (i < n_own) ? trk_rec(tv, e, lane, i) : nullptr;
            const bool act = lane != u && Ti && Ti[OR_TRK_STID] >= 5;
            const int ni = act ? min((int)(short)Ti[OR_TRK_NHITS], OR_MAXHITS_PER_TRACK) : 0;
            if (!__any_sync(0xffffffffu, act)) continue;
            int nc = 0;
            for (int j = 0; j < m; ++j) {
                float *Tj = trk_rec(tv, e, u, j);
                const bool alive_j = Tj[OR_TRK_STID] >= 5;  // same record for every lane
                int d = 0;
                if (act && alive_j) {
                    const int nj = min((int)(short)Tj[OR_TRK_NHITS], OR_MAXHITS_PER_TRACK);
                    nc += common_hits(Ti, ni, Tj, nj);
                    d = clean_decide(Ti, ni, Tj, nj, nc);
                }
                __syncwarp();
                if (d == 1) Tj[OR_TRK_STID] = 3.f;
                else if (d == 2) Ti[OR_TRK_STID] = 3.f;
                __syncwarp();
            }
        }
    }
}

// Shared hits by bytes.  Tracks as YZ tracking leaves them have at most one
// hit per plane, on planes 13..30, with channels 1..255: a track is then 18
// bytes, its channel on each plane (0: none), and the shared hits of two
// tracks are the equal non-zero bytes.
constexpr int CL_PLANE0 = 13, CL_WORDS = 5;

struct ClWarp {
    uint32_t hits[OR_TRKMAX][CL_WORDS];
    float ratio[OR_TRKMAX];     // chi2 / (nhits - 4)
    int16_t nhits[OR_TRKMAX];
    uint16_t track[OR_TRKMAX];  // slot * 16 + position
};

__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t v) { return __vcmpne4(v, 0u); }

__device__ __forceinline__ int common_bytes(const uint32_t *a, const uint32_t *nz, const uint32_t *b) {
    int c = 0;
#pragma unroll
    for (int q = 0; q < CL_WORDS; ++q) c += __popc(__vcmpeq4(a[q], b[q]) & nz[q]);
    return c >> 3;
}

// clean_decide with the precomputed ratio of each track
__device__ __forceinline__ int clean_decide_pre(float ri, int ni, float rj, int nj, int nc) {
    if (ri < rj) return ((float)nc > (float)ni * 0.3333f) ? 1 : 0;
    return ((float)nc > (float)nj * 0.3333f) ? 2 : 0;
}

// Work per event: only the tracks with stationID >= 5 are read, each once,
// into shared memory (28 bytes instead of 300), and a step of the cross-slot
// pass runs only where both sides have a live track (the lane's 16-bit mask
// of live positions; a step's demotions clear bits after it, as the writes of
// the general form land after it).  Bound: DRAM latency for the loads, then
// the lockstep order of one heavy event's steps.  The general form for every
// event took 319 us for a single uneven event, 714 us for 333 of them and
// 3,378 us for 100,000; this takes 28, 63 and 585 us.
template <int W>
__global__ void __launch_bounds__(W * 32)
    clean_kernel(or_tracks_view_t tv, const uint8_t *__restrict__ toomany, int n_events) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    ClWarp &S = reinterpret_cast<ClWarp *>(cl_smem)[w];
    for (long e = (long)blockIdx.x * W + w; e < n_events; e += (long)gridDim.x * W) {
        if (toomany[e]) continue;
        const int n_own = min((int)tv.ntracks[e * OR_NSLOTS + lane], OR_SLOTCAP);
        const int most = __reduce_max_sync(0xffffffffu, n_own);
        unsigned live = 0u;  // the lane's slot: positions with stationID >= 5
#pragma unroll 4
        for (int k = 0; k < most; ++k)
            if (k < n_own && trk_rec(tv, e, lane, k)[OR_TRK_STID] >= 5) live |= 1u << k;
        const int c = __popc(live);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        if (total < 2) continue;  // nothing to compare
        const int first = incl - c;  // the slot's first entry
        {
            int at = first;
            for (unsigned m = live; m; m &= m - 1) S.track[at++] = (uint16_t)(lane * OR_SLOTCAP + __ffs(m) - 1);
        }
        for (int i = lane; i < total * CL_WORDS; i += 32) S.hits[0][i] = 0u;
        __syncwarp();
        const float *rec = trk_rec(tv, e, 0, 0);
        bool odd = false;
#pragma unroll 2
        for (int i = lane; i < total; i += 32) {
            const float *T = rec + (long)S.track[i] * OR_NTRKPARAM;
            const int nh = min((int)(short)T[OR_TRK_NHITS], OR_MAXHITS_PER_TRACK);
            S.ratio[i] = T[OR_TRK_CHI2] / (float)(nh - 4);
            S.nhits[i] = (int16_t)nh;
        }
#pragma unroll 4
        for (int i = lane; i < total * OR_MAXHITS_PER_TRACK; i += 32) {
            const int t = i / OR_MAXHITS_PER_TRACK, h = i - t * OR_MAXHITS_PER_TRACK;
            const float *T = rec + (long)S.track[t] * OR_NTRKPARAM;
            const int nh = min((int)(short)T[OR_TRK_NHITS], OR_MAXHITS_PER_TRACK);
            const float d = T[OR_TRK_HIT_DETID + h], ch = T[OR_TRK_HIT_CHAN + h];
            if (h < nh) {
                const int di = (int)d, ci = (int)ch;
                const bool fits = d >= (float)CL_PLANE0 && d <= (float)OR_NCHAM && (float)di == d && ch >= 1.f &&
                                  ch <= 255.f && (float)ci == ch;
                if (fits) {
                    const int p = di - CL_PLANE0, sh = (p & 3) * 8;
                    const uint32_t old = atomicOr(&S.hits[t][p >> 2], (uint32_t)ci << sh);
                    odd |= ((old >> sh) & 0xFFu) != 0u;  // two hits on one plane
                } else {
                    odd = true;
                }
            }
        }
        if (__any_sync(0xffffffffu, odd)) {
            clean_event_general(tv, e, n_own);
            continue;
        }
        __syncwarp();
        const unsigned before = live;
        // entry of position k of the slot whose live mask was `m` and whose
        // first entry is f: the entries keep their places as tracks die
        auto entry = [](unsigned m, int f, int k) { return f + __popc(m & ((1u << k) - 1u)); };
        // --- pass 1: the lane's own slot (H:1789-1843) ------------------------
        if (c > 1) {
            for (unsigned mi = before; mi; mi &= mi - 1) {
                const int i = __ffs(mi) - 1;
                if (!((live >> i) & 1u)) continue;
                const int ei = entry(before, first, i);
                uint32_t a[CL_WORDS], nz[CL_WORDS];
#pragma unroll
                for (int q = 0; q < CL_WORDS; ++q) {
                    a[q] = S.hits[ei][q];
                    nz[q] = nonzero_bytes(a[q]);
                }
                const float ri = S.ratio[ei];
                const int ni = S.nhits[ei];
                int nc = 0;
                for (unsigned mj = mi & (mi - 1); mj; mj &= mj - 1) {
                    const int j = __ffs(mj) - 1;
                    if (!((live >> j) & 1u)) continue;
                    const int ej = entry(before, first, j);
                    nc += common_bytes(a, nz, S.hits[ej]);
                    const int d = clean_decide_pre(ri, ni, S.ratio[ej], S.nhits[ej], nc);
                    if (d == 1) live &= ~(1u << j);
                    else if (d == 2) live &= ~(1u << i);
                }
            }
        }
        __syncwarp();
        // --- pass 2: across slots, in lockstep (H:1846-1909) ------------------
        unsigned slots = __ballot_sync(0xffffffffu, live != 0u);
        for (; slots; slots &= slots - 1) {
            const int u = __ffs(slots) - 1;
            unsigned mu = __shfl_sync(0xffffffffu, live, u);
            const unsigned bu = __shfl_sync(0xffffffffu, before, u);
            const int fu = __shfl_sync(0xffffffffu, first, u);
            unsigned todo = __reduce_or_sync(0xffffffffu, lane != u ? live : 0u);
            for (; todo && mu; todo &= todo - 1) {
                const int i = __ffs(todo) - 1;
                const bool act = lane != u && ((live >> i) & 1u);
                const int ei = act ? entry(before, first, i) : 0;
                uint32_t a[CL_WORDS], nz[CL_WORDS];
#pragma unroll
                for (int q = 0; q < CL_WORDS; ++q) {
                    a[q] = S.hits[ei][q];
                    nz[q] = act ? nonzero_bytes(a[q]) : 0u;
                }
                const float ri = S.ratio[ei];
                const int ni = S.nhits[ei];
                int nc = 0;
                unsigned dead = 0u;
                bool own = false;
                // a step demotes track j of slot u or a lane's track i, never
                // a later j, so the slot's live tracks are those at the start
                for (unsigned mj = mu; mj; mj &= mj - 1) {
                    const int j = __ffs(mj) - 1;
                    const int ej = entry(bu, fu, j);
                    nc += common_bytes(a, nz, S.hits[ej]);
                    const int d = act ? clean_decide_pre(ri, ni, S.ratio[ej], S.nhits[ej], nc) : 0;
                    own |= d == 2;
                    if (__any_sync(0xffffffffu, d == 1)) dead |= 1u << j;
                }
                if (own) live &= ~(1u << i);
                mu &= ~dead;
                if (lane == u) live = mu;
            }
        }
        for (unsigned m = before & ~live; m; m &= m - 1) trk_rec(tv, e, lane, __ffs(m) - 1)[OR_TRK_STID] = 3.f;
        __syncwarp();
    }
}

template <int W>
static cudaError_t clean_launch(or_tracks_view_t tv, const uint8_t *toomany, int n_events, cudaStream_t stream,
                                int sm_count) {
    const size_t smem = sizeof(ClWarp) * W;
    cudaError_t err = smem_attr_once((const void *)clean_kernel<W>, (int)smem);
    if (err != cudaSuccess) return err;
    long blocks = (n_events + W - 1) / W;
    const long cap = (long)sm_count * (16 / W);  // 16 warps of ClWarp fill an SM's shared memory
    if (blocks > cap) blocks = cap;
    clean_kernel<W><<<(unsigned)blocks, W * 32, smem, stream>>>(tv, toomany, n_events);
    return cudaGetLastError();
}

cudaError_t launch_back_clean(or_tracks_view_t tv, const uint8_t *toomany, int n_events, cudaStream_t stream,
                              int sm_count, int warps) {
    if (n_events <= 0) return cudaSuccess;
    switch (warps) {
    case 1: return clean_launch<1>(tv, toomany, n_events, stream, sm_count);
    case 2: return clean_launch<2>(tv, toomany, n_events, stream, sm_count);
    case 8: return clean_launch<8>(tv, toomany, n_events, stream, sm_count);
    case 16: return clean_launch<16>(tv, toomany, n_events, stream, sm_count);
    default: return clean_launch<4>(tv, toomany, n_events, stream, sm_count);
    }
}

}  // namespace orgpu
