// window_pairs.cuh -- the x-window test of make_hitpairs_in_station
// (OnlineReconstruction/reconstruction_helper.cuh:464-549): a hit is kept when
// its wire spans some of [xmin, xmax].  The pairing of the kept hits stands
// with the stages that do it (YZ and global tracking).
#pragma once
#include "or_device.cuh"

namespace orgpu {

constexpr int WP_MAXHITS = 200;  // hits of a plane the reference's arrays hold

__device__ __forceinline__ bool wp_in_window(int det, float chan, float xmin, float xmax, const or_plane_t &P) {
    const int el = (int)chan;
    float p1x, p2x;
    if (P.deltapx[det] > 0) {
        p1x = x_bep(det, el, P);
        p2x = x_tep(det, el, P);
    } else {
        p1x = x_tep(det, el, P);
        p2x = x_bep(det, el, P);
    }
    return (p1x <= xmax) && (p2x >= xmin);
}

}  // namespace orgpu
