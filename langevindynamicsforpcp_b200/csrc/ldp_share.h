// ldp_share.h -- how a persistent FP32 launch shares few items out over its
// warps.  Plain C++ (host and device), so the CPU tests exercise it.
#pragma once

#if defined(__CUDACC__)
#define LDP_SHARE_FN __host__ __device__ __forceinline__
#else
#define LDP_SHARE_FN inline
#endif

namespace ldp {

// The warps that take items at their first claim, and the lanes each fills
// (a warp's turn past `warps` leaves the items to the others at first).
struct Share {
    unsigned warps, lanes;
};

// avail unclaimed items over `sms` SMs of `wps` warps each: as few warps to
// each scheduler (four to an SM) as hold the items, all schedulers alike.
// Every warp and every lane where there are more items than lanes, and where
// the launch has fewer warps than that takes (shapes of fewer warps to an SM
// than schedulers): warps that each fill their share only would leave items
// unclaimed beside idle lanes, and a batch's or graph's number of launches is
// bounded for slots that never idle while items remain (fp32_launch_bound).
LDP_SHARE_FN Share share_out(unsigned long long avail, unsigned sms, unsigned wps) {
    const unsigned warps = sms * wps, schedulers = sms * 4;
    const Share all{warps, 32};
    if (avail == 0 || avail > (unsigned long long)warps * 32) return all;
    const unsigned n = (unsigned)avail, k = (n + schedulers * 32 - 1) / (schedulers * 32);
    const unsigned lanes = (n + schedulers * k - 1) / (schedulers * k);   // at most 32
    const unsigned used = (n + lanes - 1) / lanes;                        // the last one fills fewer
    return used > warps ? all : Share{used, lanes};
}

}  // namespace ldp
