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
// each scheduler (four to an SM) as hold the items, all schedulers alike; all
// warps alike where the launch has fewer than that.  The shares hold every
// item: warps that left some unclaimed beside idle lanes would break the bound
// on a batch's or graph's launches (fp32_launch_bound), which counts on slots
// that never idle while items remain.  Every warp and every lane where there
// are more items than lanes.
LDP_SHARE_FN Share share_out(unsigned long long avail, unsigned sms, unsigned wps) {
    const unsigned warps = sms * wps, schedulers = sms * 4;
    if (avail == 0 || avail > (unsigned long long)warps * 32) return Share{warps, 32};
    const unsigned n = (unsigned)avail, k = (n + schedulers * 32 - 1) / (schedulers * 32);
    const unsigned share = schedulers * k < warps ? schedulers * k : warps;
    const unsigned lanes = (n + share - 1) / share;        // at most 32
    return Share{(n + lanes - 1) / lanes, lanes};          // the last one fills fewer
}

}  // namespace ldp
