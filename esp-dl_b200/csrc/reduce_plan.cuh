// How channel_reduce_kernel (reduce.cu) cuts a reduction over the middle axis of [outer][count][C] into thread blocks.  Plain C++.
#pragma once

namespace espdl {

struct ReducePlan {
    int slice_lanes; // threads side by side along the channels, one vector of V of them each
    int slices;      // blocks along the channels
    int rows;        // pixels a block takes at a time
    int cluster;     // blocks that share an image and meet through distributed shared memory
};

// C channels in vectors of V, blocks of `threads`.
inline ReducePlan reduce_plan(long long outer, long long count, int C, int V, int threads, int sms)
{
    auto low = [](long long a, long long b) { return a < b ? a : b; };
    ReducePlan q;
    const int lanes = (C + V - 1) / V;
    // about sixteen pixels a thread, so that the meeting in shared memory stays small beside the loads (7x7x1280 over 1024 images:
    // 54 us with five), and at least 128 contiguous bytes a block where the tensor has them
    const long long share = low(threads, count / 16);
    const int want = (int)(share > 1 ? share : 1), widest = threads / want > 8 ? threads / want : 8;
    q.slices = (lanes + widest - 1) / widest, q.slice_lanes = (lanes + q.slices - 1) / q.slices;
    // few images: slices whose lanes are a power of two (the short meeting), although neighbouring slices then share memory sectors;
    // never wider than the even cut above, which a block's threads hold
    int pow2 = lanes & -lanes;
    while (pow2 > q.slice_lanes) pow2 /= 2;
    if ((q.slice_lanes & (q.slice_lanes - 1)) && outer * (lanes / pow2) <= sms)
        q.slice_lanes = pow2, q.slices = lanes / pow2;
    q.rows = threads / q.slice_lanes;
    // blocks that share an image: only while they do not outnumber what the SMs hold at once, and each thread keeps a full round of loads
    const int widest_cluster = threads > 256 ? 16 : 8; // 16 needs the kernel's consent
    const long long items = outer * q.slices;
    q.cluster = 1;
    while (q.cluster < widest_cluster && items * q.cluster * 2 <= 4ll * sms && count >= 8ll * q.rows * q.cluster) q.cluster *= 2;
    return q;
}

} // namespace espdl
