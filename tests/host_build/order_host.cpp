// Host build of the bins that order a large wave's rays (sort_bin, pt.cu).  Test infrastructure,
// not part of the library.
#include "cuda_host_shim.h"
#include "../../rumi-renderer_b200/csrc/pt.cu"

extern "C" int rumi_host_sort_bins(int n, const float *lo_hi, const float *od, int *bins) {
    BvhNode root{lo_hi[0], lo_hi[1], lo_hi[2], lo_hi[3], lo_hi[4], lo_hi[5], 0, 0};
    DevScene S{};
    S.nodes = &root;
    for (int i = 0; i < n; ++i)
        bins[i] = rumi::sort_bin(S, make_float3(od[6 * i], od[6 * i + 1], od[6 * i + 2]),
                                 make_float3(od[6 * i + 3], od[6 * i + 4], od[6 * i + 5]));
    return rumi::SORT_BINS;
}
