// Region growing and instance IoU (the PointGroup helpers around partial_dense ball query)
// for sm_100a.
//
// grow_proximity: torch_points_kernels/cluster.py:8-46 of the reference runs a sequential
//   traversal on the CPU (numba): seeds in index order, a cluster = every point not yet
//   visited that can be reached from the seed along neighbour lists.  The lists are the
//   first nsample hits of a radius search, so the graph is directed (a crowded point may
//   not list a neighbour that lists it).  The traversal assigns point v to the smallest
//   index that can reach v along directed edges, which is a fixed point of "push the
//   smallest label seen so far along every edge": a few lanes own a point, push its
//   label to the points it lists (atomicMin) and shorten its own label chain (the label of
//   my label is also an ancestor of mine).  The host repeats launches until nothing changes.
// instance_iou:   cuda/src/metrics_gpu.cu:9-43: the reference compares every point of a proposal
//   with every ground-truth instance; here a CTA histograms the proposal's labels once.
#include <climits>

#include "tpk_common.cuh"

namespace tpk
{
namespace
{

constexpr int kClThreads = 256;

// LANES lanes per point, four slots of its list each.  A round is a chain of dependent loads (label,
// label of the label, list, labels of the listed points), so the loads of a lane are issued together
// (a thread per point read its list one slot at a time, up to the end: 21 us a round of 160000 points
// and 16 slots), and as few threads as that allows take part: with a lane per slot the chain is paid
// for in nine waves of CTAs, 27 us.  This: 15 us.  A label that is no larger already is left alone after the plain
// load: labels only fall, so an old value that is small enough settles it.
template <int LANES>
__global__ void __launch_bounds__(kClThreads)
    grow_labels_kernel(long long n, int nsample, const int64_t* __restrict__ neighbours, int32_t* labels,
                       int32_t* __restrict__ changed)
{
    constexpr int PER = 4;
    const long long u = (static_cast<long long>(blockIdx.x) * kClThreads + threadIdx.x) / LANES;
    const int lane = threadIdx.x & 31, slot = lane & (LANES - 1);
    const uint32_t group = ((1u << LANES) - 1u) << (lane & ~(LANES - 1));
    const bool in = u < n;
    const int64_t* row = neighbours + (in ? u : 0) * nsample;
    bool moved = false;
    int lu = 0;
    if (in)
    {
        // shorten the chain first: the label of my label reaches me too
        lu = __ldcg(labels + u);
        const int ll = __ldcg(labels + lu);
        if (ll < lu)
        {
            if (slot == 0) atomicMin(labels + u, ll);
            lu = ll;
            moved = true;
        }
    }
    bool ended = !in;
    for (int s0 = 0; s0 < nsample; s0 += LANES * PER)
    {
        const int s = s0 + slot * PER;
        long long v[PER];
        int label[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) v[i] = !ended && s + i < nsample ? __ldg(row + s + i) : -1;
        // the list ends at the first unused slot (cluster.py:25-26)
        const bool end_here = v[0] == -1 || v[1] == -1 || v[2] == -1 || v[3] == -1;
        const uint32_t end = __ballot_sync(kFullMask, end_here) & group;
        bool listed = end == 0u || lane <= __ffs(end) - 1;
#pragma unroll
        for (int i = 0; i < PER; ++i)
        {
            listed = listed && v[i] != -1;
            if (!listed || v[i] < 0 || v[i] >= n) v[i] = -1;
            label[i] = v[i] >= 0 ? __ldcg(labels + v[i]) : INT_MIN;
        }
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (label[i] > lu && atomicMin(labels + v[i], lu) > lu) moved = true;
        ended |= end != 0u;
        if (__all_sync(kFullMask, ended)) break;
    }
    if (moved) *changed = 1;
}

// One CTA per proposal: histogram of the ground-truth instance ids of its points, then one
// IoU per instance of the proposal's sample.
__global__ void __launch_bounds__(kClThreads)
    instance_iou_kernel(int n_proposals, long long total_gt, long long n_points, const int64_t* __restrict__ num_gt,
                        const int64_t* __restrict__ proposals_idx, const int64_t* __restrict__ proposals_offset,
                        const int64_t* __restrict__ instance_labels, const int64_t* __restrict__ offset_num_gt,
                        const int64_t* __restrict__ batch, const int64_t* __restrict__ instance_pointnum,
                        float* __restrict__ out)
{
    extern __shared__ int hist[];
    const int p = blockIdx.x;
    if (p >= n_proposals) return;
    const long long start = proposals_offset[p], end = proposals_offset[p + 1];
    if (end <= start) return;
    const long long first = proposals_idx[start];
    if (first < 0 || first >= n_points) return;
    const long long sample = batch[first];
    const int ninst = static_cast<int>(num_gt[sample]);
    const long long inst_off = offset_num_gt[sample];
    for (int i = threadIdx.x; i < ninst; i += kClThreads) hist[i] = 0;
    __syncthreads();
    for (long long i = start + threadIdx.x; i < end; i += kClThreads)
    {
        const long long idx = proposals_idx[i];
        if (idx < 0 || idx >= n_points) continue;
        const int lab = static_cast<int>(instance_labels[idx]);  // 0 is "no instance"
        if (lab >= 1 && lab <= ninst) atomicAdd(hist + lab - 1, 1);
    }
    __syncthreads();
    const int proposal_total = static_cast<int>(end - start);
    for (int i = threadIdx.x; i < ninst; i += kClThreads)
    {
        const int inter = hist[i];
        const int inst_total = static_cast<int>(instance_pointnum[inst_off + i]);
        // float / (float + double): evaluated in double, stored as float (metrics_gpu.cu:37-39)
        const double q = static_cast<double>(static_cast<float>(inter)) /
                         (static_cast<double>(static_cast<float>(proposal_total + inst_total - inter)) + 1e-5);
        out[static_cast<long long>(p) * total_gt + inst_off + i] = static_cast<float>(q);
    }
}

}  // namespace
}  // namespace tpk

extern "C" int tpk_grow_labels_step(int64_t n, int nsample, const int64_t* neighbours, int32_t* labels,
                                    int32_t* changed, int rounds, void* stream)
{
    using namespace tpk;
    TPK_REQUIRE(n >= 0 && nsample >= 0 && rounds >= 0, "grow_labels: negative size");
    TPK_REQUIRE(n < (1ll << 31), "grow_labels: too many points");
    if (n == 0 || rounds == 0) return TPK_OK;
    TPK_REQUIRE(labels && changed && (neighbours || nsample == 0), "grow_labels: NULL pointer");
    const int lanes = nsample <= 8 ? 2 : (nsample <= 16 ? 4 : 8);
    const unsigned g = static_cast<unsigned>((n * lanes + kClThreads - 1) / kClThreads);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    count_launches(rounds);
    for (int r = 0; r < rounds; ++r)
    {
        if (lanes == 2)
            grow_labels_kernel<2><<<g, kClThreads, 0, st>>>(n, nsample, neighbours, labels, changed);
        else if (lanes == 4)
            grow_labels_kernel<4><<<g, kClThreads, 0, st>>>(n, nsample, neighbours, labels, changed);
        else
            grow_labels_kernel<8><<<g, kClThreads, 0, st>>>(n, nsample, neighbours, labels, changed);
    }
    return check_launch("grow_labels");
}

extern "C" int tpk_instance_iou(int n_proposals, int64_t total_gt_instances, int64_t max_gt_instances, int64_t n_points,
                                const int64_t* num_gt_instances, const int64_t* proposals_idx,
                                const int64_t* proposals_offset, const int64_t* instance_labels,
                                const int64_t* offset_num_gt_instances, const int64_t* batch,
                                const int64_t* instance_pointnum, float* proposals_iou, void* stream)
{
    using namespace tpk;
    TPK_REQUIRE(n_proposals >= 0 && total_gt_instances >= 0 && max_gt_instances >= 0 && n_points >= 0,
                "instance_iou: negative size");
    if (n_proposals == 0 || total_gt_instances == 0) return TPK_OK;
    TPK_REQUIRE(num_gt_instances && proposals_idx && proposals_offset && instance_labels && offset_num_gt_instances && batch &&
                    instance_pointnum && proposals_iou,
                "instance_iou: NULL pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t err = cudaMemsetAsync(proposals_iou, 0, sizeof(float) * static_cast<size_t>(n_proposals) * total_gt_instances, s);
    if (err != cudaSuccess)
    {
        set_error("instance_iou: memset: %s", cudaGetErrorString(err));
        return TPK_ERR_CUDA;
    }
    const size_t smem = sizeof(int) * static_cast<size_t>(max_gt_instances > 0 ? max_gt_instances : 1);
    if (smem > 200 * 1024)
    {
        set_error("instance_iou: %lld instances in one sample exceed the %d the kernel holds",
                  static_cast<long long>(max_gt_instances), 200 * 1024 / 4);
        return TPK_ERR_UNSUPPORTED;
    }
    if (smem > kDynSmemOptIn)
    {
        err = cudaFuncSetAttribute(instance_iou_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess)
        {
            set_error("instance_iou: shared memory attribute: %s", cudaGetErrorString(err));
            return TPK_ERR_CUDA;
        }
    }
    count_launches(1), instance_iou_kernel<<<n_proposals, kClThreads, smem, s>>>(
        n_proposals, total_gt_instances, n_points, num_gt_instances, proposals_idx, proposals_offset, instance_labels,
        offset_num_gt_instances, batch, instance_pointnum, proposals_iou);
    return check_launch("instance_iou");
}
