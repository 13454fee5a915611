// Ball query by a scan in index order, one warp per few centres (sm_100a).
//
// The rule of the op is "the first nsample candidates within the radius", so a warp that reads 128
// consecutive points at a time meets its neighbours in the order in which they are returned, and
// leaves when the list is full: after n * nsample / hits points, 2000 of 16384 where the ball of a
// centre holds 250.  Against a grid: no build, no candidates to rank, and work for every warp of
// the GPU whatever the number of clouds (a grid in shared memory is one CTA per cloud and group of
// layers); the price is the whole cloud for a centre with fewer than nsample neighbours.  So it
// serves small problems outright, and the centres that a grid leaves over because they are
// crowded, which are the ones with the shortest scans.
//
// A walk over the whole cloud takes 0.23 us per 128 points however idle the GPU is, so where there are
// few centres, up to eight warps share one: each walks a part of the cloud and keeps up to nsample
// hits in shared memory, and the lists are joined in the order of the parts.
//
// Points are read as three 16-byte loads per lane (four points), the next block while this one is
// tested, distances with the two-wide FP32 instructions, in the arithmetic of the tests:
// dense   cuda/src/ball_query_gpu.cu:35-36, strict; packed cuda/src/ball_query_gpu.cu:78-82, inclusive.
// Bound by the issue of instructions where lists stay open, by latency where they fill up.
#include "scan.cuh"

namespace tpk
{
namespace
{

constexpr int kBsThreads = 256;
constexpr int kBsBlock = 128;  // points per step of a warp
constexpr int kBsSplitSamples = 256;  // lists of that length fit shared memory for every warp (16 KB)

// W: warps that share a centre (with Q = 1, per_warp = 1 and without `need`).
// D: blocks of points on their way.
template <bool PARTIAL, int Q, int W, int D>
__device__ __forceinline__ void
    ball_scan(long long total, int per_warp, long long n, long long m, float radius, int nsample, const float* __restrict__ y,
              const float* __restrict__ x, const int64_t* __restrict__ batch_x, const int64_t* __restrict__ batch_y,
              int64_t* __restrict__ idx_out, float* __restrict__ dist_out, const unsigned char* __restrict__ need, bool unless_most)
{
    extern __shared__ int2 s_hits[];  // W > 1: index and distance of the hits, nsample for each warp
    __shared__ int s_found[kBsThreads / 32];
    const int lane = threadIdx.x & 31, slot = threadIdx.x >> 5, part = slot % W;
    const long long warp = ((static_cast<long long>(blockIdx.x) * kBsThreads + threadIdx.x) >> 5) / W;
    const long long j0 = warp * per_warp;
    if (unless_most && mostly_left<kBsThreads>(need, total)) return;  // the tiled scan has answered them all
    if (j0 >= total) return;
    int2* hits = s_hits + static_cast<size_t>(slot) * nsample;
    const float r2 = __fmul_rn(radius, radius);
    const uint32_t below = (1u << lane) - 1u;
    bool mine = lane < per_warp && j0 + lane < total;
    // `need` (optional): one byte per centre, 0 = already answered by a grid
    if (mine && need != nullptr) mine = need[j0 + lane] != 0;
    uint32_t todo = __ballot_sync(kFullMask, mine);
    while (todo != 0u)
    {
        // up to Q centres of one cloud or segment
        long long row[Q];
        bool act[Q];
        long long lo = 0, cnt = n;
        {
            int64_t group = 0;
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                act[q] = false;
                row[q] = row[0];
                if (todo == 0u) continue;
                const long long j = j0 + __ffs(todo) - 1;
                const int64_t g = PARTIAL ? __ldg(batch_y + j) : j / m;
                if (q == 0) group = g;
                if (g != group) continue;
                todo &= todo - 1u;
                act[q] = true;
                row[q] = j;
            }
            if (PARTIAL)
            {
                lo = segment_bound(batch_x, n, group, false);
                cnt = segment_bound(batch_x, n, group, true) - lo;
            }
            else
                lo = group * n;
        }
        const long long base = PARTIAL ? lo : 0;  // dense indices are local to the cloud
        const float* p = x + lo * 3;
        float qx[Q], qy[Q], qz[Q];
        long long first[Q];
        int found[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            qx[q] = __ldg(y + row[q] * 3 + 0);
            qy[q] = __ldg(y + row[q] * 3 + 1);
            qz[q] = __ldg(y + row[q] * 3 + 2);
            first[q] = PARTIAL ? -1 : 0;
            found[q] = act[q] ? 0 : nsample;
        }
        auto open = [&]() {
            bool any = false;
#pragma unroll
            for (int q = 0; q < Q; ++q) any |= found[q] < nsample;
            return any;
        };
        // one point per lane: the points before the first 16-byte boundary and behind the last block
        auto single = [&](long long k0, int count) {
            const bool in = lane < count;
            const float* s = p + 3 * (k0 + (in ? lane : 0));
            const float cx = __ldg(s), cy = __ldg(s + 1), cz = __ldg(s + 2);
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                if (found[q] >= nsample) continue;
                const float d = PARTIAL ? sumsq_loop(cx - qx[q], cy - qy[q], cz - qz[q]) : sumsq_abc(cx - qx[q], cy - qy[q], cz - qz[q]);
                const bool hit = in && (PARTIAL ? d <= r2 : d < r2);
                const uint32_t b = __ballot_sync(kFullMask, hit);
                if (b == 0u) continue;
                if (found[q] == 0) first[q] = base + k0 + __ffs(b) - 1;
                const int at = found[q] + __popc(b & below);
                if (hit && at < nsample)
                {
                    if constexpr (W > 1)
                        hits[at] = make_int2(static_cast<int>(base + k0 + lane), __float_as_int(d));
                    else
                    {
                        idx_out[row[q] * nsample + at] = base + k0 + lane;
                        dist_out[row[q] * nsample + at] = d;
                    }
                }
                found[q] += __popc(b);
            }
        };
        // 16-byte boundaries recur every four points: 12 k = -address (mod 16)
        const long long head = min(cnt, static_cast<long long>((reinterpret_cast<uintptr_t>(p) >> 2) & 3u));
        if (part == 0 && head > 0) single(0, static_cast<int>(head));
        const float4* v = reinterpret_cast<const float4*>(p + 3 * head);
        const long long blocks = (cnt - head) / kBsBlock;
        const long long t0 = blocks * part / W, t1 = blocks * (part + 1) / W;
        float4 a[D] = {}, b[D] = {}, c[D] = {};
        auto fetch = [&](int u, long long t) {
            const float4* at = v + 3 * (kBsBlock / 4) * t + 3 * lane;
            a[u] = __ldg(at + 0);
            b[u] = __ldg(at + 1);
            c[u] = __ldg(at + 2);
        };
#pragma unroll
        for (int u = 0; u < D; ++u)
            if (t0 + u < t1) fetch(u, t0 + u);
        for (long long tb = t0; tb < t1 && open(); tb += D)
#pragma unroll
        for (int u = 0; u < D; ++u)
        {
            const long long t = tb + u;
            if (u > 0 && t >= t1) break;
            const unsigned long long x01 = pack2(a[u].x, a[u].w), x23 = pack2(b[u].z, c[u].y);
            const unsigned long long y01 = pack2(a[u].y, b[u].x), y23 = pack2(b[u].w, c[u].z);
            const unsigned long long z01 = pack2(a[u].z, b[u].y), z23 = pack2(c[u].x, c[u].w);
            if (t + D < t1) fetch(u, t + D);
            const long long k0 = head + t * kBsBlock;
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                if (found[q] >= nsample) continue;
                const unsigned long long nx = pack2(-qx[q], -qx[q]), ny = pack2(-qy[q], -qy[q]), nz = pack2(-qz[q], -qz[q]);
                const unsigned long long ax = add2(x01, nx), ay = add2(y01, ny), az = add2(z01, nz);
                const unsigned long long bx = add2(x23, nx), by = add2(y23, ny), bz = add2(z23, nz);
                const unsigned long long da = PARTIAL ? fma2(az, az, fma2(ay, ay, mul2(ax, ax))) : fma2(az, az, fma2(ax, ax, mul2(ay, ay)));
                const unsigned long long db = PARTIAL ? fma2(bz, bz, fma2(by, by, mul2(bx, bx))) : fma2(bz, bz, fma2(bx, bx, mul2(by, by)));
                float d[4];
                unpack2(da, d[0], d[1]);
                unpack2(db, d[2], d[3]);
                bool hit[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) hit[i] = PARTIAL ? d[i] <= r2 : d[i] < r2;
                const uint32_t any = __ballot_sync(kFullMask, hit[0] || hit[1] || hit[2] || hit[3]);
                if (any == 0u) continue;
                int at = found[q], all = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                {
                    const uint32_t h = __ballot_sync(kFullMask, hit[i]);
                    at += __popc(h & below);
                    all += __popc(h);
                }
                if (found[q] == 0)
                {
                    const int l = __ffs(any) - 1;
                    const int i = hit[0] ? 0 : (hit[1] ? 1 : (hit[2] ? 2 : 3));
                    first[q] = base + k0 + 4 * l + __shfl_sync(kFullMask, i, l);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (hit[i])
                    {
                        if (at < nsample)
                        {
                            if constexpr (W > 1)
                                hits[at] = make_int2(static_cast<int>(base + k0 + 4 * lane + i), __float_as_int(d[i]));
                            else
                            {
                                idx_out[row[q] * nsample + at] = base + k0 + 4 * lane + i;
                                dist_out[row[q] * nsample + at] = d[i];
                            }
                        }
                        ++at;
                    }
                found[q] += all;
            }
        }
        for (long long k = head + blocks * kBsBlock; part == W - 1 && k < cnt && open(); k += 32)
            single(k, static_cast<int>(min(32ll, cnt - k)));
        if constexpr (W > 1)
        {
            // the lists of the W warps, in the order of their parts
            if (lane == 0) s_found[slot] = min(found[0], nsample);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot / W), "n"(32 * W) : "memory");
            int before = 0, all = 0;
            long long head_hit = first[0];
#pragma unroll
            for (int w = W - 1; w >= 0; --w)
            {
                const int f = s_found[slot - part + w];
                before += w < part ? f : 0;
                all += f;
                if (f > 0) head_hit = s_hits[static_cast<size_t>(slot - part + w) * nsample].x;
            }
            for (int s = lane; s < min(found[0], nsample - before); s += 32)
            {
                idx_out[row[0] * nsample + before + s] = hits[s].x;
                dist_out[row[0] * nsample + before + s] = __int_as_float(hits[s].y);
            }
            for (int s = all + 32 * part + lane; s < nsample; s += 32 * W)
            {
                idx_out[row[0] * nsample + s] = PARTIAL ? -1 : head_hit;
                dist_out[row[0] * nsample + s] = -1.0f;
            }
            return;
        }
        else
        {
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                if (!act[q]) continue;
                for (int s = min(found[q], nsample) + lane; s < nsample; s += 32)
                {
                    idx_out[row[q] * nsample + s] = PARTIAL ? -1 : first[q];
                    dist_out[row[q] * nsample + s] = -1.0f;
                }
            }
        }
    }
}

template <bool PARTIAL, int Q, int W>
__global__ void __launch_bounds__(kBsThreads)
    ball_scan_kernel(long long total, int per_warp, long long n, long long m, float radius, int nsample,
                     const float* __restrict__ y, const float* __restrict__ x, const int64_t* __restrict__ batch_x,
                     const int64_t* __restrict__ batch_y, int64_t* __restrict__ idx_out, float* __restrict__ dist_out,
                     const unsigned char* __restrict__ need, bool unless_most)
{
    ball_scan<PARTIAL, Q, W, 1>(total, per_warp, n, m, radius, nsample, y, x, batch_x, batch_y, idx_out, dist_out, need, unless_most);
}

// Two or four warps to a centre, long walks: they are too few for an SM to hide the latency with one block on its way
// (1 x 65536 points, 1800 centres, 8 and 250 in reach 106 and 56 us with one, 99 and 50 with two, in 64
// registers, so that all run at once; but 1 x 4096, 1024 centres 8.2 and 9.8, and eight warps, 8 x 131072, 64
// centres, 64 and 67).
template <int W>
__global__ void __launch_bounds__(kBsThreads, 4)
    ball_scan_shared_kernel(long long total, int per_warp, long long n, long long m, float radius, int nsample,
                            const float* __restrict__ y, const float* __restrict__ x, const int64_t* __restrict__ batch_x,
                            const int64_t* __restrict__ batch_y, int64_t* __restrict__ idx_out, float* __restrict__ dist_out,
                            const unsigned char* __restrict__ need, bool unless_most)
{
    ball_scan<false, 1, W, 2>(total, per_warp, n, m, radius, nsample, y, x, batch_x, batch_y, idx_out, dist_out, need, unless_most);
}

template <bool PARTIAL, int Q, int W>
int launch_ball_scan(long long total, int per_warp, long long n, long long m, float radius, int nsample, const float* y,
                     const float* x, const int64_t* batch_x, const int64_t* batch_y, int64_t* idx, float* dist,
                     const unsigned char* need, bool unless_most, cudaStream_t s)
{
    const long long warps = (total + per_warp - 1) / per_warp * W;
    const long long blocks = (warps + kBsThreads / 32 - 1) / (kBsThreads / 32);
    TPK_REQUIRE(blocks < (1ll << 31), "ball_query: too many centres");
    const size_t smem = W > 1 ? sizeof(int2) * kBsThreads / 32 * nsample : 0;
    count_launches(1);
    auto kernel = ball_scan_kernel<PARTIAL, Q, W>;
    if constexpr (!PARTIAL && (W == 2 || W == 4))
        if (n >= 32768) kernel = ball_scan_shared_kernel<W>;
    prefer_max_shared(kernel);
    kernel<<<static_cast<unsigned>(blocks), kBsThreads, smem, s>>>(
        total, per_warp, n, m, radius, nsample, y, x, batch_x, batch_y, idx, dist, need, unless_most);
    return check_launch("ball_query scan");
}

template <bool PARTIAL>
int pick_ball_scan(long long total, long long n, long long m, float radius, int nsample, const float* y, const float* x,
                   const int64_t* batch_x, const int64_t* batch_y, int64_t* idx, float* dist, const unsigned char* need,
                   bool unless_most, cudaStream_t s)
{
    // Centres of a warp side by side share its loads, but the first one that stays open keeps the
    // warp; a single one each while there are too few warps to hide the latency.  4096 centres of
    // 16384 points, lists that stay open: 64 us with one, 50 with two, 63 with four; lists that fill
    // up: 31, 35, 43.
    int q = total >= 16384 ? 4 : (total >= 8192 ? 2 : 1);
    if (need != nullptr) q = 2;
    // Several warps for a centre as long as they all run at once (32 on an SM) and each has 16 steps or
    // more.
    int w = 1;
    if (!PARTIAL && need == nullptr && q == 1 && nsample <= kBsSplitSamples)
        while (w < 8 && 2 * w * total <= 32ll * num_sms() && n >= 32ll * w * kBsBlock) w *= 2;
    char text[16];
    if (test_value("ball_warp_scan_q", text, sizeof(text))) q = text[0] == '4' ? 4 : (text[0] == '2' ? 2 : 1), w = 1;  // test hook
    if (!PARTIAL && need == nullptr && nsample <= kBsSplitSamples && test_value("ball_warp_scan_w", text, sizeof(text)))  // test hook
        q = 1, w = text[0] == '8' ? 8 : (text[0] == '4' ? 4 : 2);
    long long per_warp = q;
    if (need != nullptr)
    {
        // most bytes are zero: a warp reads the bytes of several centres
        per_warp = total / (32ll * num_sms());
        per_warp = per_warp < q ? q : (per_warp > 32 ? 32 : per_warp);
    }
#define TPK_BALL_SCAN(Q, W)                                                                                             \
    launch_ball_scan<PARTIAL, Q, W>(total, static_cast<int>(per_warp), n, m, radius, nsample, y, x, batch_x, batch_y, idx, \
                                    dist, need, unless_most, s)
    if constexpr (!PARTIAL)
    {
        if (w == 8) return TPK_BALL_SCAN(1, 8);
        if (w == 4) return TPK_BALL_SCAN(1, 4);
        if (w == 2) return TPK_BALL_SCAN(1, 2);
    }
    if (q == 4) return TPK_BALL_SCAN(4, 1);
    if (q == 2) return TPK_BALL_SCAN(2, 1);
    return TPK_BALL_SCAN(1, 1);
#undef TPK_BALL_SCAN
}

}  // namespace

// Whether the scan is the better way to answer all centres of a dense problem.  us, grid / scan, lists of
// 32, 8 to 16 points in reach and 250: 1 x 1024 points 15 / 7 and 63 / 6; 1 x 16384, 4096 centres 92 / 85 and
// 120 / 46; 1 x 65536, 200 centres (eight warps each) 81 / 44 and 523 / 46; 8 x 131072, 64 centres 1750 / 88 and
// 881 / 89.  Towards the bound the grid is ahead where few points are in reach, the scan where lists fill up:
// 1 x 65536, 1800 centres 94 / 133 and 628 / 95; 1 x 32768, 3600 centres 86 / 140 and 673 / 58; 16 x 16384, 440
// centres 76 / 110 and 290 / 59.
bool ball_scan_wanted(int b, int n, int m)
{
    if (test_path("ball_warp_scan")) return true;
    if (test_path("ball_query_no_warp_scan") || test_path("ball_query_global_grid")) return false;
    return static_cast<double>(b) * n * m <= 1.2e8;
}

// Candidates around a centre from which a grid leaves it to the scan.  A grid spends about two
// instructions on a candidate, and hits^2 / 8 on the order of its hits; the scan 50 on 128 points,
// n * nsample / hits of them.  Both are the same at hits^3 = 1.9 n nsample, about 100 of 16384
// points and lists of 32; 27 cells hold 4.5 times a ball's points (6.5 in space, 2.9 on a surface).
// Where the lists stay open all the same the whole cloud is read: lists longer than sqrt(1.9 n), for
// which there is the tiled scan (tpk_ball_query_dense_ws), and centres beside a clump, 4 x 65536 points,
// 16384 centres, lists of 32, 1.8 radii from clumps 2.2 ms in the grid and 2.5, 1.3 radii 2.4 and 2.5, of
// 16 2.3 and 1.5, 16 x 16384 points 0.68 and 0.50.
float ball_scan_crowded(double n, int nsample) { return static_cast<float>(4.5 * cbrt(1.9 * n * nsample)); }

// need (optional): one byte per centre, the centres with a zero are left as they are.
// unless_most: ... and all of them where mostly_left() says so.
int ball_scan_dense(int b, int n, int m, float radius, int nsample, const float* new_xyz, const float* xyz, int64_t* idx,
                    float* dist, const unsigned char* need, bool unless_most, cudaStream_t s)
{
    return pick_ball_scan<false>(static_cast<long long>(b) * m, n, m, radius, nsample, new_xyz, xyz, nullptr, nullptr, idx,
                                   dist, need, unless_most, s);
}

int ball_scan_partial(long long size_x, long long size_y, float radius, int nsample, const float* x, const float* y,
                      const int64_t* batch_x, const int64_t* batch_y, int64_t* idx, float* dist, const unsigned char* need,
                      cudaStream_t s)
{
    return pick_ball_scan<true>(size_y, size_x, 1, radius, nsample, y, x, batch_x, batch_y, idx, dist, need, false, s);
}

}  // namespace tpk
