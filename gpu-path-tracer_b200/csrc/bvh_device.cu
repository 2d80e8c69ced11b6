// Device construction of the BVH8 (gpt_set_bvh_build(GPT_BVH_BUILD_DEVICE)). It writes the node
// format, single-triangle leaves and triangle records of the host builder (bvh8.cpp) and uses its
// surface-area-optimal 8-wide collapse, slot assignment and quantisation; the binary tree the wide
// tree is collapsed from is built on the GPU by clustering instead of the host's binned SAH:
//
// 1. Triangle boxes and centroids, and the centroids' bounds (two-pass reduction).
// 2. 30-bit Morton codes of the centroids; triangles sorted by code (cub::DeviceRadixSort).
// 3. PLOC (Meister and Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume Hierarchy
//    Construction", IEEE TVCG 2018): the clusters stay in Morton order; each finds the cluster within
//    kPlocRadius positions whose merged box has the smallest surface area (the nearer position wins a
//    tie), mutual nearest neighbours merge, and the survivors are compacted in order by prefix sums,
//    until one cluster is left. The nodes of one round get consecutive indices after those of the
//    rounds before, so every node has a larger index than its children. The cluster count stays on the
//    device, and the host reads it every kRoundsPerSync rounds only; the last rounds, with at most
//    kTailClusters clusters, run in one block.
// 4. The collapse's cost table (Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on
//    GPUs Through Compressed Wide BVHs", HPG 2017), bottom-up one round of nodes at a time.
// 5. Wide nodes level by level from the root: each collects its children from the cost table,
//    assigns them to slots by octant, quantises their boxes in double precision with outward
//    rounding and reserves consecutive indices for its inner children with one atomic.
// 6. Headers and triangle records move into their places in the child blocks, which step 5 assigned
//    (node j's children are block j + 1).
//
// Hits do not depend on the tree (the traversal is conservative and ties go to the smaller input
// index), so frames equal those of a host-built BVH bit for bit; only the traversal work differs.
#include <cfloat>
#include <cstdint>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "bvh_device.hpp"

namespace pt
{
    namespace
    {
        constexpr int kPlocRadius = 16;
        constexpr int kPlocBlock = 256;
        constexpr uint32_t kTailClusters = 1024;  // clusters (and threads) of the one-block rounds
        constexpr int kRoundsPerSync = 3;         // grids are sized by the last count read, at most 8 times too large then
        constexpr float kCollapseNodeCost = 2.0f;  // a wide-node visit against one triangle test (bvh8.cpp)
        constexpr int kCollectStack = 24;
        constexpr uint32_t kBuildErrExponent = 1u;  // quantisation exponent overflow
        constexpr uint32_t kBuildErrCollect = 2u;   // a node's child list did not fit its slots
        constexpr uint32_t kBuildErrCapacity = 4u;  // a wide-node index beyond the node array

        __device__ __forceinline__ float box_area(float4 lo, float4 hi)
        {
            const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
            if (dx < 0.0f || dy < 0.0f || dz < 0.0f) return 0.0f;
            return 2.0f * (dx * dy + dy * dz + dz * dx);
        }

        __device__ __forceinline__ float4 fmin4(float4 a, float4 b) { return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f); }
        __device__ __forceinline__ float4 fmax4(float4 a, float4 b) { return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.0f); }

        // Triangle boxes (leaf k of the sort is written later, by permutation) and centroids; per-block
        // bounds of the centroids.
        __global__ void triangle_boxes_kernel(const float* pos, uint32_t n, float4* triLo, float4* triHi, float4* cent, float4* partLo, float4* partHi)
        {
            __shared__ float4 sLo[256], sHi[256];
            float4 lo = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.0f), hi = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.0f);
            for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
            {
                const float* p = pos + static_cast<size_t>(t) * 9;
                float4 bl = make_float4(p[0], p[1], p[2], 0.0f), bh = bl;
                for (int k = 1; k < 3; k++)
                {
                    const float4 v = make_float4(p[3 * k], p[3 * k + 1], p[3 * k + 2], 0.0f);
                    bl = fmin4(bl, v);
                    bh = fmax4(bh, v);
                }
                triLo[t] = bl;
                triHi[t] = bh;
                const float4 c = make_float4(0.5f * (bl.x + bh.x), 0.5f * (bl.y + bh.y), 0.5f * (bl.z + bh.z), 0.0f);
                cent[t] = c;
                lo = fmin4(lo, c);
                hi = fmax4(hi, c);
            }
            sLo[threadIdx.x] = lo;
            sHi[threadIdx.x] = hi;
            __syncthreads();
            for (uint32_t s = blockDim.x / 2; s > 0; s >>= 1)
            {
                if (threadIdx.x < s)
                {
                    sLo[threadIdx.x] = fmin4(sLo[threadIdx.x], sLo[threadIdx.x + s]);
                    sHi[threadIdx.x] = fmax4(sHi[threadIdx.x], sHi[threadIdx.x + s]);
                }
                __syncthreads();
            }
            if (threadIdx.x == 0)
            {
                partLo[blockIdx.x] = sLo[0];
                partHi[blockIdx.x] = sHi[0];
            }
        }

        __device__ __forceinline__ uint32_t expand_bits10(uint32_t v)
        {
            v = (v * 0x00010001u) & 0xFF0000FFu;
            v = (v * 0x00000101u) & 0x0F00F00Fu;
            v = (v * 0x00000011u) & 0xC30C30C3u;
            v = (v * 0x00000005u) & 0x49249249u;
            return v;
        }

        // One block of 256 threads: the bounds of the per-block bounds, into entry 0.
        __global__ void bounds_final_kernel(float4* partLo, float4* partHi, uint32_t parts)
        {
            __shared__ float4 sLo[256], sHi[256];
            float4 lo = partLo[0], hi = partHi[0];
            for (uint32_t i = threadIdx.x; i < parts; i += blockDim.x)
            {
                lo = fmin4(lo, partLo[i]);
                hi = fmax4(hi, partHi[i]);
            }
            sLo[threadIdx.x] = lo;
            sHi[threadIdx.x] = hi;
            __syncthreads();
            for (uint32_t s = blockDim.x / 2; s > 0; s >>= 1)
            {
                if (threadIdx.x < s)
                {
                    sLo[threadIdx.x] = fmin4(sLo[threadIdx.x], sLo[threadIdx.x + s]);
                    sHi[threadIdx.x] = fmax4(sHi[threadIdx.x], sHi[threadIdx.x + s]);
                }
                __syncthreads();
            }
            if (threadIdx.x == 0)
            {
                partLo[0] = sLo[0];
                partHi[0] = sHi[0];
            }
        }

        // The Morton code of every centroid within the centroids' bounds.
        __global__ void morton_kernel(const float4* cent, uint32_t n, const float4* boundsLo, const float4* boundsHi, uint32_t* keys, uint32_t* values)
        {
            const float4 lo = boundsLo[0], hi = boundsHi[0];
            const float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
            const float sx = ex > 0.0f ? 1023.0f / ex : 0.0f, sy = ey > 0.0f ? 1023.0f / ey : 0.0f, sz = ez > 0.0f ? 1023.0f / ez : 0.0f;
            for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
            {
                const float4 c = cent[t];
                const uint32_t x = static_cast<uint32_t>(fminf(fmaxf((c.x - lo.x) * sx, 0.0f), 1023.0f));
                const uint32_t y = static_cast<uint32_t>(fminf(fmaxf((c.y - lo.y) * sy, 0.0f), 1023.0f));
                const uint32_t z = static_cast<uint32_t>(fminf(fmaxf((c.z - lo.z) * sz, 0.0f), 1023.0f));
                keys[t] = (expand_bits10(x) << 2) | (expand_bits10(y) << 1) | expand_bits10(z);
                values[t] = t;
            }
        }

        // Leaf k = the k-th triangle of the sort; every cluster starts as one leaf.
        __global__ void leaves_kernel(const uint32_t* sorted, uint32_t n, const float4* triLo, const float4* triHi, float4* lo, float4* hi,
                                      uint2* child, uint32_t* clusters)
        {
            for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
            {
                const uint32_t t = sorted[k];
                lo[k] = triLo[t];
                hi[k] = triHi[t];
                child[k] = make_uint2(kInvalid, kInvalid);
                clusters[k] = k;
            }
        }

        // Nearest neighbour of every cluster within kPlocRadius positions (surface area of the merged box).
        // Clustering state on the device: clusters left, next node index, rounds done (roundEnd[r]: first node
        // index behind round r - 1), and whether a round merged nothing.
        struct PlocState
        {
            uint32_t clusters, nodes, rounds, stalled;
        };

        __global__ void __launch_bounds__(kPlocBlock) ploc_nearest_kernel(const uint32_t* clusters, const PlocState* state, const float4* lo,
                                                                          const float4* hi, uint32_t* nn)
        {
            const uint32_t m = state->clusters;
            if (blockIdx.x * kPlocBlock >= m) return;
            __shared__ float4 sLo[kPlocBlock + 2 * kPlocRadius], sHi[kPlocBlock + 2 * kPlocRadius];
            const int start = static_cast<int>(blockIdx.x) * kPlocBlock - kPlocRadius;
            for (int k = threadIdx.x; k < kPlocBlock + 2 * kPlocRadius; k += kPlocBlock)
            {
                const int i = start + k;
                if (i >= 0 && i < static_cast<int>(m))
                {
                    const uint32_t c = clusters[i];
                    sLo[k] = lo[c];
                    sHi[k] = hi[c];
                }
            }
            __syncthreads();
            const int i = static_cast<int>(blockIdx.x) * kPlocBlock + static_cast<int>(threadIdx.x);
            if (i >= static_cast<int>(m)) return;
            const int si = i - start;
            const float4 myLo = sLo[si], myHi = sHi[si];
            const int jLo = i - kPlocRadius < 0 ? 0 : i - kPlocRadius;
            const int jHi = i + kPlocRadius > static_cast<int>(m) - 1 ? static_cast<int>(m) - 1 : i + kPlocRadius;
            float best = FLT_MAX;
            int bj = i == 0 ? 1 : i - 1;
            for (int j = jLo; j <= jHi; j++)
            {
                if (j == i) continue;
                const float a = box_area(fmin4(myLo, sLo[j - start]), fmax4(myHi, sHi[j - start]));
                if (a < best)
                {
                    best = a;
                    bj = j;
                }
            }
            nn[i] = static_cast<uint32_t>(bj);
        }

        // flags[i], low word: cluster i merges with its neighbour into a new node (mutual pair, i the smaller);
        // high word: a cluster survives at position i (unpaired, or the smaller of a pair). Entries from the
        // cluster count on are 0, so the exclusive sums at the count are the totals.
        __global__ void ploc_flags_kernel(const uint32_t* nn, const PlocState* state, uint32_t entries, unsigned long long* flags)
        {
            const uint32_t m = state->clusters;
            for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < entries; i += gridDim.x * blockDim.x)
            {
                unsigned long long f = 0;
                if (i < m)
                {
                    const uint32_t j = nn[i];
                    const bool mutual = nn[j] == i;
                    f = (mutual && i < j ? 1ull : 0ull) | (mutual && i > j ? 0ull : 1ull << 32);
                }
                flags[i] = f;
            }
        }

        __global__ void ploc_merge_kernel(const uint32_t* clusters, const PlocState* state, const uint32_t* nn, const unsigned long long* flags,
                                          const unsigned long long* positions, float4* lo, float4* hi, uint2* child, uint32_t* next)
        {
            const uint32_t m = state->clusters, nodeBase = state->nodes;
            for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
            {
                const unsigned long long f = flags[i], at = positions[i];
                if ((f >> 32) == 0) continue;
                uint32_t id = clusters[i];
                if (f & 1u)
                {
                    const uint32_t other = clusters[nn[i]];
                    const uint32_t fresh = nodeBase + static_cast<uint32_t>(at);
                    child[fresh] = make_uint2(id, other);
                    lo[fresh] = fmin4(lo[id], lo[other]);
                    hi[fresh] = fmax4(hi[id], hi[other]);
                    id = fresh;
                }
                next[at >> 32] = id;
            }
        }

        __global__ void ploc_advance_kernel(PlocState* state, const unsigned long long* positions, uint32_t* roundEnd)
        {
            const unsigned long long totals = positions[state->clusters];
            const uint32_t merged = static_cast<uint32_t>(totals), kept = static_cast<uint32_t>(totals >> 32);
            if (merged == 0 || kept != state->clusters - merged)
            {
                state->stalled = 1;
                return;
            }
            state->nodes += merged;
            state->clusters = kept;
            roundEnd[++state->rounds] = state->nodes;
        }

        // The rounds from at most kTailClusters clusters on, in one block: the same rounds (and so the same
        // nodes), with the clusters' boxes in shared memory. Half of a build's rounds have this few clusters, and
        // as launches with a read of the count they took about 70 us each.
        __global__ void __launch_bounds__(kTailClusters) ploc_tail_kernel(const uint32_t* clusters, PlocState* state, float4* lo, float4* hi,
                                                                          uint2* child, uint32_t* roundEnd)
        {
            extern __shared__ float4 boxes[];
            float4* sLo = boxes;
            float4* sHi = boxes + kTailClusters;
            __shared__ uint32_t sNear[kTailClusters], sId[kTailClusters], warpMerged[32], warpKept[32];
            const uint32_t i = threadIdx.x, lane = i & 31u, warp = i >> 5;
            uint32_t m = state->clusters, nodes = state->nodes, rounds = state->rounds;
            uint32_t id = 0;
            float4 myLo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), myHi = myLo;
            if (i < m)
            {
                id = clusters[i];
                myLo = lo[id];
                myHi = hi[id];
            }
            while (m > 1)
            {
                sLo[i] = myLo;
                sHi[i] = myHi;
                sId[i] = id;
                __syncthreads();
                uint32_t bj = i == 0 ? 1u : i - 1u;
                if (i < m)
                {
                    const uint32_t jLo = i < kPlocRadius ? 0u : i - kPlocRadius;
                    const uint32_t jHi = i + kPlocRadius > m - 1u ? m - 1u : i + kPlocRadius;
                    float best = FLT_MAX;
                    for (uint32_t j = jLo; j <= jHi; j++)
                    {
                        if (j == i) continue;
                        const float a = box_area(fmin4(myLo, sLo[j]), fmax4(myHi, sHi[j]));
                        if (a < best)
                        {
                            best = a;
                            bj = j;
                        }
                    }
                    sNear[i] = bj;
                }
                __syncthreads();
                const bool mutual = i < m && sNear[bj] == i;
                const bool merges = mutual && i < bj, keeps = i < m && !(mutual && i > bj);
                const unsigned mergedMask = __ballot_sync(0xFFFFFFFFu, merges), keptMask = __ballot_sync(0xFFFFFFFFu, keeps);
                if (lane == 0)
                {
                    warpMerged[warp] = static_cast<uint32_t>(__popc(mergedMask));
                    warpKept[warp] = static_cast<uint32_t>(__popc(keptMask));
                }
                __syncthreads();
                uint32_t mergedBefore = 0, keptBefore = 0, merged = 0, kept = 0;
                for (uint32_t w = 0; w < kTailClusters / 32; w++)
                {
                    mergedBefore += w < warp ? warpMerged[w] : 0u;
                    keptBefore += w < warp ? warpKept[w] : 0u;
                    merged += warpMerged[w];
                    kept += warpKept[w];
                }
                if (merged == 0 || kept != m - merged)
                {
                    if (i == 0) state->stalled = 1;
                    return;
                }
                const unsigned below = (1u << lane) - 1u;
                if (merges)
                {
                    const uint32_t fresh = nodes + mergedBefore + static_cast<uint32_t>(__popc(mergedMask & below));
                    child[fresh] = make_uint2(id, sId[bj]);
                    myLo = fmin4(myLo, sLo[bj]);
                    myHi = fmax4(myHi, sHi[bj]);
                    lo[fresh] = myLo;
                    hi[fresh] = myHi;
                    id = fresh;
                }
                __syncthreads();
                if (keeps)
                {
                    const uint32_t at = keptBefore + static_cast<uint32_t>(__popc(keptMask & below));
                    sId[at] = id;
                    sLo[at] = myLo;
                    sHi[at] = myHi;
                }
                __syncthreads();
                m = kept;
                nodes += merged;
                rounds++;
                if (i == 0) roundEnd[rounds] = nodes;
                if (i < m)
                {
                    id = sId[i];
                    myLo = sLo[i];
                    myHi = sHi[i];
                }
                __syncthreads();
            }
            if (i == 0)
            {
                state->clusters = m;
                state->nodes = nodes;
                state->rounds = rounds;
            }
        }

        // Collapse costs (bvh8.cpp, CollapsePlan::plan): cost[8 i + j - 1] = cost of node i taking j slots
        // of its parent, how[] the choice, split[i] the left child's share when i becomes a wide node.
        __global__ void collapse_leaf_kernel(uint32_t n, const float4* lo, const float4* hi, float* cost, uint8_t* how)
        {
            for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            {
                const float A = box_area(lo[i], hi[i]);
                for (int k = 0; k < 8; k++)
                {
                    cost[static_cast<size_t>(i) * 8 + k] = A;  // area x one triangle
                    how[static_cast<size_t>(i) * 8 + k] = 0;
                }
            }
        }

        __device__ void collapse_node(uint32_t i, const float4* lo, const float4* hi, const uint2* child, float* cost, uint8_t* how, uint8_t* split)
        {
            {
                const float A = box_area(lo[i], hi[i]);
                const uint2 c = child[i];
                const float* L = cost + static_cast<size_t>(c.x) * 8;
                const float* R = cost + static_cast<size_t>(c.y) * 8;
                float l[8], r[8];
                for (int k = 0; k < 8; k++)
                {
                    l[k] = L[k];
                    r[k] = R[k];
                }
                float D[9];
                uint8_t Dk[9] = {};
                for (int j = 2; j <= 8; j++)
                {
                    D[j] = FLT_MAX;
                    for (int k = 1; k < j; k++)
                    {
                        const float v = l[k - 1] + r[j - k - 1];
                        if (v < D[j])
                        {
                            D[j] = v;
                            Dk[j] = static_cast<uint8_t>(k);
                        }
                    }
                }
                split[i] = Dk[8];
                float C[8];
                uint8_t H[8];
                C[0] = A * kCollapseNodeCost + D[8];  // two or more triangles: never one leaf slot
                H[0] = 1;
                for (int s = 2; s <= 8; s++)
                {
                    if (D[s] < C[s - 2])
                    {
                        C[s - 1] = D[s];
                        H[s - 1] = Dk[s];
                    }
                    else
                    {
                        C[s - 1] = C[s - 2];
                        H[s - 1] = 0;
                    }
                }
                for (int k = 0; k < 8; k++)
                {
                    cost[static_cast<size_t>(i) * 8 + k] = C[k];
                    how[static_cast<size_t>(i) * 8 + k] = H[k];
                }
            }
        }

        __global__ void collapse_node_kernel(uint32_t first, uint32_t end, const float4* lo, const float4* hi, const uint2* child, float* cost,
                                             uint8_t* how, uint8_t* split)
        {
            for (uint32_t i = first + blockIdx.x * blockDim.x + threadIdx.x; i < end; i += gridDim.x * blockDim.x)
                collapse_node(i, lo, hi, child, cost, how, split);
        }

        // Rounds [firstRound, endRound) by one block, which is enough for their few nodes.
        __global__ void collapse_tail_kernel(const uint32_t* roundEnd, uint32_t firstRound, uint32_t endRound, const float4* lo, const float4* hi,
                                             const uint2* child, float* cost, uint8_t* how, uint8_t* split)
        {
            for (uint32_t r = firstRound; r < endRound; r++)
            {
                const uint32_t end = roundEnd[r + 1];
                for (uint32_t i = roundEnd[r] + threadIdx.x; i < end; i += blockDim.x) collapse_node(i, lo, hi, child, cost, how, split);
                __syncthreads();
            }
        }

        // Box padding of bvh8.cpp (WideBuilder::padBox).
        __device__ void pad_box(float4 lo, float4 hi, double dlo[3], double dhi[3])
        {
            const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
            float ext = 0.0f, mag = 0.0f;
            for (int k = 0; k < 3; k++)
            {
                ext = fmaxf(ext, h[k] - l[k]);
                mag = fmaxf(mag, fmaxf(fabsf(l[k]), fabsf(h[k])));
            }
            const double pad = 1e-5 * static_cast<double>(ext) + 1e-7 * static_cast<double>(mag) + 1e-30;
            for (int k = 0; k < 3; k++)
            {
                dlo[k] = static_cast<double>(l[k]) - pad;
                dhi[k] = static_cast<double>(h[k]) + pad;
            }
        }

        __device__ __forceinline__ uint32_t pack4(const uint8_t* q)
        {
            return static_cast<uint32_t>(q[0]) | (static_cast<uint32_t>(q[1]) << 8) | (static_cast<uint32_t>(q[2]) << 16) | (static_cast<uint32_t>(q[3]) << 24);
        }

        // One level of wide nodes: node `levelBase + w` is binary node level[w].x, its header belongs into
        // record level[w].y. Inner children get consecutive indices from *counter and enter nextLevel at
        // (index - nextBase); leaf child k (leaf position) gets its record in leafRecord[k]. Headers go to
        // headers[node], the header's record to headerRecord[node], the children's kinds to masks[node].
        // capacity: entries of these arrays and of nextLevel (an index beyond it is refused and reported).
        __global__ void emit_level_kernel(const uint2* level, uint32_t count, uint32_t levelBase, uint32_t nextBase, uint32_t n,
                                          const float4* lo, const float4* hi, const uint2* child, const uint8_t* how, const uint8_t* split,
                                          uint32_t* counter, uint2* nextLevel, Record8* headers, uint32_t* headerRecord, uint32_t* masks,
                                          uint32_t* leafRecord, uint32_t capacity, uint32_t* errorFlags)
        {
            for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < count; w += gridDim.x * blockDim.x)
            {
                const uint32_t b = level[w].x;
                uint32_t kids[8];
                bool kidLeaf[8];
                int nk = 0;
                if (b < n)
                {
                    kids[0] = b;
                    kidLeaf[0] = true;
                    nk = 1;
                }
                else
                {
                    // CollapsePlan::children / collect, left before right
                    uint32_t stNode[kCollectStack];
                    uint8_t stSlots[kCollectStack];
                    int sp = 0;
                    const uint2 c = child[b];
                    const int s = split[b];
                    stNode[sp] = c.y;
                    stSlots[sp++] = static_cast<uint8_t>(8 - s);
                    stNode[sp] = c.x;
                    stSlots[sp++] = static_cast<uint8_t>(s);
                    bool bad = false;
                    while (sp > 0)
                    {
                        const uint32_t x = stNode[--sp];
                        const int i = stSlots[sp];
                        const uint8_t h = how[static_cast<size_t>(x) * 8 + i - 1];
                        if (i == 1)
                        {
                            if (nk >= 8)
                            {
                                bad = true;
                                break;
                            }
                            kids[nk] = x;
                            kidLeaf[nk] = h == 0;
                            nk++;
                        }
                        else if (h == 0)
                        {
                            stNode[sp] = x;
                            stSlots[sp++] = static_cast<uint8_t>(i - 1);
                        }
                        else
                        {
                            if (sp + 2 > kCollectStack)
                            {
                                bad = true;
                                break;
                            }
                            const uint2 cx = child[x];
                            stNode[sp] = cx.y;
                            stSlots[sp++] = static_cast<uint8_t>(i - h);
                            stNode[sp] = cx.x;
                            stSlots[sp++] = h;
                        }
                    }
                    if (bad)
                    {
                        atomicOr(errorFlags, kBuildErrCollect);
                        continue;
                    }
                }
                // slot assignment by octant (WideBuilder::emit)
                float4 nlo = lo[kids[0]], nhi = hi[kids[0]];
                for (int i = 1; i < nk; i++)
                {
                    nlo = fmin4(nlo, lo[kids[i]]);
                    nhi = fmax4(nhi, hi[kids[i]]);
                }
                const float center[3] = {0.5f * (nlo.x + nhi.x), 0.5f * (nlo.y + nhi.y), 0.5f * (nlo.z + nhi.z)};
                int slotOf[8] = {};
                bool slotUsed[8] = {}, kidUsed[8] = {};
                for (int round = 0; round < nk; round++)
                {
                    float bestScore = -FLT_MAX;
                    int bk = -1, bs = -1;
                    for (int i = 0; i < nk; i++)
                    {
                        if (kidUsed[i]) continue;
                        const float4 cl = lo[kids[i]], ch = hi[kids[i]];
                        const float v[3] = {0.5f * (cl.x + ch.x) - center[0], 0.5f * (cl.y + ch.y) - center[1], 0.5f * (cl.z + ch.z) - center[2]};
                        for (int s = 0; s < 8; s++)
                        {
                            if (slotUsed[s]) continue;
                            const float score = ((s & 1) ? v[0] : -v[0]) + ((s & 2) ? v[1] : -v[1]) + ((s & 4) ? v[2] : -v[2]);
                            if (score > bestScore)
                            {
                                bestScore = score;
                                bk = i;
                                bs = s;
                            }
                        }
                    }
                    kidUsed[bk] = true;
                    slotUsed[bs] = true;
                    slotOf[bk] = bs;
                }
                // the children's block; inner children take consecutive indices in the order of the child list
                int inner = 0;
                for (int i = 0; i < nk; i++) inner += kidLeaf[i] ? 0 : 1;
                const uint32_t firstInner = inner ? atomicAdd(counter, static_cast<uint32_t>(inner)) : 0u;
                const uint32_t block = levelBase + w + 1u;
                uint32_t innerMask = 0, leafMask = 0;
                int r = 0;
                for (int i = 0; i < nk; i++)
                {
                    const int s = slotOf[i];
                    const uint32_t record = block * kBlockRecords + static_cast<uint32_t>(s);
                    if (kidLeaf[i])
                    {
                        leafRecord[kids[i]] = record;
                        leafMask |= 1u << s;
                    }
                    else
                    {
                        const uint32_t at = firstInner + static_cast<uint32_t>(r++);
                        if (at < capacity && at >= nextBase) nextLevel[at - nextBase] = make_uint2(kids[i], record);
                        else atomicOr(errorFlags, kBuildErrCapacity);
                        innerMask |= 1u << s;
                    }
                }
                if (levelBase + w >= capacity)
                {
                    atomicOr(errorFlags, kBuildErrCapacity);
                    continue;
                }
                // quantisation (WideBuilder::emit): power-of-two scales, origin rounded down to a 24-bit multiple
                // of a power of two, every quantised box checked in double to contain its padded child box
                double clo[8][3], chi[8][3];
                bool valid[8] = {};
                double plo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, phi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
                for (int i = 0; i < nk; i++)
                {
                    const int s = slotOf[i];
                    pad_box(lo[kids[i]], hi[kids[i]], clo[s], chi[s]);
                    valid[s] = true;
                    for (int a = 0; a < 3; a++)
                    {
                        plo[a] = fmin(plo[a], clo[s][a]);
                        phi[a] = fmax(phi[a], chi[s][a]);
                    }
                }
                // origins: multiples of 2^unit that have 24 bits; scales within the header's range of the unit
                int32_t origin[3];
                int expo[3];
                uint8_t qlo[3][8], qhi[3][8];
                int unit = kMinUnit8;
                for (int a = 0; a < 3; a++)
                {
                    int fe;
                    frexp(fmax(fabs(plo[a]), 1e-300), &fe);
                    unit = max(unit, fe - 23);
                }
                bool overflow = false;
                for (int a = 0; a < 3;)
                {
                    const double grid = ldexp(1.0, unit);
                    const double q0 = floor(plo[a] / grid);
                    const double pf = q0 * grid;
                    const double ext = phi[a] - pf;
                    int e = unit - kScaleBelow8;
                    if (ext > 0.0)
                    {
                        int fe;
                        frexp(ext / 255.0, &fe);  // ext/255 = m * 2^fe, m in [0.5, 1)
                        e = max(e, min(127, fe));
                    }
                    bool fits = fabs(q0) <= static_cast<double>(kMaxOrigin8);
                    for (; fits; e++)
                    {
                        if (e > unit + kScaleAbove8 || e > 127)
                        {
                            fits = false;
                            break;
                        }
                        const double scale = ldexp(1.0, e);
                        bool ok = true;
                        for (int s = 0; s < 8 && ok; s++)
                        {
                            if (!valid[s])
                            {
                                qlo[a][s] = 255;
                                qhi[a][s] = 0;
                                continue;
                            }
                            double ql = floor((clo[s][a] - pf) / scale);
                            double qh = ceil((chi[s][a] - pf) / scale);
                            ql = fmax(0.0, ql);
                            while (ql > 0 && pf + ql * scale > clo[s][a]) ql -= 1.0;
                            while (pf + qh * scale < chi[s][a]) qh += 1.0;
                            if (qh > 255.0 || pf + ql * scale > clo[s][a])
                            {
                                ok = false;
                                break;
                            }
                            // (boxes of triangles without a number in their coordinates are inverted)
                            qlo[a][s] = static_cast<uint8_t>(fmin(ql, 255.0));
                            qhi[a][s] = static_cast<uint8_t>(fmax(qh, 0.0));
                        }
                        if (ok) break;
                    }
                    if (!fits)
                    {
                        // a coarser origin for all axes
                        unit++;
                        if (unit > 127)
                        {
                            overflow = true;
                            break;
                        }
                        a = 0;
                        continue;
                    }
                    origin[a] = static_cast<int32_t>(q0);
                    expo[a] = e - (unit - kScaleBelow8);
                    a++;
                }
                if (overflow)
                {
                    atomicOr(errorFlags, kBuildErrExponent);
                    continue;
                }
                Record8 node;
                const uint32_t ez = static_cast<uint32_t>(expo[2]);
                node.w[0] = make_uint4((static_cast<uint32_t>(origin[0]) << 8) | innerMask,
                                       (static_cast<uint32_t>(origin[1]) << 8) | static_cast<uint32_t>(unit + kUnitBias8),
                                       (static_cast<uint32_t>(origin[2]) << 8) | ((ez & 7u) << 5) | static_cast<uint32_t>(expo[0]),
                                       (block << 8) | ((ez >> 3) << 5) | static_cast<uint32_t>(expo[1]));
                node.w[1] = make_uint4(pack4(qlo[0]), pack4(qlo[0] + 4), pack4(qlo[1]), pack4(qlo[1] + 4));
                node.w[2] = make_uint4(pack4(qlo[2]), pack4(qlo[2] + 4), pack4(qhi[0]), pack4(qhi[0] + 4));
                node.w[3] = make_uint4(pack4(qhi[1]), pack4(qhi[1] + 4), pack4(qhi[2]), pack4(qhi[2] + 4));
                headers[levelBase + w] = node;
                headerRecord[levelBase + w] = level[w].y;
                masks[levelBase + w] = block_mask(innerMask, leafMask);
            }
        }

        // Triangle records (bvh8.cpp, WideBuilder::emit_leaf): (v0, input index), (e1, model), (e2, 0), 0;
        // leaf k is the k-th triangle of the sort.
        __global__ void triangle_records_kernel(const float* pos, const uint32_t* models, const uint32_t* sorted, const uint32_t* leafRecord,
                                                uint32_t n, Record8* records)
        {
            for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
            {
                const uint32_t t = sorted[k];
                const float* p = pos + static_cast<size_t>(t) * 9;
                float4* w = reinterpret_cast<float4*>(records[leafRecord[k]].w);
                w[0] = make_float4(p[0], p[1], p[2], __uint_as_float(t));
                w[1] = make_float4(p[3] - p[0], p[4] - p[1], p[5] - p[2], __uint_as_float(models[t]));
                w[2] = make_float4(p[6] - p[0], p[7] - p[1], p[8] - p[2], 0.0f);
            }
        }

        // Headers into their records, and the masks of the blocks (block 0: the root's header).
        __global__ void header_records_kernel(const Record8* headers, const uint32_t* headerRecord, const uint32_t* nodeMasks, uint32_t nodes,
                                              Record8* records, uint32_t* blockMasks)
        {
            for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nodes; j += gridDim.x * blockDim.x)
            {
                records[headerRecord[j]] = headers[j];
                blockMasks[j + 1u] = nodeMasks[j];
                if (j == 0) blockMasks[0] = block_mask(1u, 0u);
            }
        }

        uint32_t grid_for(uint32_t items, uint32_t threads, uint32_t cap = 65535u)
        {
            const uint32_t g = (items + threads - 1) / threads;
            return g < 1 ? 1 : (g > cap ? cap : g);
        }
    }

    Status BuildBvh8Device(const float* positions, const uint32_t* models, uint32_t n, cudaStream_t s, DeviceBvh& out)
    {
        if (n == 0) return Status::Err(GPT_ERR_INVALID_ARGUMENT, "BVH build failed: scene has no triangles");
        if (n > kMaxTriangles) return Status::Err(GPT_ERR_CAPACITY, "BVH build failed: scene has more than 2^24 triangles");
        const uint32_t nodes = 2 * n - 1;
        float4 *triLo, *triHi, *cent, *partLo, *partHi, *lo, *hi;
        uint32_t *keys, *keysSorted, *values, *sorted, *clustersA, *clustersB, *nn, *roundEnd, *counter, *errorFlags, *headerRecord, *nodeMasks, *leafRecord;
        unsigned long long *flags, *ranks;
        uint2 *child, *levelA, *levelB;
        float* cost;
        uint8_t *how, *split;
        char* temp;
        Record8* wide;
        PlocState* state;
        size_t sortBytes = 0, scanBytes = 0;
        PT_CUDA("cub::DeviceRadixSort::SortPairs", cub::DeviceRadixSort::SortPairs(nullptr, sortBytes, static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                                                                 static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr), static_cast<int>(n), 0, 30, s));
        PT_CUDA("cub::DeviceScan::ExclusiveSum", cub::DeviceScan::ExclusiveSum(nullptr, scanBytes, static_cast<unsigned long long*>(nullptr),
                                                                              static_cast<unsigned long long*>(nullptr), static_cast<int>(n + 1), s));
        const size_t tempBytes = sortBytes > scanBytes ? sortBytes : scanBytes;
        const uint32_t parts = grid_for(n, 256, 1024);
        // One allocation instead of 30 and their frees, three rounds per read of the count and one block for the
        // last rounds: 22.5 -> 4.9 ms for 1.3M triangles (34 rounds with more than kTailClusters clusters).
        DeviceArena arena;
        arena.add(triLo, n);
        arena.add(triHi, n);
        arena.add(cent, n);
        arena.add(partLo, parts);
        arena.add(partHi, parts);
        arena.add(keys, n);
        arena.add(keysSorted, n);
        arena.add(values, n);
        arena.add(sorted, n);
        arena.add(lo, nodes);
        arena.add(hi, nodes);
        arena.add(child, nodes);
        arena.add(clustersA, n);
        arena.add(clustersB, n);
        arena.add(nn, n);
        arena.add(flags, size_t(n) + 1);
        arena.add(ranks, size_t(n) + 1);
        arena.add(roundEnd, size_t(n) + 1);  // every round merges at least one pair
        arena.add(cost, size_t(nodes) * 8);
        arena.add(how, size_t(nodes) * 8);
        arena.add(split, nodes);
        arena.add(levelA, n);
        arena.add(levelB, n);
        arena.add(counter, 4);
        arena.add(errorFlags, 4);
        arena.add(state, 1);
        arena.add(wide, n);  // at most one wide node per binary inner node (one for n = 1)
        arena.add(headerRecord, n);
        arena.add(nodeMasks, n);
        arena.add(leafRecord, n);
        arena.add(temp, tempBytes);
        PT_TRY(arena.allocate());
        PT_CUDA("cudaMemsetAsync", cudaMemsetAsync(errorFlags, 0, 16, s));

        // 1-2: boxes, centroids, Morton order
        triangle_boxes_kernel<<<parts, 256, 0, s>>>(positions, n, triLo, triHi, cent, partLo, partHi);
        PT_CUDA("triangle boxes", cudaGetLastError());
        bounds_final_kernel<<<1, 256, 0, s>>>(partLo, partHi, parts);
        PT_CUDA("centroid bounds", cudaGetLastError());
        morton_kernel<<<grid_for(n, 256, 4096), 256, 0, s>>>(cent, n, partLo, partHi, keys, values);
        PT_CUDA("morton codes", cudaGetLastError());
        size_t tb = tempBytes;
        PT_CUDA("cub::DeviceRadixSort::SortPairs", cub::DeviceRadixSort::SortPairs(temp, tb, keys, keysSorted, values, sorted,
                                                                                 static_cast<int>(n), 0, 30, s));
        leaves_kernel<<<grid_for(n, 256, 4096), 256, 0, s>>>(sorted, n, triLo, triHi, lo, hi, child, clustersA);
        PT_CUDA("leaves", cudaGetLastError());

        // 3: clustering rounds
        PlocState now{n, n, 0, 0};
        PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(state, &now, sizeof(now), cudaMemcpyHostToDevice, s));
        PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(roundEnd, &n, 4, cudaMemcpyHostToDevice, s));
        uint32_t* cur = clustersA;
        uint32_t* nxt = clustersB;
        while (now.clusters > kTailClusters)
        {
            const uint32_t m = now.clusters;
            for (int r = 0; r < kRoundsPerSync; r++)
            {
                ploc_nearest_kernel<<<(m + kPlocBlock - 1) / kPlocBlock, kPlocBlock, 0, s>>>(cur, state, lo, hi, nn);
                PT_CUDA("nearest clusters", cudaGetLastError());
                ploc_flags_kernel<<<grid_for(m + 1, 256, 8192), 256, 0, s>>>(nn, state, m + 1, flags);
                PT_CUDA("cluster flags", cudaGetLastError());
                tb = tempBytes;
                PT_CUDA("cub::DeviceScan::ExclusiveSum", cub::DeviceScan::ExclusiveSum(temp, tb, flags, ranks, static_cast<int>(m + 1), s));
                ploc_merge_kernel<<<grid_for(m, 256, 8192), 256, 0, s>>>(cur, state, nn, flags, ranks, lo, hi, child, nxt);
                PT_CUDA("cluster merge", cudaGetLastError());
                ploc_advance_kernel<<<1, 1, 0, s>>>(state, ranks, roundEnd);
                PT_CUDA("clustering round", cudaGetLastError());
                std::swap(cur, nxt);
            }
            PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(&now, state, sizeof(now), cudaMemcpyDeviceToHost, s));
            PT_CUDA("cudaStreamSynchronize", cudaStreamSynchronize(s));
            if (now.stalled) return Status::Err(GPT_ERR_DEVICE_FAULT, "BVH build failed: a clustering round merged no pair");
        }
        const uint32_t largeRounds = now.rounds;
        ploc_tail_kernel<<<1, kTailClusters, 2 * kTailClusters * sizeof(float4), s>>>(cur, state, lo, hi, child, roundEnd);
        PT_CUDA("last clustering rounds", cudaGetLastError());
        std::vector<uint32_t> rounds(largeRounds + 1);
        PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(rounds.data(), roundEnd, rounds.size() * 4, cudaMemcpyDeviceToHost, s));
        PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(&now, state, sizeof(now), cudaMemcpyDeviceToHost, s));
        PT_CUDA("cudaStreamSynchronize", cudaStreamSynchronize(s));
        if (now.stalled) return Status::Err(GPT_ERR_DEVICE_FAULT, "BVH build failed: a clustering round merged no pair");
        if (now.clusters != 1 || now.nodes != nodes) return Status::Err(GPT_ERR_DEVICE_FAULT, "BVH build failed: clustering left the wrong number of nodes");
        const uint32_t root = nodes - 1;

        // 4: collapse costs, one round at a time (children before parents)
        collapse_leaf_kernel<<<grid_for(n, 256, 8192), 256, 0, s>>>(n, lo, hi, cost, how);
        PT_CUDA("collapse leaves", cudaGetLastError());
        for (uint32_t r = 0; r < largeRounds; r++)
        {
            const uint32_t a = rounds[r], b = rounds[r + 1];
            collapse_node_kernel<<<grid_for(b - a, 128, 8192), 128, 0, s>>>(a, b, lo, hi, child, cost, how, split);
            PT_CUDA("collapse nodes", cudaGetLastError());
        }
        if (now.rounds > largeRounds)
        {
            collapse_tail_kernel<<<1, kTailClusters / 2, 0, s>>>(roundEnd, largeRounds, now.rounds, lo, hi, child, cost, how, split);
            PT_CUDA("collapse nodes", cudaGetLastError());
        }

        // 5: wide nodes level by level
        const uint32_t one = 1;
        const uint2 rootLevel = make_uint2(root, 0u);  // the root's header: record 0
        PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(levelA, &rootLevel, sizeof(rootLevel), cudaMemcpyHostToDevice, s));
        PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(counter, &one, 4, cudaMemcpyHostToDevice, s));
        uint32_t levelBase = 0, count = 1, depth = 0, allocated = 1;
        uint2* level = levelA;
        uint2* nextLevel = levelB;
        while (count > 0)
        {
            depth++;
            if (depth > kMaxStack) return Status::Err(GPT_ERR_CAPACITY, "BVH8 deeper than the traversal stack");
            emit_level_kernel<<<grid_for(count, 128, 16384), 128, 0, s>>>(level, count, levelBase, levelBase + count, n, lo, hi, child, how, split,
                                                                          counter, nextLevel, wide, headerRecord, nodeMasks, leafRecord, n,
                                                                          errorFlags);
            PT_CUDA("wide nodes", cudaGetLastError());
            uint32_t levelFlags = 0;
            PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(&allocated, counter, 4, cudaMemcpyDeviceToHost, s));
            PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(&levelFlags, errorFlags, 4, cudaMemcpyDeviceToHost, s));
            PT_CUDA("cudaStreamSynchronize", cudaStreamSynchronize(s));
            if (allocated > n) return Status::Err(GPT_ERR_DEVICE_FAULT, "BVH build failed: more wide nodes than the bound");
            if (levelFlags) break;  // reported below; the next level's list is incomplete
            levelBase += count;
            count = allocated - levelBase;
            std::swap(level, nextLevel);
        }
        uint32_t failed = 0;
        PT_CUDA("cudaMemcpy", cudaMemcpy(&failed, errorFlags, 4, cudaMemcpyDeviceToHost));
        if (failed & kBuildErrExponent) return Status::Err(GPT_ERR_INVALID_ARGUMENT, "BVH build failed: BVH quantisation exponent overflow");
        if (failed & kBuildErrCapacity) return Status::Err(GPT_ERR_DEVICE_FAULT, "BVH build failed: a wide-node index beyond the node array");
        if (failed) return Status::Err(GPT_ERR_DEVICE_FAULT, "BVH build failed: a wide node's child list did not fit");
        if (allocated >= kMaxBlocks) return Status::Err(GPT_ERR_CAPACITY, "BVH8 has more than 2^24 nodes");

        // 6: the child blocks (empty slots stay zero)
        out.blockCount = allocated + 1u;
        const size_t blockBytes = size_t(out.blockCount) * kBlockRecords * sizeof(Record8);
        PT_TRY(out.blocks.allocate(blockBytes));
        PT_TRY(out.blockMasks.allocate(size_t(out.blockCount) * 4));
        PT_CUDA("cudaMemsetAsync", cudaMemsetAsync(out.blocks.get<void>(), 0, blockBytes, s));
        triangle_records_kernel<<<grid_for(n, 256, 8192), 256, 0, s>>>(positions, models, sorted, leafRecord, n, out.blocks.get<Record8>());
        PT_CUDA("triangle records", cudaGetLastError());
        header_records_kernel<<<grid_for(allocated, 256, 8192), 256, 0, s>>>(wide, headerRecord, nodeMasks, allocated, out.blocks.get<Record8>(),
                                                                             out.blockMasks.get<uint32_t>());
        PT_CUDA("header records", cudaGetLastError());
        PT_CUDA("cudaStreamSynchronize", cudaStreamSynchronize(s));
        out.nodeCount = allocated;
        out.depth = depth;
        out.binaryNodes = nodes;
        out.rounds = now.rounds;
        return Status::Ok();
    }
}
