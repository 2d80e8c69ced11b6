// Host construction of the BVH8 (see bvh8.cpp).
#pragma once
#include <cstdint>
#include <vector>

#include "pt_internal.h"

namespace pt
{
    struct Bvh8
    {
        std::vector<Record8> records;  // kBlockRecords per block
        std::vector<uint32_t> masks;   // per block: block_mask of what its slots hold
        uint32_t nodeCount = 0;        // wide nodes
        uint32_t depth = 0;            // levels of the wide tree
        std::vector<Node2> nodes2;     // the binary tree the BVH8 is collapsed from, FP32 boxes (leaves in the same records)
        uint32_t depth2 = 0;           // levels of the binary tree
    };

    // positions: [n][3][3] world positions; models: shading model per triangle. withBinary: also
    // flatten the binary tree into FP32 Node2 records (nodes2, depth2).
    Bvh8 BuildBvh8(const float* positions, const uint32_t* models, uint32_t n, int threads, bool withBinary = false);

    struct Bvh8Check
    {
        uint64_t containmentViolations;  // quantised child boxes not containing their subtree (exact arithmetic)
        uint64_t trianglesNotExactlyOnce;
        uint64_t leafTriangles;
    };

    // Structural validation of a built BVH8 on the host.
    Bvh8Check CheckBvh8(const Bvh8& bvh, const float* positions, uint32_t n);
}
