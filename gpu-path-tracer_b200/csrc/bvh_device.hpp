// Device construction of the BVH8 (see bvh_device.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "runtime.hpp"

namespace pt
{
    struct DeviceBvh
    {
        DeviceBuffer blocks;       // kBlockRecords records per block, the root's block first
        DeviceBuffer blockMasks;   // uint32 per block: block_mask of what its slots hold
        uint32_t nodeCount = 0;
        uint32_t blockCount = 0;
        uint32_t depth = 0;        // levels of the wide tree
        uint32_t binaryNodes = 0;  // nodes of the clustered binary tree
        uint32_t rounds = 0;       // clustering rounds
    };

    // positions: device [n][3][3] world positions; models: device shading model per triangle (input
    // order). Builds on stream s and returns once the result is complete.
    Status BuildBvh8Device(const float* positions, const uint32_t* models, uint32_t n, cudaStream_t s, DeviceBvh& out);
}
