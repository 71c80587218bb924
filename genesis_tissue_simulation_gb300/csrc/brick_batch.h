// Batched instances on bricks (brick_batch.cu).
#pragma once
#include <vector>

#include "brick_kernels.h"

namespace gbt {

// One instance of a batch as the planner sees it: its own coloured mesh, the first of its nodes in the
// packed table, and where its colour slots went there.
struct BatchBrickInstance {
    BrickMesh mesh;
    int nodeBase;
    const int* edgeSlot;             // [E] packed slot of the instance's colour slot
    const int* tetSlot;              // [T]
    const unsigned char* edgeDead;   // [E], [T] elements that no frame projects
    const unsigned char* tetDead;
};

// The frame kernel: perType, one compliance per instance and Kuhn type (instAlpha [6 x instances]); else
// the tables' tetAlpha.
using BrickBatchKernel = void (*)(DeviceMesh m, FrameCoeffs fc, ContactParams cp, BrickTables bt, const BrickShape* shapes, const int* order,
                                  const int* start, const float2* instAlpha, unsigned* status);

// The bricks of a batch and their CTAs.  CTA c serves the bricks order[start[c]] .. order[start[c + 1] - 1]
// one after another; a brick that exchanges with others is always its CTA's first, so all of them run
// at the same time (the launch is cooperative).
// Below this many tets an SM the instances of a batch (no more than SMs) are spread over all SMs: a colour of one
// CTA is then shorter than its latency.  ms a frame of 10 substeps, spread and not: 600 tets an SM (12 instances) 0.40
// and 0.44, 2,200 (152) 0.90 and 1.15, 5,200 (152) 1.20 and 1.25, 7,700 (100) 1.22 and 1.40, 8,200 (152) 1.54 and 1.46,
// 12,200 (152) 2.10 and 1.70, 17,300 (152) 2.80 and 1.95.  With fewer instances spreading pays a little longer (100 with
// 14,800: 1.65 and 1.91; 60 with 8,700: 1.13 and 1.18).
constexpr int kSplitTets = 8000;
constexpr int kSplitThreads = 384;

struct BatchBricks {
    BrickBuffers buffers;
    BrickShape* shapes = nullptr;
    int* order = nullptr; int* start = nullptr;
    int ctas = 0, threads = 0; size_t bytes = 0;
    int bound = 0;   // threads the kernel is compiled for
    BrickBatchKernel kernel(bool damped, bool perType) const;
    bool ready() const { return ctas > 0; }
    void release();
    // Plans every instance; not ready when one does not fit.  maxBytes: shared memory of one CTA.
    cudaError_t plan(const std::vector<BatchBrickInstance>& instances, int N, int smCount, int maxBytes, bool damped,
                     cudaStream_t stream);
};

}  // namespace gbt
