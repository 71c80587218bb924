// The differentiable rollout's brick kernels (brick_rollout.cu).
#pragma once
#include "adjoint_kernels.h"
#include "brick_kernels.h"

namespace gbt {

// The reverse projection holds about 250 registers a thread.
constexpr int kReverseThreads = 256;

using BrickForwardKernel = void (*)(DeviceMesh m, DiffCoeffs dc, ContactParams cp, DiffBuffers b, BrickTables bt, unsigned* barrier,
                                    long long budget);
BrickForwardKernel brickForwardFor(bool damped, int threads);
__global__ void brickBackward(DeviceMesh m, DiffCoeffs dc, ContactParams cp, DiffBuffers b, BrickTables bt, BrickTables rt, unsigned* barrier,
                              long long budget);
__global__ void brickBackwardDamped(DeviceMesh m, DiffCoeffs dc, ContactParams cp, DiffBuffers b, BrickTables bt, BrickTables rt,
                                    unsigned* barrier, long long budget);

// Before a forward: live bits of the current topology, node state at the origin, compliances.
cudaError_t prepareRollout(const DeviceMesh& m, const DiffBuffers& b, int E, int T, float invH2, BrickBuffers& forward, BrickBuffers& reverse,
                           cudaStream_t stream);

}  // namespace gbt
