// Brick frame of a single mesh (brick_kernels.cu) and the device side of a brick plan.
#pragma once
#include <new>

#include "brick_frame.cuh"

namespace gbt {

// The frame kernel; cut: with the blade's ribbon tick between substeps.  `state` as for the other frame
// kernels ([1] and [2] zero; the exchanges run are left in [1] without a cut, the frame parity in [3]).
using BrickFrameKernel = void (*)(DeviceMesh m, FrameCoeffs fc, ToolPose from, ToolPose to, ContactParams cp, BrickTables bt, CutParams cu,
                                  unsigned* state);
// extended: the tissue guard and contact model 1 (no cut).
BrickFrameKernel brickFrameKernelFor(bool damped, bool cut, bool extended, int threads);

// A plan's tables on the device.
struct BrickBuffers {
    BrickTables t{};
    int tets = 0, edges = 0, threads = kBrickThreads;
    int asked = 0;   // bricks the plan was asked for
    // The live bits are those of the current topology: false from upload() to the first refresh(), and set
    // false by whoever changes the topology without writing these tables' bits.
    bool current = false;
    int* tetSrc = nullptr; int* edgeSrc = nullptr;
    // Uploads `plan` (of a mesh of N nodes) on `stream`, for CTAs of at most maxBytes shared memory;
    // frees what was there, and leaves nothing ready when it fails.
    cudaError_t upload(const BrickPlan& plan, int N, bool damped, int maxBytes, cudaStream_t stream);
    void release();
    bool ready() const { return t.bricks > 0; }
    size_t sharedBytes(bool damped) const { return Brick::bytes(t, damped); }
    static size_t leastBytes(const BrickPlan& plan, bool damped);   // of a CTA that reads its exchange lists from device memory
    // Live bits from the mesh's flags (`flags`: edgeLive, edgeSupport with fallback, tetMeta are current).
    cudaError_t refresh(const DeviceMesh& m, bool fallback, cudaStream_t stream);
    // Compliances over h^2 of the bricks' tets from the per-tet stiffnesses.
    cudaError_t compliances(float invH2, const float2* tetStiff, cudaStream_t stream);
private:
    void* memory_ = nullptr;   // one allocation for every table
};

// Makes a plan and its tables by `make` (a cudaError_t function of no arguments that may throw).  Bricks are
// a faster way to run a frame, not a condition of it: when host or device memory does not suffice the
// buffers are empty, as for a mesh without a plan, and the call goes on without them.
template <class Buffers, class Make> cudaError_t makeBricks(Buffers& buffers, Make&& make) {
    cudaError_t e;
    try { e = make(); } catch (const std::bad_alloc&) { e = cudaErrorMemoryAllocation; }
    if (e == cudaSuccess) return e;
    buffers.release();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();   // the failed allocation is dealt with
    return cudaSuccess;
}
#ifdef GBT_DEBUG_BOUNDS
extern int failBrickTables;   // this many table allocations to come answer that there is no memory (tests)
#endif

// Liveness flags of every edge and tet, the edges a live tet carries (with fallback: edgeSupport must
// be zero), and the nodes' inverse masses, from the current topology.
cudaError_t refreshMeshFlags(const DeviceMesh& m, int E, int T, bool fallback, cudaStream_t stream);

}  // namespace gbt
