// One frame of a single mesh on spatial bricks (brick_frame.cuh), and the upkeep of a plan's tables.
#include <type_traits>

#include "brick_kernels.h"
#include "contact_point.cuh"
#include "friction_contact.cuh"
#include "guard_feasible.cuh"
#include "particle_frame.cuh"
#include "ribbon_tick.cuh"

namespace gbt {
namespace {

// A node no element touches through substeps [s0, s1), as the brick's node phases treat its own.
template <bool Extended>
__device__ __noinline__ void idleNode(const DeviceMesh& m, int n, const FrameCoeffs& fc, const ToolPose& from, const ToolPose& to, const ContactParams& cp,
                         int s0, int s1) {
    float4 P = m.pos[n], Q = P;
    f3 V = xyz(m.vel[n]);
    if (!(P.w > 0.f)) {
        m.prev[n] = make_float4(P.x, P.y, P.z, 0.f);
        m.vel[n] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const float4 F = m.ext[n];
    const f3 a = mk(F.x, F.y, F.z) * P.w;
    for (int s = s0; s < s1; s++) {
        Q = P;
        V = V + a * fc.h;
        f3 x = xyz(P) + V * fc.h;
        const float t = fminf(1.f, (float)(fc.firstSubstep + s + 1) / (float)fc.numSubsteps);
        if (Extended && fc.friction) {
            const FrictionShapes shapes = frictionShapes(from, to, t, fmaxf(0.f, t - 1.f / (float)fc.numSubsteps), fc.jawThickness, cp.jawGapClosed);
            x = frictionPoint(x, xyz(Q), P.w, shapes, fc.contactRadius, fc.contactAlphaH2, fc.muS, fc.muD);
        }
        if (fc.contact) {
            x = contactPoint(x, P.w, V, contactFrame(from, to, t, cp, fc.contactAlphaH2), cp);
        }
        P = make_float4(x.x, x.y, x.z, P.w);
        V = ((x - xyz(Q)) * fc.invH) * fc.velScale;
    }
    m.pos[n] = P;
    m.prev[n] = make_float4(Q.x, Q.y, Q.z, 0.f);
    m.vel[n] = make_float4(V.x, V.y, V.z, 0.f);
}

// The ribbon tick after a substep of a blade frame: the crossing test of the edges near the blade over
// the whole grid, then the live bits of this brick's elements where links were severed, then fresh
// particle frames where cut points were emitted (not after the frame's last substep).  Positions and
// substep-start positions are in device memory.  Out of line: a tick is a few microseconds of the
// substep, and its registers stay out of the sweep's.  False when a barrier timed out.
struct TickState { unsigned derivedAt; int rotParity; unsigned target; bool ok; };
__device__ __noinline__ TickState ribbonTick(const DeviceMesh& m, const CutParams& cu, const BrickTables& bt, int e0, int e1, int t0, int t1,
                                             bool lastSubstep, bool rotations, unsigned* barrier, long long budget, TickState ts) {
    GridSync grid{barrier, barrier + 1, gridDim.x, ts.target, budget, 0u};
    ts.ok = false;
    const int r = grid.spreadRank(), R = grid.size();
    const unsigned pointsBefore = *(volatile unsigned*)(cu.counters + 1);
    if (!grid.sync()) return ts;
    const float* rot = rotations ? m.particleRot[ts.rotParity] : nullptr;
    if (cu.brickList && cu.tearLen2 <= 0.f) {
        const int nb = ((m.dx + kBrick - 1) / kBrick) * ((m.dy + kBrick - 1) / kBrick) * ((m.dz + kBrick - 1) / kBrick);
        for (int k = r >> 5; k < nb; k += R >> 5) brickBounds(m, cu, k, r & 31);
        if (!grid.sync()) return ts;
        const int listed = min((int)*(volatile unsigned*)cu.brickCount, nb);
        for (int j = r; j < listed * kBrickEdges; j += R) {
            int4 g;
            if (brickEdge(m, *(volatile int*)(cu.brickList + j / kBrickEdges), j % kBrickEdges, g)) tickEdgeAt(m, cu, g, true, rot);
        }
    } else {
        for (int e = r; e < cu.nGridEdges; e += R) tickEdge(m, cu, e, true, rot);
    }
    if (!grid.sync()) return ts;
    if (grid.leader() && cu.brickCount) *cu.brickCount = 0u;   // every reader has passed the barrier above
    const unsigned revision = *(volatile unsigned*)cu.counters;
    if (revision != ts.derivedAt) {
        ts.derivedAt = revision;
        unsigned* edgeWord = (unsigned*)bt.edgeWord;
        unsigned long long* tetWord = (unsigned long long*)bt.tetWord;
        for (int k = e0 + threadIdx.x; k < e1; k += blockDim.x) {
            const int e = checkRange(bt.bounds, bt.edgeSrc[k], 0, bt.meshEdges, kSiteBrickSource);
            const int2 ij = m.edgeEnds[e];
            const bool live = m.nbr[checkSlot(m, m.edgeOwner[e], kSiteEdgeSlot)] >= 0 && m.active[ij.x] != 0 && m.active[ij.y] != 0;
            edgeWord[k] = (edgeWord[k] & ~kBrickEdgeLive) | (live ? kBrickEdgeLive : 0u);
        }
        for (int k = t0 + threadIdx.x; k < t1; k += blockDim.x) {
            const int t = checkRange(bt.bounds, bt.tetSrc[k], 0, bt.meshTets, kSiteBrickSource);
            const int4 d = m.tetIds[t];
            const int* o = m.tetOwner + 3 * t;
            const bool live = m.nbr[checkSlot(m, o[0], kSiteTetSlot)] >= 0 && m.nbr[checkSlot(m, o[1], kSiteTetSlot)] >= 0 &&
                              m.nbr[checkSlot(m, o[2], kSiteTetSlot)] >= 0 && m.active[d.x] != 0 && m.active[d.y] != 0 && m.active[d.z] != 0 && m.active[d.w] != 0;
            tetWord[k] = (tetWord[k] & ~kBrickTetLive) | (live ? kBrickTetLive : 0ull);
        }
    }
    if (rotations && !lastSubstep && *(volatile unsigned*)(cu.counters + 1) != pointsBefore) {
        for (int i = m.nodeBase + r; i < m.nodeBase + m.nNodes; i += R)
            particleFrame(i, m.pos, m.nbr, m.active, m.pinned, m.particleRot[ts.rotParity], m.particleRot[ts.rotParity ^ 1]);
        ts.rotParity ^= 1;
        if (!grid.sync()) return ts;
    }
    __syncthreads();   // the live bits before the next sweep reads them
    ts.target = grid.target;
    ts.ok = true;
    return ts;
}

// The guard's slow path, when some tet is below the minimum volume: the feasibility chain on the node
// state in device memory, over the whole grid.
struct GuardResult { unsigned target; bool ok; };
__device__ __noinline__ GuardResult guardChain(const DeviceMesh& m, const FrameCoeffs& fc, int substepIndex, unsigned* barrier, unsigned target) {
    GridSync grid{barrier, barrier + 1, gridDim.x, target, fc.spinBudget, 0u};
    GuardResult g{target, false};
    if (grid.sync() && guardFeasible(m, fc, substepIndex, grid)) g.ok = true;
    g.target = grid.target;
    return g;
}

// Extended: the tissue guard and contact model 1 are compiled in.
template <bool Damped, bool Cut, bool Extended>
__device__ __forceinline__ void brickFrame(const DeviceMesh& m, const FrameCoeffs& fc, const ToolPose& from, const ToolPose& to,
                                           const ContactParams& cp, const BrickTables& bt, const CutParams& cu, unsigned* state) {
    extern __shared__ float4 shared[];
    const int tid = threadIdx.x, T = blockDim.x;
    const bool guarded = Extended && fc.guarded != 0;
    const int exchanges = bt.bricks > 1 ? fc.substeps * (bt.shape.stages + (guarded ? 1 : 0)) : 0;
    __shared__ FrictionShapes shapes[Extended ? kBrickFrames : 1];
    __shared__ float fibres[Extended ? 36 : 1];
    Brick b(bt, bt.shape, m.typeB, blockIdx.x, shared, Damped, true, exchanges, state + 2, fc.spinBudget, fc.syncTestExtra > 0 ? 1u << 30 : 0u);
    const bool stamp = fc.phaseClock != nullptr && blockIdx.x == 0 && tid == 0;
    int s = 0, slot = 0;
    auto mark = [&](unsigned tag) {
        if (stamp && slot < kPhaseRecordsPerSubstep) {
            unsigned long long ns;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(ns));
            fc.phaseClock[(size_t)s * kPhaseRecordsPerSubstep + slot++] = ((unsigned long long)tag << 56) | (ns & 0x00FFFFFFFFFFFFFFull);
        }
    };
    b.loadState(m.pos, m.vel, m.ext);
    TickState ts{Cut ? *(volatile unsigned*)cu.counters : 0u, fc.rotParity, 0u, true};
    bool havePrev = cu.havePrev != 0;
    if (Extended)   // rest lengths of the six corner-to-corner fibres of every Kuhn type (a CTA may have fewer threads)
        for (int i = tid; i < 36; i += T) {
            f3 r[3];
            typeRows(m, i / 6, r);
            fibres[i] = fibreRest(r, i % 6);
        }
    b.fibres = fibres;
    for (; s < fc.substeps; s++) {
        slot = 0;
        mark(kPhaseFrameStart);
        if (fc.contact && s % kBrickFrames == 0) {
            __syncthreads();
            if (tid < kBrickFrames && s + tid < fc.substeps) {
                const float t = fminf(1.f, (float)(fc.firstSubstep + s + tid + 1) / (float)fc.numSubsteps);
                b.frames[tid] = contactFrame(from, to, t, cp, fc.contactAlphaH2);
            }
        }
        if (Extended && fc.friction && s % kBrickFrames == 0) {
            __syncthreads();
            if (tid < kBrickFrames && s + tid < fc.substeps) {
                const float t = fminf(1.f, (float)(fc.firstSubstep + s + tid + 1) / (float)fc.numSubsteps);
                shapes[tid] = frictionShapes(from, to, t, fmaxf(0.f, t - 1.f / (float)fc.numSubsteps), fc.jawThickness, cp.jawGapClosed);
            }
        }
        for (int i = tid; i < b.d.nOwned; i += T) {
            float4 P = b.P[i];
            b.Q[i] = make_float4(P.x, P.y, P.z, 0.f);
            if (P.w > 0.f) {
                const f3 v = xyz(b.V[i]) + xyz(b.A[i]) * fc.h;
                b.V[i] = make_float4(v.x, v.y, v.z, 0.f);
                const f3 x = xyz(P) + v * fc.h;
                b.P[i] = make_float4(x.x, x.y, x.z, P.w);
            }
        }
        mark(kPhasePredict);
        if (!b.sweep<Damped, false, false, Extended>(fc, [&](bool edges) { mark(edges ? kPhaseEdges : kPhaseTets); })) return;
        if (Extended && (fc.friction || guarded)) {   // contact, then the guard's feasibility test
            for (int i = tid; i < b.d.nOwned; i += T) {
                const float4 P = b.P[i];
                if (!(P.w > 0.f)) continue;
                f3 p = xyz(P);
                if (fc.friction) p = frictionPoint(p, xyz(b.Q[i]), P.w, shapes[s % kBrickFrames], fc.contactRadius, fc.contactAlphaH2, fc.muS, fc.muD);
                if (guarded && fc.contact) p = contactPoint(p, P.w, xyz(b.V[i]), b.frames[s % kBrickFrames], cp);
                b.P[i] = make_float4(p.x, p.y, p.z, P.w);
            }
            __syncthreads();
        }
        if (guarded) {
            if (bt.bricks > 1 && !b.exchange(0, false)) return;   // the whole halo: every owned tet's nodes
            // one of three words in turn: a word is cleared while every brick is between its last read and
            // its next write
            unsigned* flag = m.guardFlags + 2;
            if (b.belowMinimum(fc.minVolume)) flag[s % 3] = 1u;
            GridSync grid{state + 1, state + 2, gridDim.x, ts.target, fc.spinBudget, 0u};
            if (!grid.sync()) return;
            ts.target = grid.target;
            const bool repair = *(volatile unsigned*)(flag + s % 3) != 0u;
            if (grid.leader()) flag[(s + 2) % 3] = 0u;   // read before this barrier, written after the next
            if (repair) {
                for (int i = tid; i < b.d.nOwned; i += T) {
                    const int n = b.node(i);
                    m.pos[n] = b.P[i];
                    m.prev[n] = b.Q[i];
                }
                const GuardResult g = guardChain(m, fc, fc.firstSubstep + s + 1, state + 1, ts.target);
                ts.target = g.target;
                if (!g.ok) return;
                for (int i = tid; i < b.d.nOwned; i += T) b.P[i] = m.pos[b.node(i)];
            }
        }
        for (int i = tid; i < b.d.nOwned; i += T) {
            float4 P = b.P[i];
            f3 v = mk(0.f, 0.f, 0.f);
            if (P.w > 0.f) {
                if (fc.contact && !guarded) {
                    const f3 p = contactPoint(xyz(P), P.w, xyz(b.V[i]), b.frames[s % kBrickFrames], cp);
                    P = make_float4(p.x, p.y, p.z, P.w);
                    b.P[i] = P;
                }
                v = ((xyz(P) - xyz(b.Q[i])) * fc.invH) * fc.velScale;
            }
            b.V[i] = make_float4(v.x, v.y, v.z, 0.f);
        }
        mark(kPhaseVelocity);
        if (Cut) {   // the first tick after the blade is set only takes the position snapshot
            if (havePrev) {
                for (int i = tid; i < b.d.nOwned; i += T) {
                    const int n = b.node(i);
                    m.pos[n] = b.P[i];
                    m.prev[n] = b.Q[i];
                }
                for (int i = blockIdx.x * T + tid; i < bt.nIdle; i += gridDim.x * T) idleNode<Extended>(m, checkNode(m, bt.idle[i], kSiteBrickNode), fc, from, to, cp, s, s + 1);
                ts = ribbonTick(m, cu, bt, b.edgeOff[0], b.edgeOff[b.s.nE], b.tetOff[0], b.tetOff[b.s.nT],
                                fc.firstSubstep + s + 1 >= fc.numSubsteps, fc.rotations != 0, state + 1, fc.spinBudget, ts);
                if (!ts.ok) return;
                mark(kPhaseTick);
            } else {
                for (int i = blockIdx.x * T + tid; i < bt.nIdle; i += gridDim.x * T) idleNode<Extended>(m, checkNode(m, bt.idle[i], kSiteBrickNode), fc, from, to, cp, s, s + 1);
            }
            havePrev = true;
        }
    }
    for (int i = tid; i < b.d.nOwned; i += T) {
        const int n = b.node(i);
        m.pos[n] = b.P[i];
        m.prev[n] = b.Q[i];
        m.vel[n] = b.V[i];
    }
    if (!Cut)
        for (int i = blockIdx.x * T + tid; i < bt.nIdle; i += gridDim.x * T) idleNode<Extended>(m, checkNode(m, bt.idle[i], kSiteBrickNode), fc, from, to, cp, 0, fc.substeps);
    if (blockIdx.x == 0 && tid == 0) {
        if (!Cut && !guarded) state[1] = (unsigned)exchanges;   // with ticks or the guard it is the grid barrier's counter, which others may still read
        state[3] = (unsigned)ts.rotParity;
    }
}

__global__ void meshFlagsKernel(DeviceMesh m, int E, int T, int fallback) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < E) refreshEdge(m, i);
    if (i < T) {
        refreshTet(m, i);
        if (fallback && (m.tetMeta[i] & 8))
            for (int o = 0; o < 3; o++) m.edgeSupport[checkSlot(m, m.tetOwner[3 * i + o], kSiteTetSlot)] = 1;
    }
    if (i < m.nNodes) m.pos[i].w = nodeInvMass(m, i);
}

__global__ void brickLiveKernel(DeviceMesh m, int meshEdges, int edges, const int* edgeSrc, unsigned* edgeWord, int meshTets, int tets,
                                const int* tetSrc, unsigned long long* tetWord, int fallback) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < edges) {
        const int e = checkRange(m.bounds, edgeSrc[i], 0, meshEdges, kSiteBrickSource);
        const bool live = m.edgeLive[e] != 0 && !(fallback && m.edgeSupport[checkSlot(m, m.edgeOwner[e], kSiteEdgeSlot)]);
        edgeWord[i] = (edgeWord[i] & ~kBrickEdgeLive) | (live ? kBrickEdgeLive : 0u);
    }
    if (i < tets) tetWord[i] = (tetWord[i] & ~kBrickTetLive) | ((m.tetMeta[checkRange(m.bounds, tetSrc[i], 0, meshTets, kSiteBrickSource)] & 8) ? kBrickTetLive : 0ull);
}

__global__ void brickAlphaKernel(int tets, const int* tetSrc, float invH2, const float2* stiff, float2* alpha) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < tets) { const float2 s = stiff[tetSrc[i]]; alpha[i] = make_float2(invH2 / s.x, invH2 / s.y); }
}

}  // namespace

template <bool Damped, bool Cut, bool Extended, int Threads>
static __global__ void __launch_bounds__(Threads, 1)
brickFrameKernel(const __grid_constant__ DeviceMesh m, const __grid_constant__ FrameCoeffs fc, const __grid_constant__ ToolPose from,
                 const __grid_constant__ ToolPose to, const __grid_constant__ ContactParams cp, const __grid_constant__ BrickTables bt,
                 const __grid_constant__ CutParams cu, unsigned* state) {
    brickFrame<Damped, Cut, Extended>(m, fc, from, to, cp, bt, cu, state);
}
template <int Threads> static BrickFrameKernel frameKernelFor(bool damped, bool cut, bool extended) {
    if (extended) return damped ? brickFrameKernel<true, false, true, Threads> : brickFrameKernel<false, false, true, Threads>;
    return damped ? (cut ? brickFrameKernel<true, true, false, Threads> : brickFrameKernel<true, false, false, Threads>)
                  : (cut ? brickFrameKernel<false, true, false, Threads> : brickFrameKernel<false, false, false, Threads>);
}
BrickFrameKernel brickFrameKernelFor(bool damped, bool cut, bool extended, int threads) {
    return threads <= kNarrowThreads ? frameKernelFor<kNarrowThreads>(damped, cut, extended) : frameKernelFor<kBrickThreads>(damped, cut, extended);
}

#ifdef GBT_DEBUG_BOUNDS
int failBrickTables = 0;
#endif

void BrickBuffers::release() {
    if (memory_) cudaFree(memory_);
    memory_ = nullptr;
    t = BrickTables{};
    tets = edges = 0;
    current = false;
}

size_t BrickBuffers::leastBytes(const BrickPlan& plan, bool damped) {
    BrickTables q{};
    q.shape = plan.shape();
    q.maxLocal = plan.maxLocal; q.maxOwned = plan.maxOwned;
    return Brick::bytes(q, damped);
}

cudaError_t BrickBuffers::upload(const BrickPlan& plan, int N, bool damped, int maxBytes, cudaStream_t stream) {
    release();
    tets = (int)plan.tetWord.size(); edges = (int)plan.edgeWord.size();
    asked = plan.asked;
    threads = plan.tetWidth <= kNarrowColour ? (plan.threads < kNarrowThreads ? plan.threads : kNarrowThreads)
                                            : (plan.threads < kBrickThreads ? plan.threads : kBrickThreads);
    BrickTables q{};
    q.shape = plan.shape();
    q.maxLocal = plan.maxLocal; q.maxOwned = plan.maxOwned; q.nIdle = (int)plan.idle.size(); q.N = N;
    // every table in one allocation, 256-byte aligned: first pass sizes, second pass copies
    const size_t mail = plan.bricks > 1 ? 2 * (size_t)N : 0;
    char* base = nullptr;
    size_t at = 0;
    cudaError_t e = cudaSuccess;
    auto put = [&](auto** to, const void* from, size_t count) {   // from null: zeroed
        using T = std::remove_cv_t<std::remove_pointer_t<std::remove_pointer_t<decltype(to)>>>;
        const size_t bytes = count * sizeof(T);
        if (base && e == cudaSuccess) {
            *to = (T*)(base + at);
            if (bytes) e = from ? cudaMemcpyAsync(base + at, from, bytes, cudaMemcpyHostToDevice, stream) : cudaMemsetAsync(base + at, 0, bytes, stream);
        }
        at += (bytes + 255) & ~(size_t)255;
    };
    for (int pass = 0; pass < 2; pass++) {
        at = 0;
        put(&q.desc, plan.desc.data(), plan.desc.size());
        put(&q.head, plan.head.data(), plan.head.size());
        put(&q.localNode, plan.localNode.data(), plan.localNode.size());
        put(&q.idle, plan.idle.data(), plan.idle.size());
        put(&q.importList, plan.importList.data(), plan.importList.size());
        put(&q.exportList, plan.exportList.data(), plan.exportList.size());
        put(&q.tetWord, plan.tetWord.data(), plan.tetWord.size());
        put(&q.edgeWord, plan.edgeWord.data(), plan.edgeWord.size());
        put(&q.edgeRest, plan.edgeRest.data(), plan.edgeRest.size());
        put(&tetSrc, plan.tetSrc.data(), plan.tetSrc.size());
        put(&edgeSrc, plan.edgeSrc.data(), plan.edgeSrc.size());
        put(&q.ownTet, plan.ownTet.data(), plan.ownTet.size());
        put(&q.tetAlpha, nullptr, plan.tetWord.size());
        put(&q.mail, nullptr, mail);
        put(&q.mailStart, nullptr, damped ? mail : 0);
        put(&q.epoch, nullptr, plan.bricks);
        if (pass == 0) {
#ifdef GBT_DEBUG_BOUNDS
            if (failBrickTables > 0) { failBrickTables--; return cudaErrorMemoryAllocation; }
#endif
            e = cudaMalloc(&memory_, at ? at : 1);
            if (e != cudaSuccess) { memory_ = nullptr; return e; }
            base = (char*)memory_;
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);   // the plan's host tables may go
    if (e != cudaSuccess) { release(); return e; }
    q.tetSrc = tetSrc; q.edgeSrc = edgeSrc;
    q.meshEdges = plan.meshEdges; q.meshTets = plan.meshTets;
    q.bricks = plan.bricks;
    // the exchange lists, next to the node state, when shared memory holds both
    q.maxList = plan.maxList;
    q.listsShared = 1;
    if (Brick::bytes(q, damped) > (size_t)maxBytes) q.listsShared = 0;
    t = q;
    return cudaSuccess;
}

cudaError_t BrickBuffers::refresh(const DeviceMesh& m, bool fallback, cudaStream_t stream) {
    const int n = tets > edges ? tets : edges;
    if (n) brickLiveKernel<<<(n + 255) / 256, 256, 0, stream>>>(m, t.meshEdges, edges, edgeSrc, (unsigned*)t.edgeWord, t.meshTets, tets,
                                                               tetSrc, (unsigned long long*)t.tetWord, fallback ? 1 : 0);
    const cudaError_t e = cudaGetLastError();
    current = e == cudaSuccess;
    return e;
}

cudaError_t BrickBuffers::compliances(float invH2, const float2* tetStiff, cudaStream_t stream) {
    if (tets) brickAlphaKernel<<<(tets + 255) / 256, 256, 0, stream>>>(tets, tetSrc, invH2, tetStiff, (float2*)t.tetAlpha);
    return cudaGetLastError();
}

cudaError_t refreshMeshFlags(const DeviceMesh& m, int E, int T, bool fallback, cudaStream_t stream) {
    if (fallback) {
        const cudaError_t e = cudaMemsetAsync(m.edgeSupport, 0, (size_t)6 * m.nNodes * sizeof(int), stream);
        if (e != cudaSuccess) return e;
    }
    int n = E > T ? E : T;
    if (m.nNodes > n) n = m.nNodes;
    meshFlagsKernel<<<(n + 255) / 256, 256, 0, stream>>>(m, E, T, fallback ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace gbt
