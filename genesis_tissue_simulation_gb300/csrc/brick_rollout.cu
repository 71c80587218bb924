// The differentiable rollout on spatial bricks (brick_frame.cuh): forward with checkpoints, and the
// backward's recompute and reverse sweep, in one launch each.
//
// The whole-GPU kernels (adjoint_kernels.cu) close each of the 37 colours of a substep, forward and
// reverse, with a grid barrier and gather through L2; here a brick's positions, and in reverse its
// nodes' adjoints, stay in shared memory between exchanges.  The reverse sweep runs the colours from
// last to first, so it has a plan of its own over the same bricks.  An element near a brick's faces is
// differentiated by several bricks for the node adjoints they need; the brick that owns the element's
// first node also records its tape and accumulates its own adjoints (compliance, rest shape), so each
// has one writer that adds in substep order.  The tape passes between bricks: one grid barrier stands
// between a segment's recompute and its reverse sweep, and one before the next segment overwrites it.
// 32 x 16 x 32 cells, 200 substeps: forward 20.1 -> 7.4 ms, forward and backward 75.5 -> 32.3 ms; bound by the
// reverse projection's dependent chain (~1.5 us a colour) on one or two warps a scheduler.
#include "brick_rollout.h"
#include "adjoint_rollout.cuh"

namespace gbt {
namespace {

// One substep from the state in `b`; with Record, tape slot j of the segment.
template <bool Damped, bool Record>
__device__ __forceinline__ bool rollSubstep(Brick& b, const FrameCoeffs& fc, const DiffCoeffs& dc, const ContactParams& cp,
                                            const DiffBuffers& db, int g, int N, int j, int nodes, int E, int T) {
    const int tid = threadIdx.x, step = blockDim.x;
    for (int i = tid; i < b.d.nOwned; i += step) {
        const float4 P = b.P[i];
        float4 V = b.V[i];
        b.Q[i] = make_float4(P.x, P.y, P.z, 0.f);
        if (P.w > 0.f) {
            const f3 v = xyz(V) + xyz(b.A[i]) * dc.h;
            V = make_float4(v.x, v.y, v.z, 0.f);
            b.V[i] = V;
            const f3 x = xyz(P) + v * dc.h;
            b.P[i] = make_float4(x.x, x.y, x.z, P.w);
        }
        if (Record) {
            const size_t at = (size_t)j * nodes + b.node(i);
            db.tapeQ[at] = P;
            db.tapeV[at] = V;
        }
    }
    const BrickTape tape{Record ? db.tapeEdge + 2 * (size_t)j * E : nullptr, Record ? db.tapeTet + 4 * (size_t)j * T : nullptr};
    if (!b.sweep<Damped, Record>(fc, [](bool) {}, tape)) return false;
    Capsule cap{};
    if (dc.contact) cap = capsuleAt(db, dc, g, N);
    for (int i = tid; i < b.d.nOwned; i += step) {
        const float4 P = b.P[i];
        if (Record) db.tapeX[(size_t)j * nodes + b.node(i)] = P;
        f3 x = xyz(P);
        if (dc.contact) x = capsuleContact(x, P.w, xyz(b.V[i]), cap, cp);
        b.P[i] = f4(x, P.w);
        f3 v = P.w > 0.f ? (x - xyz(b.Q[i])) * dc.invH : mk(0.f, 0.f, 0.f);
        v = P.w > 0.f ? v * dc.velScale : mk(0.f, 0.f, 0.f);
        b.V[i] = f4(v, 0.f);
    }
    return true;
}

__device__ __forceinline__ FrameCoeffs rollCoeffs(const DiffCoeffs& dc) {
    FrameCoeffs fc = frameCoeffs(dc);
    fc.doEdges = dc.doEdges; fc.doStrain = dc.doStrain;
    return fc;
}

template <bool Damped>
__device__ __forceinline__ void forwardBricks(const DeviceMesh& m, const DiffCoeffs& dc, const ContactParams& cp, const DiffBuffers& db,
                                              const BrickTables& bt, unsigned* barrier, long long budget) {
    extern __shared__ float4 shared[];
    const int N = db.total / db.frames, tid = threadIdx.x, step = blockDim.x;
    const FrameCoeffs fc = rollCoeffs(dc);
    Brick b(bt, bt.shape, m.typeB, blockIdx.x, shared, Damped, true, bt.bricks > 1 ? db.total * bt.shape.stages : 0, barrier + 1, budget, 0u);
    b.loadState(m.pos, m.vel, m.ext);
    for (int g = 0; g < db.total; g++) {
        if (g % db.every == 0) {
            const size_t base = (size_t)(g / db.every) * m.nNodes;
            for (int i = tid; i < b.d.nOwned; i += step) {
                const int n = b.node(i);
                db.ckPos[base + n] = b.P[i];
                db.ckVel[base + n] = b.V[i];
            }
        }
        if (!rollSubstep<Damped, false>(b, fc, dc, cp, db, g, N, 0, m.nNodes, 0, 0)) return;
    }
    for (int i = tid; i < b.d.nOwned; i += step) {
        const int n = b.node(i);
        m.pos[n] = b.P[i];
        m.prev[n] = make_float4(b.Q[i].x, b.Q[i].y, b.Q[i].z, 0.f);
        m.vel[n] = b.V[i];
    }
    for (int i = blockIdx.x * step + tid; i < bt.nIdle; i += gridDim.x * step) {   // idle nodes are immobile (checked by the host)
        const int n = checkNode(m, bt.idle[i], kSiteBrickNode);
        const float4 P = m.pos[n];
        m.prev[n] = make_float4(P.x, P.y, P.z, 0.f);
        m.vel[n] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// The reverse sweep of one brick; P holds the adjoint of the positions, Q the substep-start positions
// (damped), A their adjoint's accumulator (damped), V the adjoint of the velocities.
template <bool Damped>
__device__ __forceinline__ bool reverseSweep(Brick& b, const DeviceMesh& m, const DiffCoeffs& dc, const DiffBuffers& db, int j, int E, int T) {
    const int tid = threadIdx.x, step = blockDim.x;
    const int nE = b.s.nE, nT = b.s.nT;
    int st = 0;
    countChecks(b.bt.bounds, b.edgeOff[nE] - b.edgeOff[0] + b.tetOff[nT] - b.tetOff[0]);
    __syncthreads();
    if (dc.doStrain) {
        // Records two elements ahead (their tape slots), tape one ahead: neither is waited for.  Position
        // of an element of this thread: colour c, index k; a colour without one counts as an empty slot.
        struct Slot { BrickTet t; int src; bool valid; };
        const float4* tape = db.tapeTet + 4 * (size_t)j * T;
        int fc = 0, fk = nT > 0 ? b.tetOff[0] + tid : 0;   // the next slot to fetch
        auto fetch = [&]() {
            Slot s;
            s.valid = fc < nT && fk < b.tetOff[fc + 1];
            if (s.valid) { s.t = b.tetAt<false>(fk); s.src = b.tetSlot(fk); }
            if (fc < nT) {
                if (fk + step < b.tetOff[fc + 1]) fk += step;
                else { fc++; if (fc < nT) fk = b.tetOff[fc] + tid; }
            }
            return s;
        };
        Slot s0 = fetch();
        Slot s1 = fetch();
        float4 P0[4];
        if (s0.valid) { const float4* t = tape + 4 * (size_t)s0.src; P0[0] = t[0]; P0[1] = t[1]; P0[2] = t[2]; P0[3] = t[3]; }
        for (int c = 0; c < nT; c++) {
            if (b.exchangeAt(c)) { if (!b.exchange(st, false)) return false; st++; }
            const int hi = b.tetOff[c + 1];
            for (int k = b.tetOff[c] + tid;; k += step) {
                const Slot cur = s0;
                const float4 P[4] = {P0[0], P0[1], P0[2], P0[3]};
                s0 = s1;
                if (s0.valid) { const float4* t = tape + 4 * (size_t)s0.src; P0[0] = t[0]; P0[1] = t[1]; P0[2] = t[2]; P0[3] = t[3]; }
                s1 = fetch();
                if (cur.valid && (cur.t.word & kBrickTetLive)) {
                    const bool owner = (cur.t.word & kBrickTetOwner) != 0;
                    int id[4];
                    b.tetNodes(cur.t.word, id);
                    int slot = 0;
                    float th0 = 0.f;
                    if (owner) { slot = db.slotStorage[cur.src]; th0 = db.gTheta[slot]; }
                    f3 q[4], go[4];
#pragma unroll
                    for (int n = 0; n < 4; n++) { q[n] = Damped ? xyz(b.Q[id[n]]) : xyz(P[n]); go[n] = xyz(b.P[id[n]]); }
                    TetAdjoint adj;
                    const float2 a = cur.t.alpha;
                    tetVJP(b.typeB + 9 * Brick::tetType(cur.t.word), P, q, a.x, a.y, Damped ? dc.dampingOverH : 0.f, dc.omega, go, owner && db.gB != nullptr, adj);
#pragma unroll
                    for (int n = 0; n < 4; n++) {
                        b.P[id[n]] = f4(adj.gp[n], 0.f);
                        if (Damped && id[n] < b.d.nOwned) b.A[id[n]] = f4(xyz(b.A[id[n]]) + adj.gq[n], 0.f);
                    }
                    if (owner) {
                        db.gTheta[slot] = th0 + (adj.gad * a.x + adj.gah * a.y);
                        if (db.gB) {
                            float* gb = db.gB + (size_t)9 * cur.src;
#pragma unroll
                            for (int n = 0; n < 9; n++) gb[n] += adj.gB[n];
                        }
                    }
                }
                if (k + step >= hi) break;
            }
            __syncthreads();
        }
    } else {
        for (int c = 0; c < nT; c++)
            if (b.exchangeAt(c)) { if (!b.exchange(st, false)) return false; st++; }
    }
    const float4* tape = db.tapeEdge + 2 * (size_t)j * E;
    for (int c = 0; c < nE; c++) {
        if (b.exchangeAt(nT + c)) { if (!b.exchange(st, false)) return false; st++; }
        if (!dc.doEdges) continue;
        for (int k = b.edgeOff[c] + tid; k < b.edgeOff[c + 1]; k += step) {
            const BrickEdge e = b.edgeAt(k);
            if (!(e.word & kBrickEdgeLive)) continue;
            const int src = b.edgeSlot(k), x = b.local(e.word), y = b.local(e.word >> kBrickNodeBits);
            const float4 P0 = tape[2 * (size_t)src], P1 = tape[2 * (size_t)src + 1];
            const f3 qx = Damped ? xyz(b.Q[x]) : xyz(P0), qy = Damped ? xyz(b.Q[y]) : xyz(P1);
            const EdgeAdjoint adj = edgeVJP(P0, P1, qx, qy, e.rest, dc.alphaTilde, dc.betaGammaHS, dc.omega, xyz(b.P[x]), xyz(b.P[y]));
            b.P[x] = f4(adj.gpi, 0.f);
            b.P[y] = f4(adj.gpj, 0.f);
            if (Damped && dc.betaGammaHS != 0.f) {
                if (x < b.d.nOwned) b.A[x] = f4(xyz(b.A[x]) + adj.gqi, 0.f);
                if (y < b.d.nOwned) b.A[y] = f4(xyz(b.A[y]) + adj.gqj, 0.f);
            }
            if (db.gRest && (e.word & kBrickEdgeOwner)) db.gRest[src] += adj.grest;
        }
        __syncthreads();
    }
    return true;
}

template <bool Damped>
__device__ __forceinline__ void backwardBricks(const DeviceMesh& m, const DiffCoeffs& dc, const ContactParams& cp, const DiffBuffers& db,
                                               const BrickTables& bt, const BrickTables& rt, unsigned* barrier, long long budget) {
    extern __shared__ float4 shared[];
    const int N = db.total / db.frames, tid = threadIdx.x, step = blockDim.x, nodes = m.nNodes;
    const int E = m.nEdgeColors > 0 ? m.edgeRange[m.nEdgeColors - 1].y : 0, T = m.nTetColors > 0 ? m.tetRange[m.nTetColors - 1].y : 0;
    const FrameCoeffs fc = rollCoeffs(dc);
    GridSync grid{barrier, barrier + 1, gridDim.x, 0u, budget, 0u};
    Brick b(bt, bt.shape, m.typeB, blockIdx.x, shared, Damped, true, bt.bricks > 1 ? db.total * bt.shape.stages : 0, barrier + 1, budget, 0u);
    Brick v(rt, rt.shape, m.typeB, blockIdx.x, shared + Brick::bytes(bt, Damped) / sizeof(float4), Damped, true,
            rt.bricks > 1 ? db.total * rt.shape.stages : 0, barrier + 1, budget, 0u);
    for (int i = tid; i < v.d.nOwned; i += step) {
        v.P[i] = db.gx[v.node(i)];
        v.V[i] = v.A[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const f3 zero = mk(0.f, 0.f, 0.f);
    const int segments = (db.total + db.every - 1) / db.every;
    for (int seg = segments - 1; seg >= 0; seg--) {
        const int g0 = seg * db.every, g1 = min(db.total, g0 + db.every);
        const size_t base = (size_t)seg * nodes;
        __syncthreads();
        b.loadState(db.ckPos + base, db.ckVel + base, m.ext);
        for (int g = g0; g < g1; g++)
            if (!rollSubstep<Damped, true>(b, fc, dc, cp, db, g, N, g - g0, nodes, E, T)) return;
        if (!grid.sync()) return;   // the segment's tape is whole
        for (int g = g1 - 1; g >= g0; g--) {
            const int j = g - g0;
            Capsule cap{};
            if (dc.contact) cap = capsuleAt(db, dc, g, N);
            float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int i = tid; i < v.d.nOwned; i += step) {   // velocity update and contact, in reverse
                const size_t at = (size_t)j * nodes + v.node(i);
                const float w = b.P[i].w;
                f3 gx = xyz(v.P[i]), gqv = zero;
                if (w > 0.f) {
                    const f3 t = (xyz(v.V[i]) * dc.velScale) * dc.invH;
                    gx = gx + t;
                    gqv = zero - t;
                }
                if (dc.contact) {
                    f3 gsa = zero, gsb = zero;
                    gx = capsuleContactVJP(xyz(db.tapeX[at]), w, xyz(db.tapeV[at]), cap, cp, gx, gsa, gsb);
                    acc[0] += gsa.x; acc[1] += gsa.y; acc[2] += gsa.z; acc[3] += gsb.x; acc[4] += gsb.y; acc[5] += gsb.z;
                }
                v.P[i] = f4(gx, 0.f);
                v.A[i] = f4(gqv, 0.f);
            }
            if (Damped)
                for (int i = tid; i < v.d.nLocal; i += step) v.Q[i] = db.tapeQ[(size_t)j * nodes + v.node(i)];
            if (dc.contact) blockSum6(acc, db.pathPartial + ((size_t)g * gridDim.x + blockIdx.x) * 6);
            if (!reverseSweep<Damped>(v, m, dc, db, j, E, T)) return;
            for (int i = tid; i < v.d.nOwned; i += step) {   // predict: x1 = x + h v1, v1 = v + h a, prev = x
                const f3 g1x = xyz(v.P[i]);
                v.V[i] = f4(b.P[i].w > 0.f ? g1x * dc.h : zero, 0.f);
                v.P[i] = f4(g1x + xyz(v.A[i]), 0.f);
            }
        }
        if (seg > 0 && !grid.sync()) return;   // every reader is done with the tape
    }
    for (int i = tid; i < v.d.nOwned; i += step) {
        const int n = v.node(i);
        db.gx[n] = v.P[i];
        db.gv[n] = v.V[i];
        db.gq[n] = v.A[i];
    }
}

// Before a forward: the session's nodes at the origin with their inverse masses, and the compliances.
__global__ void rolloutSetup(DeviceMesh m, DiffBuffers b, int T, float invH2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < T) m.tetAlpha[i] = tetAlphaFromLog(b.theta[b.slotStorage[i]], b.young, b.bake[i], invH2);
    if (i < m.nNodes) {
        float4 P = b.originPos[i];
        P.w = nodeInvMass(m, i);
        m.pos[i] = P;
        m.vel[i] = b.originVel[i];
    }
}
__global__ void gatherCompliances(int n, const int* src, const float2* from, float2* to) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) to[i] = from[src[i]];
}

}  // namespace

template <bool Damped, int Threads>
static __global__ void __launch_bounds__(Threads, 1) brickForward(DeviceMesh m, DiffCoeffs dc, ContactParams cp, DiffBuffers b, BrickTables bt,
                                                                  unsigned* barrier, long long budget) {
    forwardBricks<Damped>(m, dc, cp, b, bt, barrier, budget);
}
BrickForwardKernel brickForwardFor(bool damped, int threads) {
    return threads <= kNarrowThreads ? (damped ? brickForward<true, kNarrowThreads> : brickForward<false, kNarrowThreads>)
                                     : (damped ? brickForward<true, kBrickThreads> : brickForward<false, kBrickThreads>);
}
__global__ void __launch_bounds__(kReverseThreads, 1) brickBackward(DeviceMesh m, DiffCoeffs dc, ContactParams cp, DiffBuffers b, BrickTables bt,
                                                                    BrickTables rt, unsigned* barrier, long long budget) {
    backwardBricks<false>(m, dc, cp, b, bt, rt, barrier, budget);
}
__global__ void __launch_bounds__(kReverseThreads, 1) brickBackwardDamped(DeviceMesh m, DiffCoeffs dc, ContactParams cp, DiffBuffers b,
                                                                          BrickTables bt, BrickTables rt, unsigned* barrier, long long budget) {
    backwardBricks<true>(m, dc, cp, b, bt, rt, barrier, budget);
}

cudaError_t prepareRollout(const DeviceMesh& m, const DiffBuffers& b, int E, int T, float invH2, BrickBuffers& forward, BrickBuffers& reverse,
                           cudaStream_t stream) {
    cudaError_t e = refreshMeshFlags(m, E, T, false, stream);
    if (e != cudaSuccess) return e;
    const int n = T > m.nNodes ? T : m.nNodes;
    rolloutSetup<<<(n + 255) / 256, 256, 0, stream>>>(m, b, T, invH2);
    for (BrickBuffers* k : {&forward, &reverse}) {
        e = k->refresh(m, false, stream);
        if (e != cudaSuccess) return e;
        if (k->tets) gatherCompliances<<<(k->tets + 255) / 256, 256, 0, stream>>>(k->tets, k->tetSrc, m.tetAlpha, (float2*)k->t.tetAlpha);
    }
    return cudaGetLastError();
}

}  // namespace gbt
