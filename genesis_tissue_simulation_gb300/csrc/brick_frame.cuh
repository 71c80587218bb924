// The coloured sweep of one brick in one CTA (host side: brick_plan.cpp).
//
// What bounds the sweep of a single mesh is the number of times the whole GPU has to agree: a frame
// kernel that closes every colour with a grid barrier and gathers positions through L2 spent about
// 1.3 us a colour in the barrier and 2 us in dependent L2 round trips, 37 colours a substep, with the
// issue slots nearly idle.  Here each CTA keeps the positions of its brick and of a halo in shared
// memory and runs several colours between two exchanges, projecting the elements near its faces
// redundantly; a colour then costs one gather from shared memory, the projection and __syncthreads.
// Frames of 64 x 32 x 48 cells, 20 substeps: 2.44 -> 1.21 ms; of 16 x 8 x 16 cells, 10 substeps: 0.79 (on one
// thread-block cluster) -> 0.33 ms.  Now bound by one projection's dependent chain a colour (~0.65 us with
// up to two warps a scheduler, ~1.0 us with 350 tets a brick) and ~2 us an exchange.
//
// Exchange: an owner publishes the values its neighbours need as 16-byte records (x, y, z, epoch), one
// relaxed 128-bit store each, into one of two buffers (by epoch parity), and a reader polls each record
// it needs until the epoch matches.  Data and flag arrive in one access, so an exchange costs one store
// and one load through L2 and no fence.  A buffer is written again two epochs later: by then every
// reader has published its next epoch (the plan makes neighbours read from each other every time).
#pragma once
#include "brick_plan.h"
#include "grid_sync.cuh"
#include "tissue_device.cuh"

namespace gbt {

constexpr int kBrickThreads = 512;
// Plans whose widest tet colour has at most kNarrowColour elements a brick run in CTAs of kNarrowThreads: twice the
// registers a thread and fewer warps at each barrier pay for the few second rounds.  The line is by the widest
// tet colour of a brick (edge colours may be twice as wide); us a frame of 20 substeps with 512 -> 256 threads:
// 211 wide (24 x 14 x 20 cells) 700 -> 678, 291 (32 x 16 x 32) 768 -> 764, 322 (44 x 20 x 36) 869 -> 869, 341 (40 x 20 x 30)
// 840 -> 832, 374 (48 x 24 x 36) 943 -> 982, 441 (64 x 16 x 48) 997 -> 1,097, 482 (64 x 32 x 48) 1,205 -> 1,366.
constexpr int kNarrowThreads = 256, kNarrowColour = 320;
constexpr int kBrickFrames = 32;   // instrument frames held in shared memory at a time

struct BrickTables {
    int bricks, maxLocal, maxOwned, nIdle, N;
    BrickShape shape;                                          // a batch keeps one per instance elsewhere
    const BrickDesc* desc; const int* head; const int* localNode; const int* idle;
    const int2* importList; const int2* exportList;            // (local index, node)
    int maxList;                                               // exchange records of one brick, kept in shared memory when listsShared
    int listsShared;
    const unsigned long long* tetWord; const float2* tetAlpha;
    const unsigned* edgeWord; const float* edgeRest;
    const int* ownTet;                                         // words of each brick's own tets (plans with a tensile pass)
    const int* tetSrc; const int* edgeSrc;                     // colour slots of the mesh's tables
    float4* mail;                                              // [2 x N] published values
    float4* mailStart;                                         // [2 x N] published substep-start positions (damped sweeps)
    unsigned* epoch;                                           // [bricks] exchanges so far, the same in every brick
    unsigned* bounds; int meshEdges, meshTets;                 // debug build: the gather record; colour slots of the mesh
};

__device__ __forceinline__ void publish(float4* to, f3 v, unsigned epoch) {
    const unsigned long long lo = (unsigned long long)__float_as_uint(v.x) | (unsigned long long)__float_as_uint(v.y) << 32;
    const unsigned long long hi = (unsigned long long)__float_as_uint(v.z) | (unsigned long long)epoch << 32;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" :: "l"(to), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ void peek(const float4* from, unsigned long long& lo, unsigned long long& hi) {
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}" : "=l"(lo), "=l"(hi) : "l"(from) : "memory");
}

// Checks of one brick's exchange records in the debug build; nothing otherwise.
#ifdef GBT_DEBUG_BOUNDS
struct ListCheck {
    unsigned* rec; int nOwned, nLocal, N;
    __device__ int2 given(int2 e) const { return make_int2(checkRange(rec, e.x, 0, nOwned, kSiteBrickList), checkRange(rec, e.y, 0, N, kSiteBrickList)); }
    __device__ int2 taken(int2 e) const { return make_int2(checkRange(rec, e.x, nOwned, nLocal - nOwned, kSiteBrickList), checkRange(rec, e.y, 0, N, kSiteBrickList)); }
};
#else
struct ListCheck {
    __device__ __forceinline__ int2 given(int2 e) const { return e; }
    __device__ __forceinline__ int2 taken(int2 e) const { return e; }
};
#endif

// One thread's records e[0 .. count) of an exchange, all polled together until each has its epoch.
constexpr int kTake = 4;
template <class Put>
__device__ __forceinline__ bool take(const float4* from, const int2 (&e)[kTake], unsigned waiting, unsigned want, unsigned* status,
                                     long long budget, Put&& put) {
    long long start = 0;
    for (unsigned rounds = 1; waiting != 0u; rounds++) {
        unsigned long long lo[kTake], hi[kTake];
#pragma unroll
        for (int u = 0; u < kTake; u++) if (waiting >> u & 1u) peek(from + e[u].y, lo[u], hi[u]);
#pragma unroll
        for (int u = 0; u < kTake; u++)
            if ((waiting >> u & 1u) && (unsigned)(hi[u] >> 32) == want) {
                put(e[u].x, mk(__uint_as_float((unsigned)lo[u]), __uint_as_float((unsigned)(lo[u] >> 32)), __uint_as_float((unsigned)hi[u])));
                waiting &= ~(1u << u);
            }
        if ((rounds & 31u) == 0u && waiting != 0u) {
            if (start == 0) start = clock64();
            if (*(volatile unsigned*)status != 0u) return false;
            if (clock64() - start > budget) { atomicOr(status, kSyncTimeout); return false; }
        }
    }
    return true;
}
// Publishes the listed values and takes the neighbours'.  A function of values, out of line: the sweep
// around it keeps its registers, and P and Q stay shared-memory addresses there.
// A record can not be there sooner than about kFlight cycles after neighbours in step began to publish,
// and polls before that only hold the stores up.  64 x 32 x 48 cells: 64.1 us a substep polling at once,
// 62.1 after 800 cycles, 60.4 after 1200; 32 x 16 x 32 cells: 41.3, 39.0 and 38.3; 16 x 8 x 16 cells: 34.2,
// 33.5 and 33.0; 23 x 13 x 19 cells: 34.9, 34.0 and 34.6.
constexpr int kFlight = 1100;
static __device__ __noinline__ bool exchangeRecords(float4* box, float4* boxStart, float4* P, float4* Q, const int2* exports, int nExports,
                                                    const int2* imports, int nImports, unsigned epoch, unsigned lag, unsigned* status,
                                                    long long budget, ListCheck check) {
    const int T = blockDim.x, tid = threadIdx.x;
    const long long start = clock64();
    for (int i = tid; i < nExports; i += T) {
        const int2 e = check.given(exports[i]);
        publish(box + e.y, xyz(P[e.x]), epoch);
        if (boxStart) publish(boxStart + e.y, xyz(Q[e.x]), epoch);
    }
    while (clock64() - start < kFlight) {}
    bool bad = false;
    for (int i = tid; i < nImports; i += kTake * T) {
        int2 e[kTake];
        unsigned mine = 0u;
#pragma unroll
        for (int u = 0; u < kTake; u++) if (i + u * T < nImports) { e[u] = check.taken(imports[i + u * T]); mine |= 1u << u; }
        bad = !take(box, e, mine, epoch + lag, status, budget, [&](int at, f3 v) { float4& p = P[at]; p.x = v.x; p.y = v.y; p.z = v.z; }) || bad;
        if (boxStart) bad = !take(boxStart, e, mine, epoch + lag, status, budget, [&](int at, f3 v) { Q[at] = make_float4(v.x, v.y, v.z, 0.f); }) || bad;
    }
    return __syncthreads_or(bad ? 1 : 0) == 0;
}

// Where a recorded sweep writes every element's node positions before its projection (by colour slot;
// the element's owner writes them).
struct BrickTape { float4* edge; float4* tet; };

struct BrickTet { unsigned long long word; float2 alpha; };
struct BrickEdge { unsigned word; float rest; };

struct Brick {
    const BrickTables& bt;
    const BrickShape& s;   // in the kernel's parameters or in shared memory
    BrickDesc d;
    float4* P;        // [maxLocal] positions (w = inverse mass)
    float4* Q;        // [maxLocal] damped sweeps, else [maxOwned]: substep-start positions
    float4* V;        // [maxOwned] velocities
    float4* A;        // [maxOwned] accelerations
    ContactFrame* frames;   // [kBrickFrames]
    float* typeB;     // [6 x 9] rest inverses
    const float* fibres;       // [6 x 6] rest lengths of the tensile fibres per Kuhn type (guarded sweeps)
    const float2* typeAlpha;   // [6] compliances per Kuhn type (sweeps without one per tet)
    int* head;        // offsets of this brick (brick_plan.h)
    const int *edgeOff, *tetOff, *impOff, *expOff;
    int2 *imports, *exports;   // this brick's lists in shared memory (listsShared)
    unsigned epoch;   // of the last exchange
    unsigned* status; // barrier status word: kSyncTimeout once a wait ran out
    long long budget; unsigned lag;   // lag: epochs awaited beyond the published one (timeout test)

    // Shared memory of a resident brick of the tables' largest sizes (the lists of the widest brick).
    static __host__ __device__ size_t bytes(const BrickTables& t, bool damped) {
        const size_t head = (size_t)t.shape.nE + t.shape.nT + t.shape.nTensile + 2 * t.shape.stages + 6;
        const size_t all = sizeof(float4) * ((size_t)t.maxLocal + (damped ? t.maxLocal : t.maxOwned) + 2 * (size_t)t.maxOwned) +
                           kBrickFrames * sizeof(ContactFrame) + 54 * sizeof(float) + head * sizeof(int) +
                           (t.listsShared ? sizeof(int2) * (size_t)t.maxList : 0);
        return (all + 15) & ~(size_t)15;
    }
    // Shared-memory layout, offsets and exchange lists.  Closed by a barrier.
    // resident: velocities, accelerations and substep-start positions live here too; else the caller keeps
    // them in device memory (damped sweeps still read Q).
    __device__ __forceinline__ Brick(const BrickTables& t, const BrickShape& shape, const float (&rest)[6][9], int b, float4* shared, bool damped,
                                     bool resident, int exchanges, unsigned* statusWord, long long spinBudget, unsigned lagEpochs)
        : bt(t), s(shape), d(t.desc[b]), status(statusWord), budget(spinBudget), lag(lagEpochs) {
        P = shared;
        Q = P + d.nLocal;
        V = Q + (damped ? d.nLocal : resident ? d.nOwned : 0);
        A = V + (resident ? d.nOwned : 0);
        frames = (ContactFrame*)(A + (resident ? d.nOwned : 0));
        typeB = (float*)(frames + (resident ? kBrickFrames : 0));
        head = (int*)(typeB + 54);
        edgeOff = head; tetOff = edgeOff + s.nE + 1; impOff = tetOff + s.nT + s.nTensile + 1; expOff = impOff + s.stages + 1;
        const int words = s.nE + s.nT + s.nTensile + 2 * s.stages + 4;
        imports = (int2*)(head + (words + 1) / 2 * 2);
        for (int i = threadIdx.x; i < words; i += blockDim.x) head[i] = t.head[d.head + i];
        for (int i = threadIdx.x; i < 54; i += blockDim.x) typeB[i] = rest[i / 9][i % 9];
        epoch = s.bricks > 1 ? t.epoch[b] : 0u;
        __syncthreads();
        exports = imports + (impOff[s.stages] - impOff[0]);
        if (t.listsShared) {
            for (int i = threadIdx.x; i < impOff[s.stages] - impOff[0]; i += blockDim.x) imports[i] = t.importList[impOff[0] + i];
            for (int i = threadIdx.x; i < expOff[s.stages] - expOff[0]; i += blockDim.x) exports[i] = t.exportList[expOff[0] + i];
            __syncthreads();
        }
        if (s.bricks > 1 && threadIdx.x == 0) t.epoch[b] = epoch + (unsigned)exchanges;   // also when a wait runs out
    }

    // Node of a local index, and the local nodes of an element's word.
    __device__ __forceinline__ int node(int l) const { return checkRange(bt.bounds, bt.localNode[d.nodeBase + l], 0, bt.N, kSiteBrickNode); }
    __device__ __forceinline__ int local(unsigned bits) const { return checkRange(bt.bounds, (int)(bits & kBrickNodeMask), 0, d.nLocal, kSiteBrickLocal); }
    __device__ __forceinline__ void tetNodes(unsigned long long word, int (&id)[4]) const {
        const unsigned lo = (unsigned)word, hi = (unsigned)(word >> 28);
        id[0] = local(lo); id[1] = local(lo >> kBrickNodeBits); id[2] = local(hi); id[3] = local(hi >> kBrickNodeBits);
    }
    static __device__ __forceinline__ int tetType(unsigned long long word) { return (int)((unsigned)(word >> 56) & 7u); }
    __device__ __forceinline__ int edgeSlot(int k) const { return checkRange(bt.bounds, bt.edgeSrc[k], 0, bt.meshEdges, kSiteBrickSource); }
    __device__ __forceinline__ int tetSlot(int k) const { return checkRange(bt.bounds, bt.tetSrc[k], 0, bt.meshTets, kSiteBrickSource); }
    __device__ __forceinline__ ListCheck listCheck() const {
#ifdef GBT_DEBUG_BOUNDS
        return {bt.bounds, d.nOwned, d.nLocal, bt.N};
#else
        return {};
#endif
    }

    // The positions of owned and halo nodes, and the owned nodes' accelerations and velocities.
    __device__ __forceinline__ void loadState(const float4* pos, const float4* vel, const float4* ext) {
        for (int i = threadIdx.x; i < d.nLocal; i += blockDim.x) P[i] = pos[node(i)];
        for (int i = threadIdx.x; i < d.nOwned; i += blockDim.x) {
            const int n = node(i);
            const float4 F = ext[n];
            const f3 a = mk(F.x, F.y, F.z) * pos[n].w;
            A[i] = make_float4(a.x, a.y, a.z, 0.f);
            V[i] = vel[n];
        }
    }

    // The values stage `st` needs: publish this brick's, take the neighbours'.  All threads, after a
    // barrier; closes with one.  False when a neighbour did not publish within the budget.
    __device__ __forceinline__ bool exchange(int st, bool withStart) {
        epoch++;
        const size_t box = (size_t)(epoch & 1u) * bt.N;
        const int oe = expOff[st], ne = expOff[st + 1] - oe, oi = impOff[st], ni = impOff[st + 1] - oi;
        return exchangeRecords(bt.mail + box, withStart ? bt.mailStart + box : nullptr, P, Q,
                               bt.listsShared ? exports + (oe - expOff[0]) : bt.exportList + oe, ne,
                               bt.listsShared ? imports + (oi - impOff[0]) : bt.importList + oi, ni, epoch, lag, status, budget, listCheck());
    }

    __device__ __forceinline__ bool exchangeAt(int p) const { return (s.before[p >> 6] >> (p & 63)) & 1ull; }
    template <bool PerType>
    __device__ __forceinline__ BrickTet tetAt(int k) const {
        BrickTet t;
        t.word = bt.tetWord[k];
        if (!PerType) t.alpha = bt.tetAlpha[k];
        return t;
    }
    __device__ __forceinline__ BrickEdge edgeAt(int e) const { return {bt.edgeWord[e], bt.edgeRest[e]}; }

    template <bool Damped, bool Record>
    __device__ __forceinline__ void edge(const BrickEdge& w, const FrameCoeffs& fc, int k, const BrickTape& tape) {
        if (!(w.word & kBrickEdgeLive)) return;
        const int a = local(w.word), b = local(w.word >> kBrickNodeBits);
        EdgeRecord r;
        r.live = 1; r.rest = w.rest;
        if (Damped) { r.qi = xyz(Q[a]); r.qj = xyz(Q[b]); } else r.qi = r.qj = mk(0.f, 0.f, 0.f);
        float4 oa, ob;
        const float4 pa = P[a], pb = P[b];
        if (Record && (w.word & kBrickEdgeOwner)) {
            float4* t = tape.edge + 2 * (size_t)edgeSlot(k);
            t[0] = pa; t[1] = pb;
        }
        if (solveEdge(r, fc, pa, pb, oa, ob)) { P[a] = oa; P[b] = ob; }
    }
    // Guarded: the tissue guard's form when `guarded` (damping then includes the bulk's).
    template <bool Damped, bool Record, bool PerType, bool Guarded>
    __device__ __forceinline__ void tet(const BrickTet& w, const FrameCoeffs& fc, int k, const BrickTape& tape) {
        if (!(w.word & kBrickTetLive)) return;
        int id[4];
        tetNodes(w.word, id);
        const int type = tetType(w.word);
        const float4 p[4] = {P[id[0]], P[id[1]], P[id[2]], P[id[3]]};
        if (Record && (w.word & kBrickTetOwner)) {
            float4* t = tape.tet + 4 * (size_t)tetSlot(k);
            t[0] = p[0]; t[1] = p[1]; t[2] = p[2]; t[3] = p[3];
        }
        f3 q[4], o[4];
#pragma unroll
        for (int c = 0; c < 4; c++) q[c] = Damped ? xyz(Q[id[c]]) : mk(0.f, 0.f, 0.f);
        if (!solveTet(typeB + 9 * type, p, q, PerType ? typeAlpha[type] : w.alpha, fc, Damped && tetDamped(fc, Guarded && fc.guarded != 0), Guarded && fc.guarded != 0, o)) return;
#pragma unroll
        for (int c = 0; c < 4; c++) P[id[c]] = make_float4(o[c].x, o[c].y, o[c].z, p[c].w);
    }

    // Tensile reinforcement of one tet (one pass: its multipliers start at zero).
    __device__ __forceinline__ void tensile(const BrickTet& w, const FrameCoeffs& fc) {
        if (!(w.word & kBrickTetLive) || !(fc.tensileStrength > 0.f)) return;
        int id[4];
        tetNodes(w.word, id);
        const int type = tetType(w.word);
        const float4 q[4] = {P[id[0]], P[id[1]], P[id[2]], P[id[3]]};
        f3 p[4] = {xyz(q[0]), xyz(q[1]), xyz(q[2]), xyz(q[3])};
        float rest[6], lambda[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int f = 0; f < 6; f++) rest[f] = fibres[6 * type + f];
        solveTensile(rest, q, w.alpha.x / fmaxf(fc.tensileStrength, 1e-10f), lambda, p);
#pragma unroll
        for (int c = 0; c < 4; c++) P[id[c]] = make_float4(p[c].x, p[c].y, p[c].z, q[c].w);
    }
    // Whether any live tet that this brick owns is below the minimum relative volume (the guard's test),
    // by this thread.
    __device__ __forceinline__ bool belowMinimum(float minimum) const {
        bool below = false;
        for (int k = threadIdx.x; k < d.nOwn; k += blockDim.x) {
            const unsigned long long w = bt.tetWord[checkRange(bt.bounds, bt.ownTet[d.ownFirst + k], tetOff[0], tetOff[s.nT] - tetOff[0], kSiteBrickSource)];
            if (!(w & kBrickTetLive)) continue;
            int id[4];
            tetNodes(w, id);
            const float* B = typeB + 9 * tetType(w);
            const f3 b0 = mk(B[0], B[1], B[2]), b1 = mk(B[3], B[4], B[5]), b2 = mk(B[6], B[7], B[8]);
            const f3 a = xyz(P[id[0]]), u = xyz(P[id[1]]) - a, v = xyz(P[id[2]]) - a, x = xyz(P[id[3]]) - a;
            const float J = dot(u, cross(v, x)) * dot(b0, cross(b1, b2));
            below = below || !isfinite(J) || J < minimum;
        }
        return below;
    }

    // One sweep over the colours from the positions in P (owned nodes current, halo by the first
    // exchange).  A thread always holds the record of its next element, loaded while it projects the one
    // before, across colours and exchanges.  Opens and closes with a barrier; false on a timeout.
    // after(edges) is called when a colour is done.
    template <bool Damped, bool Record = false, bool PerType = false, bool Guarded = false, class After>
    __device__ __forceinline__ bool sweep(const FrameCoeffs& fc, After&& after, const BrickTape& tape = BrickTape()) {
        const int T = blockDim.x, tid = threadIdx.x;
        const int nE = s.nE, nT = s.nT + (Guarded ? s.nTensile : 0);
        int st = 0;
        countChecks(bt.bounds, edgeOff[nE] - edgeOff[0] + tetOff[nT] - tetOff[0]);
        BrickEdge nextEdge;
        BrickTet nextTet;
        if (fc.doEdges && nE > 0 && edgeOff[0] + tid < edgeOff[1]) nextEdge = edgeAt(edgeOff[0] + tid);
        if (fc.doStrain && nT > 0 && tetOff[0] + tid < tetOff[1]) nextTet = tetAt<PerType>(tetOff[0] + tid);
        __syncthreads();
        {   // offsets two colours ahead: none is waited for (all zero when the phase is off)
            int lo = fc.doEdges ? edgeOff[0] : 0, hi = fc.doEdges ? edgeOff[min(1, nE)] : 0, hi2 = fc.doEdges ? edgeOff[min(2, nE)] : 0;
            for (int c = 0; c < nE; c++) {
                const int hi3 = fc.doEdges ? edgeOff[min(c + 3, nE)] : 0;
                if (exchangeAt(c)) { if (!exchange(st, Damped && st == 0)) return false; st++; }
                for (int k = lo + tid;;) {
                    const bool have = k < hi, last = k + T >= hi;
                    const BrickEdge cur = nextEdge;
                    const int kn = last ? hi + tid : k + T;
                    if (kn < (last ? hi2 : hi)) nextEdge = edgeAt(kn);
                    if (have) edge<Damped, Record>(cur, fc, k, tape);
                    if (last) break;
                    k = kn;
                }
                lo = hi; hi = hi2; hi2 = hi3;
                __syncthreads();
                after(true);
            }
        }
        {   // offsets two colours ahead: none is waited for (all zero when the phase is off)
            int lo = fc.doStrain ? tetOff[0] : 0, hi = fc.doStrain ? tetOff[min(1, nT)] : 0, hi2 = fc.doStrain ? tetOff[min(2, nT)] : 0;
            for (int c = 0; c < nT; c++) {
                const int hi3 = fc.doStrain ? tetOff[min(c + 3, nT)] : 0;
                if (exchangeAt(nE + c)) { if (!exchange(st, Damped && st == 0)) return false; st++; }
                for (int k = lo + tid;;) {
                    const bool have = k < hi, last = k + T >= hi;
                    const BrickTet cur = nextTet;
                    const int kn = last ? hi + tid : k + T;
                    if (kn < (last ? hi2 : hi)) nextTet = tetAt<PerType>(kn);
                    if (Guarded && c >= s.nT) { if (have) tensile(cur, fc); }
                    else if (have) tet<Damped, Record, PerType, Guarded>(cur, fc, k, tape);
                    if (last) break;
                    k = kn;
                }
                lo = hi; hi = hi2; hi2 = hi3;
                __syncthreads();
                after(false);
            }
        }
        return true;
    }
};

}  // namespace gbt
