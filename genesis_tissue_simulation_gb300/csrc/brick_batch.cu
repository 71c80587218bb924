// Frames of batched instances on bricks: an instance's nodes in the shared memory of one CTA, or of
// several that exchange halo values (brick_frame.cuh).
//
// The lockstep grid (frame_kernels.cu) sweeps colour c of all instances together and closes it with a
// grid barrier; its gathers go through L2 and stall most of the frame (issue slots 23 % busy).  An
// instance is independent of the others, so here its colours are closed by its own CTA's barrier and its
// gathers are shared-memory reads.  256 instances of 8..32 cells, 10 substeps: 4.5 -> 2.3 ms a frame, issue
// slots 46 % busy; bound by issue and dependent latency together.
#include <algorithm>
#include <numeric>

#include "brick_batch.h"
#include "contact_point.cuh"
#include "host_parallel.h"

namespace gbt {
namespace {

// Velocity, contact and next predict of up to kNodes of this thread's nodes at a time: all their loads
// are issued before any store.
constexpr int kNodes = 2;

template <bool Damped, bool PerType>
__device__ __forceinline__ void batchFrame(const DeviceMesh& m, const FrameCoeffs& fc, const ContactParams& cp, const BrickTables& bt,
                                           const BrickShape* shapes, const int* order, const int* start, const float2* instAlpha,
                                           unsigned* status) {
    extern __shared__ float4 shared[];
    __shared__ float2 typeAlpha[6];
    __shared__ ContactFrame tool;
    __shared__ BrickShape shape;
    const int tid = threadIdx.x, T = blockDim.x;
    for (int at = start[blockIdx.x]; at < start[blockIdx.x + 1]; at++) {
        const int id = order[at], instance = bt.desc[id].shape;
        if (tid == 0) shape = shapes[instance];
        __syncthreads();
        if (PerType && tid < 6) typeAlpha[tid] = instAlpha[6 * instance + tid];
        Brick b(bt, shape, m.typeB, id, shared, Damped, false, shape.bricks > 1 ? fc.substeps * shape.stages : 0, status, fc.spinBudget, 0u);
        b.typeAlpha = typeAlpha;
        for (int i = tid; i < b.d.nLocal; i += T) b.P[i] = m.pos[b.node(i)];
        // owned nodes are predicted by the thread that loaded them; immobile ones never change
        for (int i = tid; i < b.d.nOwned; i += T) {
            const float4 P = b.P[i];
            if (Damped) b.Q[i] = P;
            if (!(P.w > 0.f)) continue;
            const int n = b.node(i);
            const float4 F = m.ext[n];
            m.prev[n] = make_float4(P.x, P.y, P.z, 0.f);
            const f3 v = xyz(m.vel[n]) + (mk(F.x, F.y, F.z) * P.w) * fc.h;
            m.vel[n] = make_float4(v.x, v.y, v.z, 0.f);
            const f3 x = xyz(P) + v * fc.h;
            b.P[i] = make_float4(x.x, x.y, x.z, P.w);
        }
        for (int s = 0; s < fc.substeps; s++) {
            const bool last = s + 1 == fc.substeps;
            if (fc.contact && tid < (int)(sizeof(ContactFrame) / 4))   // read after the sweep's barriers
                ((unsigned*)&tool)[tid] = ((const unsigned*)(m.contactFrames + (size_t)(fc.firstSubstep + s) * m.nInstances + instance))[tid];
            if (!b.sweep<Damped, false, PerType>(fc, [](bool) {})) return;
            for (int i0 = tid; i0 < b.d.nOwned; i0 += kNodes * T) {
                int n[kNodes];
                float4 P[kNodes], Q[kNodes], V[kNodes], F[kNodes];
#pragma unroll
                for (int u = 0; u < kNodes; u++) {
                    const int i = i0 + u * T;
                    n[u] = -1;
                    if (i >= b.d.nOwned) continue;
                    P[u] = b.P[i];
                    if (P[u].w > 0.f) n[u] = b.node(i);
                }
#pragma unroll
                for (int u = 0; u < kNodes; u++)
                    if (n[u] >= 0) {
                        Q[u] = m.prev[n[u]];
                        if (fc.contact) V[u] = m.vel[n[u]];
                        if (!last) F[u] = m.ext[n[u]];
                    }
#pragma unroll
                for (int u = 0; u < kNodes; u++) {
                    if (n[u] < 0) continue;
                    const int i = i0 + u * T;
                    f3 p = xyz(P[u]);
                    if (fc.contact) p = contactPoint(p, P[u].w, xyz(V[u]), tool, cp);
                    f3 v = ((p - xyz(Q[u])) * fc.invH) * fc.velScale;
                    if (!last) {
                        m.prev[n[u]] = make_float4(p.x, p.y, p.z, 0.f);
                        if (Damped) b.Q[i] = make_float4(p.x, p.y, p.z, 0.f);
                        v = v + (mk(F[u].x, F[u].y, F[u].z) * P[u].w) * fc.h;
                        p = p + v * fc.h;
                    }
                    m.vel[n[u]] = make_float4(v.x, v.y, v.z, 0.f);
                    b.P[i] = make_float4(p.x, p.y, p.z, P[u].w);
                }
            }
            __syncthreads();   // the next substep's instrument frame replaces this one
        }
        for (int i = tid; i < b.d.nOwned; i += T) {
            const float4 P = b.P[i];
            if (P.w > 0.f) m.pos[b.node(i)] = P;
        }
        __syncthreads();   // shared memory passes to the next brick
    }
}

// Shared memory of one brick of a batch: positions (and substep-start positions), rest inverses, offsets.
size_t brickBytes(const BrickPlan& p, const BrickDesc& d, bool damped) {
    return sizeof(float4) * (size_t)d.nLocal * (damped ? 2 : 1) + 54 * sizeof(float) +
           ((size_t)p.nEdgeColors + p.nTetColors + 2 * p.stages + 6) * sizeof(int);
}

}  // namespace

template <bool Damped, bool PerType, int Threads>
static __global__ void __launch_bounds__(Threads, 1) brickBatchFrame(DeviceMesh m, FrameCoeffs fc, ContactParams cp, BrickTables bt,
                                                                           const BrickShape* shapes, const int* order, const int* start,
                                                                           const float2* instAlpha, unsigned* status) {
    batchFrame<Damped, PerType>(m, fc, cp, bt, shapes, order, start, instAlpha, status);
}
template <int Threads> static BrickBatchKernel batchKernelFor(bool damped, bool perType) {
    return damped ? (perType ? brickBatchFrame<true, true, Threads> : brickBatchFrame<true, false, Threads>)
                  : (perType ? brickBatchFrame<false, true, Threads> : brickBatchFrame<false, false, Threads>);
}
BrickBatchKernel BatchBricks::kernel(bool damped, bool perType) const {
    return bound == kNarrowThreads ? batchKernelFor<kNarrowThreads>(damped, perType)
           : bound == kSplitThreads ? batchKernelFor<kSplitThreads>(damped, perType) : batchKernelFor<kBrickThreads>(damped, perType);
}

void BatchBricks::release() {
    buffers.release();
    for (void* p : {(void*)shapes, (void*)order, (void*)start}) if (p) cudaFree(p);
    shapes = nullptr; order = nullptr; start = nullptr;
    ctas = 0;
}

cudaError_t BatchBricks::plan(const std::vector<BatchBrickInstance>& in, int N, int smCount, int maxBytes, bool damped,
                              cudaStream_t stream) {
    release();
    const int count = (int)in.size();
    std::vector<long long> tets(count);
    long long all = 0;
    for (int i = 0; i < count; i++) { tets[i] = in[i].mesh.nTetColors ? in[i].mesh.tetOff[in[i].mesh.nTetColors] : 0; all += tets[i]; }
    const int record = damped ? 32 : 16, fixed = 2048;
    std::vector<int> bricks(count, 1);
    // One CTA of up to 512 threads an SM (256 instances of 8..32 cells, 2 frames: 5.0 ms; two CTAs of 256
    // threads an SM with half the shared memory each split more instances: 6.4 ms).
    const int slots = smCount, room = maxBytes;
    const bool spread = count <= smCount && all <= (long long)kSplitTets * smCount;
    if (spread) {
        // few tets an SM: a colour is shorter than its latency, so every instance is spread over its share of
        // the SMs
        for (int i = 0; i < count; i++) bricks[i] = (int)std::max<long long>(1, all ? tets[i] * smCount / all : 1);
        int sum = std::accumulate(bricks.begin(), bricks.end(), 0);
        for (; sum > slots; sum--) (*std::max_element(bricks.begin(), bricks.end()))--;
    } else {
        // many: only the instances well above a CTA's share, and those that do not fit one, are split
        // (splitting above 1.1, 1.25 and 1.6 shares: 5.4, 5.0 and 5.5 ms)
        const double roomNodes = (double)((room - fixed) / record);
        std::vector<int> served(count);
        for (int i = 0; i < count; i++) served[i] = (int)std::count_if(in[i].mesh.active, in[i].mesh.active + in[i].mesh.N, [](int a) { return a != 0; });
        bool fits = false;
        double share = 1.05 * (double)all / slots;
        for (int attempt = 0; attempt < 24 && !fits; attempt++, share *= 1.1) {
            long long split = 0;
            for (int i = 0; i < count; i++) {
                // a brick of a split instance keeps about a third more nodes than it owns
                const int need = served[i] <= roomNodes ? 1 : (int)std::ceil(1.35 * served[i] / roomNodes);
                bricks[i] = std::max(need, (double)tets[i] <= 1.25 * share ? 1 : (int)std::ceil((double)tets[i] / share));
                if (bricks[i] > 1) split += bricks[i];
            }
            fits = split <= slots;
        }
        if (!fits) return cudaSuccess;   // not ready: the instances' nodes do not fit side by side
    }
    std::vector<BrickPlan> plans(count);
    parallelFor(count, 16, [&](int i) {
        Team team(std::min(planThreads(in[i].mesh.N, in[i].mesh.active, bricks[i]), std::max(1, 16 / count)));   // 16 threads over all instances
        for (int more = 0; more < 3 && !plans[i].ok(); more++)   // a brick whose halo does not fit: smaller ones
            plans[i] = buildBrickPlan(in[i].mesh, bricks[i] + more, (room - fixed) / record, bricks[i] + more, damped, false, team);
    });
    struct Item { int id, instance; double work; bool tied; };
    std::vector<Item> items;
    bytes = 0;
    int tiedCount = 0;
    for (int i = 0; i < count; i++) {
        if (!plans[i].ok()) return cudaSuccess;   // not ready: the batch keeps its other shapes
        const BrickPlan& p = plans[i];
        for (int b = 0; b < p.bricks; b++) {
            bytes = std::max(bytes, brickBytes(p, p.desc[b], damped));
            const int* h = p.head.data() + p.desc[b].head;
            const double work = (h[p.nEdgeColors + 1 + p.nTetColors] - h[p.nEdgeColors + 1]) + 0.15 * (h[p.nEdgeColors] - h[0]);
            items.push_back({(int)items.size(), i, work, p.bricks > 1});
            if (p.bricks > 1) tiedCount++;
        }
    }
    if (bytes > (size_t)room || tiedCount > slots) return cudaSuccess;
    // one table of all bricks
    BrickPlan sum;
    std::vector<BrickShape> shape(count);
    sum.bricks = (int)items.size();
    for (int i = 0; i < count; i++) {
        const BrickPlan& p = plans[i];
        const BatchBrickInstance& q = in[i];
        shape[i] = p.shape();
        const int node0 = (int)sum.localNode.size(), edge0 = (int)sum.edgeWord.size(), tet0 = (int)sum.tetWord.size(),
                  imp0 = (int)sum.importList.size(), exp0 = (int)sum.exportList.size();
        for (const BrickDesc& d : p.desc) {
            sum.desc.push_back({d.nodeBase + node0, d.nOwned, d.nLocal, (int)sum.head.size(), i, 0, 0});
            const int* h = p.head.data() + d.head;
            auto put = [&](int n, int base) { for (int k = 0; k < n; k++) sum.head.push_back(*h++ + base); };
            put(p.nEdgeColors + 1, edge0); put(p.nTetColors + 1, tet0); put(p.stages + 1, imp0); put(p.stages + 1, exp0);
        }
        for (int n : p.localNode) sum.localNode.push_back(n + q.nodeBase);
        for (int2 e : p.importList) sum.importList.push_back(make_int2(e.x, e.y + q.nodeBase));
        for (int2 e : p.exportList) sum.exportList.push_back(make_int2(e.x, e.y + q.nodeBase));
        for (size_t k = 0; k < p.edgeWord.size(); k++) {
            sum.edgeWord.push_back(q.edgeDead[p.edgeSrc[k]] ? p.edgeWord[k] & ~kBrickEdgeLive : p.edgeWord[k]);
            sum.edgeRest.push_back(p.edgeRest[k]);
            sum.edgeSrc.push_back(q.edgeSlot[p.edgeSrc[k]]);
        }
        for (size_t k = 0; k < p.tetWord.size(); k++) {
            sum.tetWord.push_back(q.tetDead[p.tetSrc[k]] ? p.tetWord[k] & ~kBrickTetLive : p.tetWord[k]);
            sum.tetSrc.push_back(q.tetSlot[p.tetSrc[k]]);
        }
        sum.maxLocal = std::max(sum.maxLocal, p.maxLocal);
        sum.maxOwned = std::max(sum.maxOwned, p.maxOwned);
        sum.threads = std::max(sum.threads, p.threads);
        sum.tetWidth = std::max(sum.tetWidth, p.tetWidth);
        sum.meshEdges += p.meshEdges; sum.meshTets += p.meshTets;
    }
    // narrow colours: CTAs of kNarrowThreads with the whole register file (brick_frame.cuh); spread instances
    // with wider ones: 384 threads of 168 registers, which hold the node pass without spilling (ms a frame of 10
    // substeps with 384 and 512: 12 instances of 8..20 cells 0.40 and 0.44, 24 of them 0.49 and 0.53, 60 0.74 and 0.75,
    // 152 of 8..16 1.20 and 1.20, 100 of 8..24 1.22 and 1.21); else 512 (256 instances, 2 frames: 4.95 ms, 5.09 with 384)
    bound = sum.tetWidth <= kNarrowColour ? kNarrowThreads : spread ? kSplitThreads : kBrickThreads;
    threads = std::min(bound, sum.threads);
    // CTAs: exchanging bricks first, one each, then the others by longest processing time
    std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.tied != b.tied ? a.tied : a.work > b.work; });
    const int used = std::min(slots, (int)items.size());
    std::vector<std::vector<int>> lists(used);
    std::vector<double> load(used, 0.);
    for (const Item& it : items) {
        int best = -1;
        for (int c = 0; c < used; c++)
            if (!(it.tied && !lists[c].empty()) && (best < 0 || load[c] < load[best])) best = c;
        lists[best].push_back(it.id);
        load[best] += it.work;
    }
    std::vector<int> orderHost, startHost(1, 0);
    for (auto& l : lists) { orderHost.insert(orderHost.end(), l.begin(), l.end()); startHost.push_back((int)orderHost.size()); }
    cudaError_t e = buffers.upload(sum, N, damped, 0, stream);
    auto put = [&](auto** to, const auto& from) {
        if (e == cudaSuccess) e = cudaMalloc(to, from.size() * sizeof(from[0]));
        if (e == cudaSuccess) e = cudaMemcpyAsync(*to, from.data(), from.size() * sizeof(from[0]), cudaMemcpyHostToDevice, stream);
    };
    put(&shapes, shape); put(&order, orderHost); put(&start, startHost);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) { release(); return e; }
    ctas = used;
    return cudaSuccess;
}

}  // namespace gbt
