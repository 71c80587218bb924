// Spatial bricks of a coloured lattice mesh: which elements every CTA of the brick kernel projects,
// and which node values it takes from its neighbours when (brick_plan.cpp, brick_frame.cuh).
#pragma once
#include <cstdint>
#include <memory>
#include <new>
#include <utility>
#include <vector>
#include <cuda_runtime.h>

namespace gbt {

// One brick.  All offsets index the plan's concatenated tables.  `head` is the start of its header
// words: edgeOff[nEdgeColors + 1], tetOff[nTetColors + 1], importOff[stages + 1], exportOff[stages + 1],
// each absolute.
struct BrickDesc {
    int nodeBase, nOwned, nLocal;   // localNode[nodeBase + l]: node of local index l, owned nodes first
    int head;
    int shape;                      // of a batch: the instance's plan
    int ownFirst, nOwn;             // ownTet[ownFirst .. ownFirst + nOwn): the words of the tets it owns (plans with a tensile pass)
};

// The sweep of one plan: colours, stages, and the phases an exchange precedes (bit p: phase p).
struct BrickShape {
    int nE, nT, stages, bricks;
    int nTensile;                   // colours that follow the nT tet colours: the tets once more per tensile pass
    unsigned long long before[2];
};

// Element words.  A tet: local nodes in bits 0-13, 14-27, 28-41 and 42-55, Kuhn type 56-58, live 59.
// An edge: local ends in bits 0-13 and 14-27, live 28.  Bit 60 (tets) and 29 (edges): the brick owns the
// element's first node, so exactly one brick has it set.
constexpr int kBrickNodeBits = 14, kBrickMaxLocal = 1 << kBrickNodeBits;
constexpr unsigned kBrickNodeMask = kBrickMaxLocal - 1;
constexpr uint64_t kBrickTetLive = 1ull << 59, kBrickTetOwner = 1ull << 60;
constexpr unsigned kBrickEdgeLive = 1u << 28, kBrickEdgeOwner = 1u << 29;

struct BrickMesh {   // the coloured mesh a plan is made for; nodes on an nx * ny * nz lattice
    int N, nx, ny, nz;
    const int* active;                                              // [N]
    int nEdgeColors, nTetColors;
    const int* edgeOff; const int2* edgeEnds; const float* edgeRest;   // colour order
    const int* tetOff; const int4* tetIds; const int* tetMeta;
    int tensilePasses = 0;                                          // sweeps over the tet colours after the projection's
};

// A table that is sized without being filled first (its makers write every entry, each thread its own pages).
template <class T> struct Unfilled : std::allocator<T> {
    template <class U> struct rebind { using other = Unfilled<U>; };
    template <class U> void construct(U* p) { ::new ((void*)p) U; }
    template <class U, class A, class... Rest> void construct(U* p, A&& a, Rest&&... rest) { ::new ((void*)p) U(std::forward<A>(a), std::forward<Rest>(rest)...); }
};
template <class T> using PlanTable = std::vector<T, Unfilled<T>>;

struct BrickPlan {
    int bricks = 0, stages = 1, nEdgeColors = 0, nTetColors = 0, maxLocal = 0, maxOwned = 0, maxList = 0;
    int tensilePasses = 0;                 // nTetColors counts the tet colours of every pass
    int asked = 0;                         // the brick count the split was chosen for
    int threads = 32;                      // of a CTA: the widest phase, in whole warps
    int meshEdges = 0, meshTets = 0;       // colour slots the words come from
    int tetWidth = 0;                      // elements of the widest tet phase of a brick
    uint64_t exchangeBefore[2] = {0, 0};   // bit p: neighbours' values are taken before phase p (edge colours, then tet colours)
    std::vector<BrickDesc> desc;
    std::vector<int> head, idle, ownTet;
    PlanTable<int> localNode;
    PlanTable<int2> importList, exportList;   // (local index, node)
    PlanTable<uint64_t> tetWord; PlanTable<int> tetSrc;
    PlanTable<unsigned> edgeWord; PlanTable<float> edgeRest; PlanTable<int> edgeSrc;
    bool ok() const { return bricks > 0; }
    BrickShape shape() const { return {nEdgeColors, nTetColors / (1 + tensilePasses), stages, bricks, nTetColors / (1 + tensilePasses) * tensilePasses, {exchangeBefore[0], exchangeBefore[1]}}; }
};

class Team;
// The plan of `mesh` on at most `maxBricks` CTAs that keep at most `maxLocal` nodes each; forced > 0
// asks for about that many bricks instead of one, or one per CTA, by the nodes served.  wholeHalo: the
// first exchange takes every halo node (damped sweeps read all of them at the substep's start).  reverse:
// the sweep runs tet colours and then edge colours from last to first.  Returns a plan without bricks when
// none fits.  The loops run on `team` (planThreads: the threads worth starting for it).
BrickPlan buildBrickPlan(const BrickMesh& mesh, int maxBricks, int maxLocal, int forced, bool wholeHalo, bool reverse, Team& team);
int planThreads(int N, const int* active, int forced);

}  // namespace gbt
