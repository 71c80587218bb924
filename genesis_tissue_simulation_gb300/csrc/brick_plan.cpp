// Host construction of the brick plan (brick_plan.h).
//
// The lattice is cut into a grid of boxes, one per CTA.  A sweep is a sequence of phases, one per
// colour, in which an element reads and writes its own nodes only.  The phases are grouped into
// stages; at the start of a stage a brick takes its neighbours' current values of the halo nodes it
// needs, and runs the stage's phases without talking to anyone: it projects every element that its
// owned nodes' values at the end of the stage depend on, found by walking the stage's phases from
// last to first (an element that touches a needed node is needed, and so are all its nodes).
// Elements near a brick's faces are projected by more than one brick, from the same values with the
// same operations, so every brick's owned nodes end exactly as one sweep over the whole mesh leaves them.
//
// A session waits for its plan when it opens, so a few threads share the bricks, lists are flat, and sorted ones
// come out of bitmaps (milliseconds on 16 threads: 16 x 8 x 16 cells 1.4, 11 x 6 x 13 in reverse 0.95, 64 x 32 x 48
// 6.2; with a vector and a sort per brick and colour 3.3, 2.1 and 25).
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <memory>

#include "brick_plan.h"
#include "host_parallel.h"

namespace gbt {
namespace {

// Model time of one phase of n elements and of one exchange of n halo nodes in a CTA, microseconds
// (fitted to frames of 8 x 4 x 8 to 64 x 32 x 48 cells on 1 to 152 bricks).
constexpr double kEdgePhase = 0.25, kEdgeEach = 0.0007, kTetPhase = 0.55, kTetEach = 0.0019;
constexpr double kExchange = 1.5, kImportEach = 0.0006;

// The reverse projection of a tet costs about three times the forward one.
constexpr double kReverseTetPhase = 1.6, kReverseTetEach = 0.0065;

struct Phases {
    const BrickMesh& m;
    bool reverse;
    int nT;                // tet colours of all passes
    int count;
    std::unique_ptr<int[]> at;   // [edge colours, then tet colours][N] the colour's element at the node, or -1
    std::unique_ptr<std::atomic<unsigned char>[]> ends;   // [N] whether any element ends at the node
    Phases(const BrickMesh& mesh, bool rev, Team& team)
        : m(mesh), reverse(rev), nT(mesh.nTetColors * (1 + mesh.tensilePasses)), count(mesh.nEdgeColors + nT),
          at(new int[(size_t)(mesh.nEdgeColors + mesh.nTetColors) * mesh.N]), ends(new std::atomic<unsigned char>[mesh.N]()) {
        team.run(m.nEdgeColors + m.nTetColors, [&](int row, int) {
            int* a = at.get() + (size_t)row * m.N;
            std::fill(a, a + m.N, -1);
            auto put = [&](int n, int k) { a[n] = k; ends[n].store(1, std::memory_order_relaxed); };
            if (row < m.nEdgeColors) {
                for (int k = m.edgeOff[row]; k < m.edgeOff[row + 1]; k++) { put(m.edgeEnds[k].x, k); put(m.edgeEnds[k].y, k); }
            } else {
                const int c = row - m.nEdgeColors;
                for (int k = m.tetOff[c]; k < m.tetOff[c + 1]; k++) { const int4 t = m.tetIds[k]; put(t.x, k); put(t.y, k); put(t.z, k); put(t.w, k); }
            }
        });
    }
    bool isEdge(int p) const { return reverse ? p >= nT : p < m.nEdgeColors; }
    int colour(int p) const {   // of the mesh (a tensile pass repeats the tet colours)
        if (!reverse) return p < m.nEdgeColors ? p : (p - m.nEdgeColors) % m.nTetColors;
        return p < nT ? (nT - 1 - p) % m.nTetColors : m.nEdgeColors - 1 - (p - nT);
    }
    const int* elementsAt(int p) const { return at.get() + (size_t)(isEdge(p) ? colour(p) : m.nEdgeColors + colour(p)) * m.N; }
    int first(int p) const { return (isEdge(p) ? m.edgeOff : m.tetOff)[colour(p)]; }
    int nodes(int p, int k, int out[4]) const {
        if (isEdge(p)) { out[0] = m.edgeEnds[k].x; out[1] = m.edgeEnds[k].y; return 2; }
        const int4 t = m.tetIds[k];
        out[0] = t.x; out[1] = t.y; out[2] = t.z; out[3] = t.w;
        return 4;
    }
    int widest() const {   // elements of the widest colour
        int w = 0;
        for (int c = 0; c < m.nEdgeColors; c++) w = std::max(w, m.edgeOff[c + 1] - m.edgeOff[c]);
        for (int c = 0; c < m.nTetColors; c++) w = std::max(w, m.tetOff[c + 1] - m.tetOff[c]);
        return w;
    }
};

// A set of nodes cleared by one increment.
struct Marks {
    std::vector<unsigned> at; unsigned now = 0;
    explicit Marks(size_t n) : at(n, 0) {}
    void clear() { now++; }
    bool add(int i) { if (at[i] == now) return false; at[i] = now; return true; }
};

// A set of small numbers that gives them back in order, and is empty afterwards.
struct Bits {
    std::vector<uint64_t> word; int lo = INT_MAX, hi = -1;
    explicit Bits(size_t n) : word(n / 64 + 1, 0) {}
    bool add(int i) {
        const int w = i >> 6;
        const uint64_t b = 1ull << (i & 63);
        if (word[w] & b) return false;
        word[w] |= b;
        lo = std::min(lo, w); hi = std::max(hi, w);
        return true;
    }
    template <class Each> void drain(Each&& each) {
        for (int w = lo; w <= hi; w++) {
            for (uint64_t b = word[w]; b; b &= b - 1) each(64 * w + __builtin_ctzll(b));
            word[w] = 0;
        }
        lo = INT_MAX; hi = -1;
    }
};

// One thread's workspace.
struct Scratch {
    Marks node; Bits element, nodes, halo;
    std::vector<int> need;
    std::unique_ptr<int[]> localOf;
    Scratch(int N, int widest) : node(N), element(widest), nodes(N), halo(N), localOf(new int[N]) {}
};

// One step of the backward walk: the elements of phase p that touch s.need, whose nodes join it.  Returns their
// number; `elements` takes them in order.
int widen(const Phases& ph, int p, Scratch& s, std::vector<int>* elements) {
    const int* at = ph.elementsAt(p);
    const int first = ph.first(p);
    int count = 0;
    const size_t had = s.need.size();
    for (size_t i = 0; i < had; i++) {
        const int k = at[s.need[i]];
        if (k < 0 || !s.element.add(k - first)) continue;
        count++;
        int nd[4];
        const int c = ph.nodes(p, k, nd);
        for (int j = 0; j < c; j++) if (s.node.add(nd[j])) s.need.push_back(nd[j]);
    }
    if (elements) s.element.drain([&](int e) { elements->push_back(first + e); });
    else s.element.drain([](int) {});
    return count;
}
void startWalk(Scratch& s, const int* owned, int n) {
    s.need.assign(owned, owned + n);
    s.node.clear();
    for (int i = 0; i < n; i++) s.node.add(owned[i]);
}

// The cheapest split of the phases into stages for a brick that owns `owned` (bricks > 1): for every
// end of a stage one backward walk prices its starts, up to kLongest phases back (the longest stage of
// any measured plan that paid was 9).  A walk ends where its stage no longer fits; false when none does.
constexpr int kLongest = 10;
template <class Mine> bool chooseStages(const Phases& ph, const std::vector<int>& owned, Team& team, Mine&& mine, int maxLocal, std::vector<char>& before) {
    const int P = ph.count;
    struct Price { double work; int imports; };
    std::vector<Price> price((size_t)(P + 1) * kLongest, Price{0., -1});   // [end][phases back - 1]
    team.run(P, [&](int at, int worker) {
        const int end = P - at;   // the longest walks first
        Scratch& s = mine(worker);
        startWalk(s, owned.data(), (int)owned.size());
        double work = 0.;
        for (int p = end - 1; p >= std::max(0, end - kLongest); p--) {
            const int count = widen(ph, p, s, nullptr);
            work += ph.isEdge(p) ? kEdgePhase + kEdgeEach * count
                    : ph.reverse ? kReverseTetPhase + kReverseTetEach * count : kTetPhase + kTetEach * count;
            if ((int)s.need.size() > maxLocal && p < end - 1) break;
            price[(size_t)end * kLongest + (end - 1 - p)] = {work, (int)(s.need.size() - owned.size())};
        }
    });
    std::vector<double> best(P + 1, 1e30);
    std::vector<int> from(P + 1, 0);
    best[0] = 0.;
    for (int end = 1; end <= P; end++)
        for (int p = end - 1; p >= std::max(0, end - kLongest); p--) {
            const Price& q = price[(size_t)end * kLongest + (end - 1 - p)];
            if (q.imports < 0) break;
            const double c = best[p] + q.work + kExchange + kImportEach * (double)q.imports;
            if (c < best[end]) { best[end] = c; from[end] = p; }
        }
    before.assign(P, 0);
    for (int e = P; e > 0; e = from[e]) before[from[e]] = 1;
    return best[P] < 1e30;
}

struct Split { int a, b, c; };
constexpr int kOneBrick = 800;

// One brick while its tables are made: the elements of its phases and the nodes it takes and gives by stage.
struct Build {
    const int* owned; int nOwned;
    std::vector<int> elements, phaseAt, phaseCount;   // phase p: elements[phaseAt[p] .. + phaseCount[p])
    std::vector<int> imports, importAt;               // stage st: imports[importAt[st] .. importAt[st + 1])
    std::vector<int> halo, exports, exportAt, ownTet;
};

}  // namespace

// A thread takes about 64 nodes' share of a plan to pay for itself; a mesh that is one brick has none to share.
int planThreads(int N, const int* active, int forced) {
    const int count = (int)std::count_if(active, active + N, [](int a) { return a != 0; });
    return forced == 1 || (forced == 0 && count <= kOneBrick) ? 1 : std::min(16, 1 + count / 64);
}

BrickPlan buildBrickPlan(const BrickMesh& m, int maxBricks, int maxLocal, int forced, bool wholeHalo, bool reverse, Team& team) {
    BrickPlan none;
    maxLocal = std::min(maxLocal, kBrickMaxLocal);
    const int nT = m.nTetColors * (1 + m.tensilePasses), P = m.nEdgeColors + nT;
    if (P == 0 || P > 128 || m.N <= 0) return none;
    int active = 0;
    for (int i = 0; i < m.N; i++) active += m.active[i] != 0;
    if ((active + maxBricks - 1) / maxBricks > maxLocal) return none;   // before anything is sized by the mesh
    const Phases ph(m, reverse, team);
    std::vector<std::unique_ptr<Scratch>> scratch(team.threads());
    const int widest = ph.widest();
    auto mine = [&](int worker) -> Scratch& {
        if (!scratch[worker]) scratch[worker].reset(new Scratch(m.N, widest));
        return *scratch[worker];
    };
    // nodes the bricks serve: active ones and ends of any element; the rest never meet a constraint
    std::vector<unsigned char> used(m.N);
    struct Box { int lo[3], hi[3], served; };
    const int chunk = 4096, chunks = (m.N + chunk - 1) / chunk;
    std::vector<Box> part(chunks);
    team.run(chunks, [&](int q, int) {
        const int i0 = q * chunk, i1 = std::min(m.N, i0 + chunk);
        for (int i = i0; i < i1; i++) used[i] = m.active[i] != 0 || ph.ends[i].load(std::memory_order_relaxed) != 0;
        Box b{{m.nx, m.ny, m.nz}, {-1, -1, -1}, 0};
        int c[3] = {i0 % m.nx, i0 / m.nx % m.ny, i0 / (m.nx * m.ny)};
        for (int i = i0; i < i1; i++) {
            if (used[i]) {
                b.served++;
                for (int a = 0; a < 3; a++) { b.lo[a] = std::min(b.lo[a], c[a]); b.hi[a] = std::max(b.hi[a], c[a]); }
            }
            if (++c[0] == m.nx) { c[0] = 0; if (++c[1] == m.ny) { c[1] = 0; c[2]++; } }
        }
        part[q] = b;
    });
    int lo[3] = {m.nx, m.ny, m.nz}, hi[3] = {-1, -1, -1}, served = 0;
    for (const Box& b : part) {
        served += b.served;
        for (int a = 0; a < 3; a++) { lo[a] = std::min(lo[a], b.lo[a]); hi[a] = std::max(hi[a], b.hi[a]); }
    }
    if (served == 0) return none;
    if ((served + maxBricks - 1) / maxBricks > maxLocal) return none;
    const int ext[3] = {hi[0] - lo[0] + 1, hi[1] - lo[1] + 1, hi[2] - lo[2] + 1};
    // the box grid of at most `count` bricks whose widest brick with two cells of halo is smallest
    auto boxes = [&](int count) {
        Split best{1, 1, 1};
        double cost = 1e30;
        for (int a = 1; a <= std::min(count, ext[0]); a++)
            for (int b = 1; a * b <= count && b <= ext[1]; b++) {
                const int c = std::min(count / (a * b), ext[2]);
                auto side = [&](int n, int parts) { const double w = std::ceil((double)n / parts); return parts == 1 ? w : std::min(w + 4., n + 0.); };
                const double v = side(ext[0], a) * side(ext[1], b) * side(ext[2], c);
                if (v < cost) { cost = v; best = {a, b, c}; }
            }
        return best;
    };
    // One brick, or one per SM: a mesh of up to kOneBrick nodes runs its colours faster in one CTA without any
    // exchange, beyond that more CTAs are faster (us a substep on one brick and on one per SM: 360 nodes 24.0
    // and 27.7, 600 26.4 and 29.1, 847 30.0 and 29.5, 1176 34.7 and 29.2, 2601 60 and 33; 8 bricks lie between).
    const int count = forced > 0 ? std::min(forced, maxBricks) : served <= kOneBrick ? 1 : maxBricks;
    const Split split = boxes(count);
    const int B = split.a * split.b * split.c;
    if (B == 1 && served > maxLocal) return none;
    // owners, and every brick's own nodes in order
    std::vector<int> slice[3];   // brick coordinate of a lattice coordinate, times its stride
    const int parts[3] = {split.a, split.b, split.c}, stride[3] = {1, split.a, split.a * split.b}, dims[3] = {m.nx, m.ny, m.nz};
    for (int a = 0; a < 3; a++) {
        slice[a].assign(dims[a], 0);
        for (int x = lo[a]; x <= hi[a]; x++) slice[a][x] = (x - lo[a]) * parts[a] / ext[a] * stride[a];
    }
    BrickPlan plan;
    std::vector<int> ownerOf(m.N, -1), ownedAt(B + 1, 0), ownedNodes(served);
    auto eachNode = [&](auto&& body) {
        for (int z = 0, i = 0; z < m.nz; z++)
            for (int y = 0; y < m.ny; y++) {
                const int yz = slice[1][y] + slice[2][z];
                for (int x = 0; x < m.nx; x++, i++) body(i, used[i] ? slice[0][x] + yz : -1);
            }
    };
    eachNode([&](int i, int b) { if (b >= 0) ownedAt[b + 1]++; else plan.idle.push_back(i); });
    for (int b = 0; b < B; b++) ownedAt[b + 1] += ownedAt[b];
    {
        std::vector<int> cursor(ownedAt.begin(), ownedAt.end() - 1);
        eachNode([&](int i, int b) { if (b >= 0) { ownerOf[i] = b; ownedNodes[cursor[b]++] = i; } });
    }
    std::vector<char> before(P, 0);
    std::vector<int> stageStart;
    const int mid = split.a / 2 + split.a * (split.b / 2 + split.b * (split.c / 2));   // the brick with the most halo
    if (B > 1) {
        // the brick at the middle of the grid stands for all
        const std::vector<int> owned(ownedNodes.begin() + ownedAt[mid], ownedNodes.begin() + ownedAt[mid + 1]);
        if (owned.empty() || (int)owned.size() > maxLocal) return none;
        if (!chooseStages(ph, owned, team, mine, maxLocal, before)) return none;
    }
    before[0] = 1;
    for (int p = 0; p < P; p++) if (before[p]) stageStart.push_back(p);
    const int S = (int)stageStart.size();
    stageStart.push_back(P);
    std::vector<Build> build(B);
    // which bricks take values from which (rows: the reader)
    std::vector<unsigned char> reads((size_t)B * B, 0);
    std::atomic<bool> fits{true};
    std::atomic<size_t> likely[2] = {{0}, {0}};   // sizes of a brick's lists, as far as seen
    auto walk = [&](int b, int worker) {
        if (!fits.load(std::memory_order_relaxed)) return;
        Scratch& s = mine(worker);
        Build& q = build[b];
        q.owned = ownedNodes.data() + ownedAt[b]; q.nOwned = ownedAt[b + 1] - ownedAt[b];
        q.phaseAt.assign(P, 0); q.phaseCount.assign(P, 0); q.importAt.assign(1, 0);
        q.elements.reserve(likely[0].load(std::memory_order_relaxed)); q.imports.reserve(likely[1].load(std::memory_order_relaxed));
        int local = q.nOwned;
        for (int st = 0; st < S; st++) {
            startWalk(s, q.owned, q.nOwned);
            for (int p = stageStart[st + 1] - 1; p >= stageStart[st]; p--) {
                q.phaseAt[p] = (int)q.elements.size();
                q.phaseCount[p] = widen(ph, p, s, &q.elements);
            }
            for (size_t i = q.nOwned; i < s.need.size(); i++) {
                const int n = s.need[i];
                q.imports.push_back(n);
                reads[(size_t)b * B + ownerOf[n]] = 1;
                if (s.halo.add(n)) local++;
            }
            q.importAt.push_back((int)q.imports.size());
        }
        s.halo.drain([](int) {});
        likely[0].store(std::max(likely[0].load(std::memory_order_relaxed), q.elements.size()), std::memory_order_relaxed);
        likely[1].store(std::max(likely[1].load(std::memory_order_relaxed), q.imports.size()), std::memory_order_relaxed);
        if (local > maxLocal) fits.store(false, std::memory_order_relaxed);
    };
    const bool asked = served > maxLocal;   // a mesh that does not fit is told by its middle brick
    if (asked) {
        walk(mid, 0);
        if (!fits) return none;
    }
    team.run(B, [&](int b, int worker) { if (!asked || b != mid) walk(b, worker); });
    if (!fits) return none;
    // Neighbours take values from each other in every stage: a brick may overwrite a published value
    // two exchanges later, which is safe only once its readers have published their next ones.
    for (int a = 0; a < B; a++)
        for (int b = 0; b < a; b++)
            reads[(size_t)a * B + b] = reads[(size_t)b * B + a] = reads[(size_t)a * B + b] | reads[(size_t)b * B + a];
    const std::unique_ptr<std::atomic<unsigned char>[]> exported(new std::atomic<unsigned char>[(size_t)S * m.N]());   // [stage][node]: some neighbour takes it
    team.run(B, [&](int b, int worker) {
        Scratch& s = mine(worker);
        Build& q = build[b];
        std::vector<int> raw;
        raw.swap(q.imports);
        const std::vector<int> rawAt = q.importAt;
        q.imports.reserve(raw.size() + (wholeHalo ? raw.size() : 0) + (size_t)S * 26);
        std::vector<unsigned char> met(B);
        for (int st = 0; st < S; st++) {
            std::fill(met.begin(), met.end(), 0);
            const int hiEnd = st == 0 && wholeHalo ? rawAt[S] : rawAt[st + 1];   // the first exchange takes every halo node
            for (int i = rawAt[st]; i < hiEnd; i++) { met[ownerOf[raw[i]]] = 1; s.nodes.add(raw[i]); }
            for (int c = 0; c < B; c++) if (reads[(size_t)b * B + c] && !met[c]) s.nodes.add(ownedNodes[ownedAt[c]]);
            s.nodes.drain([&](int n) {
                q.imports.push_back(n);
                s.halo.add(n);
                exported[(size_t)st * m.N + n].store(1, std::memory_order_relaxed);
            });
            q.importAt[st + 1] = (int)q.imports.size();
        }
        s.halo.drain([&](int n) { q.halo.push_back(n); });
    });
    team.run(B, [&](int b, int) {
        Build& q = build[b];
        q.exportAt.assign(1, 0);
        for (int st = 0; st < S; st++) {
            const std::atomic<unsigned char>* e = exported.get() + (size_t)st * m.N;
            for (int i = 0; i < q.nOwned; i++) if (e[q.owned[i]].load(std::memory_order_relaxed)) q.exports.push_back(q.owned[i]);
            q.exportAt.push_back((int)q.exports.size());
        }
    });
    // table offsets, then the tables brick by brick
    const int headWords = m.nEdgeColors + 1 + nT + 1 + 2 * (S + 1);
    plan.desc.resize(B);
    plan.head.resize((size_t)B * headWords);
    int nNode = 0, nEdge = 0, nTet = 0, nImp = 0, nExp = 0;
    // phase of the c-th edge and tet colour of the sweep
    auto edgePhase = [&](int c) { return reverse ? nT + c : c; };
    auto tetPhase = [&](int c) { return reverse ? c : m.nEdgeColors + c; };
    for (int b = 0; b < B; b++) {
        const Build& q = build[b];
        int* h = plan.head.data() + (size_t)b * headWords;
        plan.desc[b] = {nNode, q.nOwned, q.nOwned + (int)q.halo.size(), b * headWords, 0, 0, 0};
        nNode += plan.desc[b].nLocal;
        for (int c = 0; c < m.nEdgeColors; c++) { *h++ = nEdge; nEdge += q.phaseCount[edgePhase(c)]; }
        *h++ = nEdge;
        for (int c = 0; c < nT; c++) { *h++ = nTet; nTet += q.phaseCount[tetPhase(c)]; }
        *h++ = nTet;
        for (int st = 0; st <= S; st++) *h++ = nImp + q.importAt[st];
        nImp += q.importAt[S];
        for (int st = 0; st <= S; st++) *h++ = nExp + q.exportAt[st];
        nExp += q.exportAt[S];
        plan.maxLocal = std::max(plan.maxLocal, plan.desc[b].nLocal);
        plan.maxOwned = std::max(plan.maxOwned, q.nOwned);
        plan.maxList = std::max(plan.maxList, q.importAt[S] + q.exportAt[S]);
        for (int p = 0; p < P; p++) {
            plan.threads = std::max(plan.threads, (q.phaseCount[p] + 31) / 32 * 32);
            if (!ph.isEdge(p)) plan.tetWidth = std::max(plan.tetWidth, q.phaseCount[p]);
        }
    }
    if (plan.maxLocal > maxLocal) return none;
    plan.localNode.resize(nNode); plan.importList.resize(nImp); plan.exportList.resize(nExp);
    plan.edgeWord.resize(nEdge); plan.edgeRest.resize(nEdge); plan.edgeSrc.resize(nEdge);
    plan.tetWord.resize(nTet); plan.tetSrc.resize(nTet);
    team.run(B, [&](int b, int worker) {
        int* local = mine(worker).localOf.get();
        Build& q = build[b];
        const BrickDesc& d = plan.desc[b];
        const int* h = plan.head.data() + d.head;
        const int* edgeOff = h; const int* tetOff = h + m.nEdgeColors + 1;
        const int* impOff = tetOff + nT + 1; const int* expOff = impOff + S + 1;
        std::copy(q.owned, q.owned + q.nOwned, plan.localNode.begin() + d.nodeBase);
        std::copy(q.halo.begin(), q.halo.end(), plan.localNode.begin() + d.nodeBase + d.nOwned);
        for (int l = 0; l < d.nLocal; l++) local[plan.localNode[d.nodeBase + l]] = l;
        for (int c = 0; c < m.nEdgeColors; c++) {
            const int* list = q.elements.data() + q.phaseAt[edgePhase(c)];
            for (int at = edgeOff[c]; at < edgeOff[c + 1]; at++, list++) {
                const int2 e = m.edgeEnds[*list];
                plan.edgeWord[at] = (unsigned)local[e.x] | (unsigned)local[e.y] << kBrickNodeBits | kBrickEdgeLive |
                                    (ownerOf[e.x] == b ? kBrickEdgeOwner : 0u);
                plan.edgeRest[at] = m.edgeRest[*list];
                plan.edgeSrc[at] = *list;
            }
        }
        for (int c = 0; c < nT; c++) {
            const int* list = q.elements.data() + q.phaseAt[tetPhase(c)];
            for (int at = tetOff[c]; at < tetOff[c + 1]; at++, list++) {
                const int4 t = m.tetIds[*list];
                const bool own = ownerOf[t.x] == b;
                plan.tetWord[at] = (uint64_t)local[t.x] | (uint64_t)local[t.y] << kBrickNodeBits | (uint64_t)local[t.z] << (2 * kBrickNodeBits) |
                                   (uint64_t)local[t.w] << (3 * kBrickNodeBits) | (uint64_t)(m.tetMeta[*list] & 7) << 56 | kBrickTetLive |
                                   (own ? kBrickTetOwner : 0ull);
                plan.tetSrc[at] = *list;
                if (m.tensilePasses > 0 && c < m.nTetColors && own) q.ownTet.push_back(at);
            }
        }
        for (int i = 0; i < q.importAt[S]; i++) plan.importList[impOff[0] + i] = make_int2(local[q.imports[i]], q.imports[i]);
        for (int i = 0; i < q.exportAt[S]; i++) plan.exportList[expOff[0] + i] = make_int2(local[q.exports[i]], q.exports[i]);
        std::vector<int> own;
        own.swap(q.ownTet);
        q = Build();   // given back by the threads that filled them
        q.ownTet.swap(own);
    });
    for (int b = 0; b < B && m.tensilePasses > 0; b++) {
        plan.desc[b].ownFirst = (int)plan.ownTet.size();
        plan.desc[b].nOwn = (int)build[b].ownTet.size();
        plan.ownTet.insert(plan.ownTet.end(), build[b].ownTet.begin(), build[b].ownTet.end());
    }
    plan.meshEdges = m.nEdgeColors ? m.edgeOff[m.nEdgeColors] : 0; plan.meshTets = m.nTetColors ? m.tetOff[m.nTetColors] : 0;
    plan.bricks = B; plan.asked = count; plan.stages = S; plan.nEdgeColors = m.nEdgeColors; plan.nTetColors = nT; plan.tensilePasses = m.tensilePasses;
    for (int p = 0; p < P; p++) if (before[p] && B > 1) plan.exchangeBefore[p >> 6] |= 1ull << (p & 63);
    return plan;
}

}  // namespace gbt
