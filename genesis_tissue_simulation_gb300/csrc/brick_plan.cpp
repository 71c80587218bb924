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
#include <algorithm>
#include <atomic>
#include <cmath>

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
    std::vector<int> at;   // [count x N] element of the phase at the node, or -1
    Phases(const BrickMesh& mesh, bool rev) : m(mesh), reverse(rev), nT(mesh.nTetColors * (1 + mesh.tensilePasses)), count(mesh.nEdgeColors + nT) {
        at.assign((size_t)count * m.N, -1);
        for (int p = 0; p < count; p++) {
            int* a = at.data() + (size_t)p * m.N;
            int lo, hi;
            range(p, lo, hi);
            for (int k = lo; k < hi; k++)
                if (isEdge(p)) { a[m.edgeEnds[k].x] = k; a[m.edgeEnds[k].y] = k; }
                else { const int4 t = m.tetIds[k]; a[t.x] = k; a[t.y] = k; a[t.z] = k; a[t.w] = k; }
        }
    }
    bool isEdge(int p) const { return reverse ? p >= nT : p < m.nEdgeColors; }
    int colour(int p) const {   // of the mesh (a tensile pass repeats the tet colours)
        if (!reverse) return p < m.nEdgeColors ? p : (p - m.nEdgeColors) % m.nTetColors;
        return p < nT ? (nT - 1 - p) % m.nTetColors : m.nEdgeColors - 1 - (p - nT);
    }
    int pass(int p) const { return isEdge(p) ? 0 : (reverse ? nT - 1 - p : p - m.nEdgeColors) / m.nTetColors; }
    void range(int p, int& lo, int& hi) const {
        const int* off = isEdge(p) ? m.edgeOff : m.tetOff;
        lo = off[colour(p)]; hi = off[colour(p) + 1];
    }
    int nodes(int p, int k, int out[4]) const {
        if (isEdge(p)) { out[0] = m.edgeEnds[k].x; out[1] = m.edgeEnds[k].y; return 2; }
        const int4 t = m.tetIds[k];
        out[0] = t.x; out[1] = t.y; out[2] = t.z; out[3] = t.w;
        return 4;
    }
};

// Marks with a generation, so that clearing a set is one increment.
struct Marks {
    std::vector<unsigned> at; unsigned now = 0;
    explicit Marks(size_t n) : at(n, 0) {}
    void clear() { now++; }
    bool add(int i) { if (at[i] == now) return false; at[i] = now; return true; }
    bool has(int i) const { return at[i] == now; }
};

struct Scratch {
    Marks node, edge, tet;
    Scratch(int N, int E, int T) : node(N), edge(E), tet(T) {}
};

// One step of the backward walk: the elements of phase p that touch `need`, whose nodes join it.
void widen(const Phases& ph, int p, std::vector<int>& need, Scratch& s, std::vector<int>* elements, int& count) {
    const int* at = ph.at.data() + (size_t)p * ph.m.N;
    Marks& seen = ph.isEdge(p) ? s.edge : s.tet;
    const int mark0 = ph.isEdge(p) ? 0 : ph.pass(p) * ph.m.tetOff[ph.m.nTetColors];   // a tet once per pass
    count = 0;
    const size_t had = need.size();
    for (size_t i = 0; i < had; i++) {
        const int k = at[need[i]];
        if (k < 0 || !seen.add(mark0 + k)) continue;
        count++;
        if (elements) elements->push_back(k);
        int nd[4];
        const int c = ph.nodes(p, k, nd);
        for (int j = 0; j < c; j++) if (s.node.add(nd[j])) need.push_back(nd[j]);
    }
}

// The cheapest split of the phases into stages for a brick that owns `owned` (bricks > 1): for every
// end of a stage one backward walk prices its starts, up to kLongest phases back (the longest stage of
// any measured plan that paid was 9) and while the stage alone is cheaper than the whole sweep's bound.
constexpr int kLongest = 10;
double chooseStages(const Phases& ph, const std::vector<int>& owned, Scratch& s, int maxLocal, std::vector<char>& before) {
    const int P = ph.count;
    std::vector<double> best(P + 1, 1e30);
    std::vector<int> from(P + 1, 0);
    best[0] = 0.;
    for (int end = 1; end <= P; end++) {
        std::vector<int> need = owned;
        s.node.clear(); s.edge.clear(); s.tet.clear();
        for (int n : owned) s.node.add(n);
        double work = 0.;
        for (int p = end - 1; p >= std::max(0, end - kLongest); p--) {
            int count;
            widen(ph, p, need, s, nullptr, count);
            work += ph.isEdge(p) ? kEdgePhase + kEdgeEach * count
                    : ph.reverse ? kReverseTetPhase + kReverseTetEach * count : kTetPhase + kTetEach * count;
            if ((int)need.size() > maxLocal && p < end - 1) break;
            const double c = best[p] + work + kExchange + kImportEach * (double)(need.size() - owned.size());
            if (c < best[end]) { best[end] = c; from[end] = p; }
            if (work > best[end]) break;
        }
    }
    before.assign(P, 0);
    for (int e = P; e > 0; e = from[e]) before[from[e]] = 1;
    return best[P];
}

struct Split { int a, b, c; };
constexpr int kOneBrick = 800;

}  // namespace

BrickPlan buildBrickPlan(const BrickMesh& m, int maxBricks, int maxLocal, int forced, bool wholeHalo, bool reverse, int maxThreads) {
    BrickPlan none;
    maxLocal = std::min(maxLocal, kBrickMaxLocal);
    const int E = m.nEdgeColors ? m.edgeOff[m.nEdgeColors] : 0, T = m.nTetColors ? m.tetOff[m.nTetColors] : 0;
    const int nT = m.nTetColors * (1 + m.tensilePasses), P = m.nEdgeColors + nT;
    if (P == 0 || P > 128 || m.N <= 0) return none;
    // nodes the bricks serve: active ones and ends of any element; the rest never meet a constraint
    std::vector<unsigned char> used(m.N, 0);
    for (int i = 0; i < m.N; i++) used[i] = m.active[i] != 0;
    for (int k = 0; k < E; k++) used[m.edgeEnds[k].x] = used[m.edgeEnds[k].y] = 1;
    for (int k = 0; k < T; k++) { const int4 t = m.tetIds[k]; used[t.x] = used[t.y] = used[t.z] = used[t.w] = 1; }
    int lo[3] = {m.nx, m.ny, m.nz}, hi[3] = {-1, -1, -1}, served = 0;
    for (int i = 0; i < m.N; i++) {
        if (!used[i]) continue;
        served++;
        const int c[3] = {i % m.nx, i / m.nx % m.ny, i / (m.nx * m.ny)};
        for (int a = 0; a < 3; a++) { lo[a] = std::min(lo[a], c[a]); hi[a] = std::max(hi[a], c[a]); }
    }
    if (served == 0) return none;
    if ((served + maxBricks - 1) / maxBricks > maxLocal) return none;   // before anything is sized by the mesh
    const int ext[3] = {hi[0] - lo[0] + 1, hi[1] - lo[1] + 1, hi[2] - lo[2] + 1};
    Phases ph(m, reverse);
    Scratch s(m.N, std::max(E, 1), std::max(T * (1 + m.tensilePasses), 1));
    auto brickOf = [&](const Split& q, int i) {
        const int x = (i % m.nx - lo[0]) * q.a / ext[0], y = (i / m.nx % m.ny - lo[1]) * q.b / ext[1],
                  z = (i / (m.nx * m.ny) - lo[2]) * q.c / ext[2];
        return x + q.a * (y + q.b * z);
    };
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
    std::vector<char> before(P, 0);
    double cost = 0.;
    if (split.a * split.b * split.c == 1) {
        if (served > maxLocal) return none;
    } else {
        // the brick at the middle of the grid stands for all (it has the most halo)
        const int mid = split.a / 2 + split.a * (split.b / 2 + split.b * (split.c / 2));
        std::vector<int> owned;
        for (int i = 0; i < m.N; i++) if (used[i] && brickOf(split, i) == mid) owned.push_back(i);
        if (owned.empty() || (int)owned.size() > maxLocal) return none;
        cost = chooseStages(ph, owned, s, maxLocal, before);
    }
    if (cost >= 1e30) return none;

    BrickPlan plan;
    const int B = split.a * split.b * split.c;
    std::vector<int> stageStart;
    if (B == 1) before.assign(P, 0);
    before[0] = 1;
    for (int p = 0; p < P; p++) if (before[p]) stageStart.push_back(p);
    const int S = (int)stageStart.size();
    stageStart.push_back(P);
    std::vector<int> ownerOf(m.N, -1);
    std::vector<std::vector<int>> owned(B);
    for (int i = 0; i < m.N; i++) {
        if (!used[i]) { plan.idle.push_back(i); continue; }
        const int b = brickOf(split, i);
        ownerOf[i] = b;
        owned[b].push_back(i);
    }
    std::vector<std::vector<std::vector<int>>> elements(B, std::vector<std::vector<int>>(P)), imports(B, std::vector<std::vector<int>>(S));
    // body(brick, the thread's own workspace)
    auto parallel = [&](auto&& workspace, auto&& body) { parallelFor(B, std::min(maxThreads, 1 + served / 200), workspace, body); };
    // which bricks take values from which (rows: the reader)
    std::vector<unsigned char> reads((size_t)B * B, 0);
    parallel([&]() { return Scratch(m.N, std::max(E, 1), std::max(T * (1 + m.tensilePasses), 1)); }, [&](int b, Scratch& sc) {
        for (int st = 0; st < S; st++) {
            std::vector<int> need = owned[b];
            sc.node.clear(); sc.edge.clear(); sc.tet.clear();
            for (int n : need) sc.node.add(n);
            for (int p = stageStart[st + 1] - 1; p >= stageStart[st]; p--) {
                int count;
                widen(ph, p, need, sc, &elements[b][p], count);
                std::sort(elements[b][p].begin(), elements[b][p].end());
            }
            imports[b][st].assign(need.begin() + owned[b].size(), need.end());
            for (int n : imports[b][st]) reads[(size_t)b * B + ownerOf[n]] = 1;
        }
        if (wholeHalo)
            for (int st = 1; st < S; st++) imports[b][0].insert(imports[b][0].end(), imports[b][st].begin(), imports[b][st].end());
    });
    // Neighbours take values from each other in every stage: a brick may overwrite a published value
    // two exchanges later, which is safe only once its readers have published their next ones.
    for (int a = 0; a < B; a++)
        for (int b = 0; b < a; b++)
            reads[(size_t)a * B + b] = reads[(size_t)b * B + a] = reads[(size_t)a * B + b] | reads[(size_t)b * B + a];
    std::vector<std::vector<int>> halo(B);
    std::vector<std::atomic<unsigned char>> exported((size_t)S * m.N);   // [stage][node]: some neighbour takes it
    parallel([&]() { return std::make_pair(Marks(m.N), Marks(B)); }, [&](int b, std::pair<Marks, Marks>& mk) {
        Marks& seen = mk.first;
        Marks& met = mk.second;
        for (auto& list : imports[b]) {
            met.clear();
            for (int n : list) met.add(ownerOf[n]);
            for (int c = 0; c < B; c++) if (reads[(size_t)b * B + c] && !met.has(c)) list.push_back(owned[c][0]);
            std::sort(list.begin(), list.end());
            list.erase(std::unique(list.begin(), list.end()), list.end());
        }
        seen.clear();
        for (int st = 0; st < S; st++)
            for (int n : imports[b][st]) {
                if (seen.add(n)) halo[b].push_back(n);
                exported[(size_t)st * m.N + n].store(1, std::memory_order_relaxed);
            }
        std::sort(halo[b].begin(), halo[b].end());
    });
    std::vector<std::vector<std::vector<int>>> exports(B, std::vector<std::vector<int>>(S));
    for (int b = 0; b < B; b++) {
        for (int st = 0; st < S; st++)
            for (int n : owned[b]) if (exported[(size_t)st * m.N + n].load(std::memory_order_relaxed)) exports[b][st].push_back(n);
        plan.maxLocal = std::max(plan.maxLocal, (int)(owned[b].size() + halo[b].size()));
        plan.maxOwned = std::max(plan.maxOwned, (int)owned[b].size());
    }
    if (plan.maxLocal > maxLocal) return none;
    // table offsets, then the tables brick by brick
    const int headWords = m.nEdgeColors + 1 + nT + 1 + 2 * (S + 1);
    plan.desc.resize(B);
    plan.head.resize((size_t)B * headWords);
    int nNode = 0, nEdge = 0, nTet = 0, nImp = 0, nExp = 0;
    auto phaseOf = [&](bool edge, int colour) {
        if (!reverse) return edge ? colour : m.nEdgeColors + colour;
        return edge ? nT + (m.nEdgeColors - 1 - colour) : nT - 1 - colour;
    };
    for (int b = 0; b < B; b++) {
        int* h = plan.head.data() + (size_t)b * headWords;
        plan.desc[b] = {nNode, (int)owned[b].size(), (int)(owned[b].size() + halo[b].size()), b * headWords, 0, 0, 0};
        nNode += plan.desc[b].nLocal;
        // colours in sweep order
        for (int c = 0; c < m.nEdgeColors; c++) { *h++ = nEdge; nEdge += (int)elements[b][phaseOf(true, reverse ? m.nEdgeColors - 1 - c : c)].size(); }
        *h++ = nEdge;
        for (int c = 0; c < nT; c++) { *h++ = nTet; nTet += (int)elements[b][phaseOf(false, reverse ? nT - 1 - c : c)].size(); }
        *h++ = nTet;
        for (int st = 0; st < S; st++) { *h++ = nImp; nImp += (int)imports[b][st].size(); }
        *h++ = nImp;
        for (int st = 0; st < S; st++) { *h++ = nExp; nExp += (int)exports[b][st].size(); }
        *h++ = nExp;
    }
    plan.localNode.resize(nNode); plan.importList.resize(nImp); plan.exportList.resize(nExp);
    plan.edgeWord.resize(nEdge); plan.edgeRest.resize(nEdge); plan.edgeSrc.resize(nEdge);
    plan.tetWord.resize(nTet); plan.tetSrc.resize(nTet);
    parallel([&]() { return std::vector<int>(m.N); }, [&](int b, std::vector<int>& localOf) {
        const BrickDesc& d = plan.desc[b];
        const int* h = plan.head.data() + d.head;
        const int* edgeOff = h; const int* tetOff = h + m.nEdgeColors + 1;
        const int* impOff = tetOff + nT + 1; const int* expOff = impOff + S + 1;
        std::copy(owned[b].begin(), owned[b].end(), plan.localNode.begin() + d.nodeBase);
        std::copy(halo[b].begin(), halo[b].end(), plan.localNode.begin() + d.nodeBase + d.nOwned);
        for (int l = 0; l < d.nLocal; l++) localOf[plan.localNode[d.nodeBase + l]] = l;
        auto local = [&](int n) { return localOf[n]; };
        for (int c = 0; c < m.nEdgeColors; c++) {
            int at = edgeOff[c];
            for (int k : elements[b][phaseOf(true, reverse ? m.nEdgeColors - 1 - c : c)]) {
                const int2 e = m.edgeEnds[k];
                plan.edgeWord[at] = (unsigned)local(e.x) | (unsigned)local(e.y) << kBrickNodeBits | kBrickEdgeLive |
                                    (ownerOf[e.x] == b ? kBrickEdgeOwner : 0u);
                plan.edgeRest[at] = m.edgeRest[k];
                plan.edgeSrc[at++] = k;
            }
        }
        for (int c = 0; c < nT; c++) {
            int at = tetOff[c];
            for (int k : elements[b][phaseOf(false, reverse ? nT - 1 - c : c)]) {
                const int4 t = m.tetIds[k];
                plan.tetWord[at] = (uint64_t)local(t.x) | (uint64_t)local(t.y) << kBrickNodeBits | (uint64_t)local(t.z) << (2 * kBrickNodeBits) |
                                   (uint64_t)local(t.w) << (3 * kBrickNodeBits) | (uint64_t)(m.tetMeta[k] & 7) << 56 | kBrickTetLive |
                                   (ownerOf[t.x] == b ? kBrickTetOwner : 0ull);
                plan.tetSrc[at++] = k;
            }
        }
        for (int st = 0; st < S; st++) {
            int at = impOff[st];
            for (int n : imports[b][st]) plan.importList[at++] = make_int2(local(n), n);
            at = expOff[st];
            for (int n : exports[b][st]) plan.exportList[at++] = make_int2(local(n), n);
        }
    });
    for (int b = 0; b < B; b++) {
        int records = 0;
        for (int st = 0; st < S; st++) records += (int)(imports[b][st].size() + exports[b][st].size());
        plan.maxList = std::max(plan.maxList, records);
    }
    for (auto& lists : elements)
        for (int p = 0; p < P; p++) {
            plan.threads = std::max(plan.threads, ((int)lists[p].size() + 31) / 32 * 32);
            if (!ph.isEdge(p)) plan.tetWidth = std::max(plan.tetWidth, (int)lists[p].size());
        }
    if (m.tensilePasses > 0)
        for (int b = 0; b < B; b++) {
            const int* tetOff = plan.head.data() + plan.desc[b].head + m.nEdgeColors + 1;
            plan.desc[b].ownFirst = (int)plan.ownTet.size();
            for (int k = tetOff[0]; k < tetOff[m.nTetColors]; k++) if (plan.tetWord[k] & kBrickTetOwner) plan.ownTet.push_back(k);
            plan.desc[b].nOwn = (int)plan.ownTet.size() - plan.desc[b].ownFirst;
        }
    plan.bricks = B; plan.asked = count; plan.stages = S; plan.nEdgeColors = m.nEdgeColors; plan.nTetColors = nT; plan.tensilePasses = m.tensilePasses; plan.cost = cost;
    for (int p = 0; p < P; p++) if (before[p] && B > 1) plan.exchangeBefore[p >> 6] |= 1ull << (p & 63);
    return plan;
}

}  // namespace gbt
