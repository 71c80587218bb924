// Checks of the brick planner on the host: every index of a plan's tables is in range, every value a brick
// reads in a stage is one it owns or has taken in that stage from an owner that gave it, and one sweep of the
// bricks leaves every node as one sweep of the whole mesh does (values are hashes, so any wrong order, missing
// element or stale value shows).
//   brick_plan_check dx dy dz hole-permille forced max-local whole reverse tensile-passes
// prints "bricks stages" and exits 0, or prints what is wrong and exits 1.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "brick_plan.h"
#include "host_parallel.h"

using namespace gbt;
typedef unsigned long long u64;

static const int kKuhn[6][4] = {{0, 1, 3, 7}, {0, 3, 2, 7}, {0, 2, 6, 7}, {0, 6, 4, 7}, {0, 4, 5, 7}, {0, 5, 1, 7}};
[[noreturn]] static void wrong(const char* what) { printf("%s\n", what); exit(1); }
static void expect(bool ok, const char* what) { if (!ok) wrong(what); }
static u64 mix(u64 a, u64 b) {
    u64 x = a * 0x9E3779B97F4A7C15ull ^ (b + 0x7F4A7C15ull + (a << 6) + (a >> 2));
    x ^= x >> 29; x *= 0xBF58476D1CE4E5B9ull; x ^= x >> 32;
    return x;
}
// The stand-in for a projection: every node of the element becomes a function of all of them.
static void project(u64* value, const int* node, int n, u64 key) {
    u64 all = key;
    for (int j = 0; j < n; j++) all = mix(all, value[node[j]]);
    for (int j = 0; j < n; j++) value[node[j]] = mix(all, value[node[j]] + j);
}

// A lattice with some nodes inactive: its edges, its cells' tets, each coloured greedily, in colour order.
struct Mesh {
    int nx, ny, nz, N;
    std::vector<int> active, edgeOff, tetOff, meta; std::vector<int2> edges; std::vector<float> rest; std::vector<int4> tets;
};
static std::vector<int> colourOrder(int N, const std::vector<std::vector<int>>& elements, std::vector<int>& off) {
    std::vector<u64> taken(N, 0);
    std::vector<int> colour(elements.size());
    int colours = 0;
    for (size_t e = 0; e < elements.size(); e++) {
        u64 busy = 0;
        for (int n : elements[e]) busy |= taken[n];
        colour[e] = __builtin_ctzll(~busy);
        colours = std::max(colours, colour[e] + 1);
        for (int n : elements[e]) taken[n] |= 1ull << colour[e];
    }
    off.assign(colours + 1, 0);
    for (int c : colour) off[c + 1]++;
    for (int c = 0; c < colours; c++) off[c + 1] += off[c];
    std::vector<int> at(off.begin(), off.end() - 1), order(elements.size());
    for (size_t e = 0; e < elements.size(); e++) order[at[colour[e]]++] = (int)e;
    return order;
}
static Mesh lattice(int dx, int dy, int dz, int hole) {
    Mesh m;
    m.nx = dx + 1; m.ny = dy + 1; m.nz = dz + 1; m.N = m.nx * m.ny * m.nz;
    std::mt19937 random(5);
    m.active.assign(m.N, 1);
    for (int& a : m.active) a = (int)(random() % 1000) >= hole;
    std::vector<std::vector<int>> edges, tets;
    std::vector<int> kind;
    const int step[3] = {1, m.nx, m.nx * m.ny}, dims[3] = {dx, dy, dz};
    for (int p = 0; p < m.N; p++) {
        const int c[3] = {p % m.nx, p / m.nx % m.ny, p / step[2]};
        for (int a = 0; a < 3; a++) if (c[a] < dims[a] && m.active[p] && m.active[p + step[a]]) edges.push_back({p, p + step[a]});
        if (c[0] == dx || c[1] == dy || c[2] == dz) continue;
        int corner[8];
        bool full = true;
        for (int q = 0; q < 8; q++) { corner[q] = p + (q & 1) + (q >> 1 & 1) * step[1] + (q >> 2) * step[2]; full = full && m.active[corner[q]]; }
        for (int t = 0; full && t < 6; t++) { tets.push_back({corner[kKuhn[t][0]], corner[kKuhn[t][1]], corner[kKuhn[t][2]], corner[kKuhn[t][3]]}); kind.push_back(t); }
    }
    for (int e : colourOrder(m.N, edges, m.edgeOff)) { m.edges.push_back(make_int2(edges[e][0], edges[e][1])); m.rest.push_back(1.f + e); }
    for (int t : colourOrder(m.N, tets, m.tetOff)) { m.tets.push_back(make_int4(tets[t][0], tets[t][1], tets[t][2], tets[t][3])); m.meta.push_back(kind[t] | 8); }
    return m;
}

int main(int argc, char** argv) {
    if (argc != 10) wrong("nine arguments");
    int arg[9];
    for (int i = 0; i < 9; i++) arg[i] = atoi(argv[i + 1]);
    const int forced = arg[4], maxLocal = arg[5], passes = arg[8];
    const bool whole = arg[6] != 0, reverse = arg[7] != 0;
    const Mesh m = lattice(arg[0], arg[1], arg[2], arg[3]);
    const BrickMesh bm{m.N, m.nx, m.ny, m.nz, m.active.data(), (int)m.edgeOff.size() - 1, (int)m.tetOff.size() - 1, m.edgeOff.data(), m.edges.data(),
                       m.rest.data(), m.tetOff.data(), m.tets.data(), m.meta.data(), passes};
    Team team(planThreads(bm.N, bm.active, forced));
    const BrickPlan p = buildBrickPlan(bm, 152, maxLocal, forced, whole, reverse, team);
    team.dismiss();
    printf("%d %d\n", p.bricks, p.stages);
    if (!p.ok()) return 0;
    const int B = p.bricks, S = p.stages, nE = bm.nEdgeColors, nT = bm.nTetColors * (1 + passes), P = nE + nT;
    expect(B <= 152 && p.nEdgeColors == nE && p.nTetColors == nT && p.maxLocal <= maxLocal, "shape");
    // every node is owned once or idle, and a brick's tables name its own nodes
    std::vector<int> owner(m.N, -1);
    for (int b = 0; b < B; b++)
        for (int l = 0; l < p.desc[b].nLocal; l++) {
            const int n = p.localNode[p.desc[b].nodeBase + l];
            expect(n >= 0 && n < m.N, "local node out of range");
            if (l < p.desc[b].nOwned) { expect(owner[n] == -1, "owned twice"); owner[n] = b; }
        }
    for (int n : p.idle) { expect(owner[n] == -1 && !m.active[n], "idle node"); owner[n] = -2; }
    for (int n = 0; n < m.N; n++) expect(owner[n] != -1, "node lost");
    struct Tables { const int *edge, *tet, *imports, *exports; };
    std::vector<Tables> t(B);
    std::vector<std::vector<u64>> value(B);
    std::vector<std::vector<char>> first(B);   // taken by the first exchange
    std::vector<u64> start(m.N), mail(m.N), single;
    for (int n = 0; n < m.N; n++) start[n] = mix(n, 77);
    single = start;
    for (int b = 0; b < B; b++) {
        const int* h = p.head.data() + p.desc[b].head;
        t[b] = {h, h + nE + 1, h + nE + 1 + nT + 1, h + nE + 1 + nT + 1 + S + 1};
        expect(t[b].edge[nE] <= (int)p.edgeWord.size() && t[b].tet[nT] <= (int)p.tetWord.size() && t[b].imports[S] <= (int)p.importList.size() &&
               t[b].exports[S] <= (int)p.exportList.size(), "table offsets");
        expect(t[b].imports[S] - t[b].imports[0] + t[b].exports[S] - t[b].exports[0] <= p.maxList, "exchange lists");
        expect(p.desc[b].nLocal <= p.maxLocal && p.desc[b].nOwned <= p.maxOwned, "node counts");
        value[b].assign(p.desc[b].nLocal, ~0ull);
        first[b].assign(p.desc[b].nLocal, 0);
        for (int l = 0; l < p.desc[b].nOwned; l++) value[b][l] = start[p.localNode[p.desc[b].nodeBase + l]];
    }
    int stage = 0;
    std::vector<char> neighbours, seen((size_t)B * B);
    for (int phase = 0; phase < P; phase++) {
        const bool edge = reverse ? phase >= nT : phase < nE;
        const int at = reverse ? (edge ? phase - nT : phase) : (edge ? phase : phase - nE);   // among the sweep's edge or tet colours
        const int colour = reverse ? (edge ? nE : nT) - 1 - at : at;
        if (p.exchangeBefore[phase >> 6] >> (phase & 63) & 1) {
            std::vector<char> given(m.N, 0);
            for (int b = 0; b < B; b++)
                for (int i = t[b].exports[stage]; i < t[b].exports[stage + 1]; i++) {
                    const int2 e = p.exportList[i];
                    expect(e.x >= 0 && e.x < p.desc[b].nOwned && p.localNode[p.desc[b].nodeBase + e.x] == e.y, "export");
                    mail[e.y] = value[b][e.x]; given[e.y] = 1;
                }
            std::fill(seen.begin(), seen.end(), 0);
            for (int b = 0; b < B; b++)
                for (int i = t[b].imports[stage]; i < t[b].imports[stage + 1]; i++) {
                    const int2 e = p.importList[i];
                    expect(e.x >= p.desc[b].nOwned && e.x < p.desc[b].nLocal && p.localNode[p.desc[b].nodeBase + e.x] == e.y, "import");
                    expect(given[e.y], "taken but not given");
                    value[b][e.x] = mail[e.y];
                    if (stage == 0) first[b][e.x] = 1;
                    seen[(size_t)b * B + owner[e.y]] = 1;
                }
            for (int a = 0; a < B; a++) for (int b = 0; b < B; b++) expect(seen[(size_t)a * B + b] == seen[(size_t)b * B + a], "one-way neighbours");
            expect(stage == 0 || seen == neighbours, "neighbours differ between exchanges");
            if (stage == 0) neighbours = seen;
            stage++;
        }
        const int meshColour = edge ? colour : colour % bm.nTetColors;
        if (edge) for (int k = m.edgeOff[meshColour]; k < m.edgeOff[meshColour + 1]; k++) project(single.data(), &m.edges[k].x, 2, k);
        else for (int k = m.tetOff[meshColour]; k < m.tetOff[meshColour + 1]; k++) project(single.data(), &m.tets[k].x, 4, k + (1ull << 40));
        for (int b = 0; b < B; b++) {
            const int* off = edge ? t[b].edge : t[b].tet;
            expect((off[at + 1] - off[at] + 31) / 32 * 32 <= p.threads && (edge || off[at + 1] - off[at] <= p.tetWidth), "phase width");
            for (int k = off[at]; k < off[at + 1]; k++) {
                int node[4];
                const int n = edge ? 2 : 4, src = edge ? p.edgeSrc[k] : p.tetSrc[k];
                expect(src >= 0 && src < (int)(edge ? m.edges.size() : m.tets.size()), "element");
                const int* ends = edge ? &m.edges[src].x : &m.tets[src].x;
                for (int j = 0; j < n; j++) {
                    node[j] = (int)((edge ? (u64)p.edgeWord[k] : p.tetWord[k]) >> (kBrickNodeBits * j) & kBrickNodeMask);
                    expect(node[j] < p.desc[b].nLocal && p.localNode[p.desc[b].nodeBase + node[j]] == ends[j], "element node");
                    expect(!whole || node[j] < p.desc[b].nOwned || first[b][node[j]], "not in the first exchange");
                }
                if (edge) expect((p.edgeWord[k] & kBrickEdgeLive) && !!(p.edgeWord[k] & kBrickEdgeOwner) == (owner[ends[0]] == b) && p.edgeRest[k] == m.rest[src], "edge word");
                else expect((p.tetWord[k] & kBrickTetLive) && !!(p.tetWord[k] & kBrickTetOwner) == (owner[ends[0]] == b) && (int)(p.tetWord[k] >> 56 & 7) == (m.meta[src] & 7), "tet word");
                project(value[b].data(), node, n, edge ? src : src + (1ull << 40));
            }
        }
    }
    expect(B == 1 || stage == S, "stages");
    for (int b = 0; b < B; b++)
        for (int l = 0; l < p.desc[b].nOwned; l++) expect(value[b][l] == single[p.localNode[p.desc[b].nodeBase + l]], "another value than one sweep of the mesh");
    if (passes > 0) {   // every tet is some brick's own, once
        std::vector<int> own(m.tets.size(), 0);
        for (int b = 0; b < B; b++)
            for (int i = 0; i < p.desc[b].nOwn; i++) {
                const int k = p.ownTet[p.desc[b].ownFirst + i];
                expect(k >= t[b].tet[0] && k < t[b].tet[bm.nTetColors], "own tet");
                own[p.tetSrc[k]]++;
            }
        expect(std::all_of(own.begin(), own.end(), [](int n) { return n == 1; }), "own tets");
    }
    return 0;
}
