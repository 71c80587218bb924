// The blade's ribbon tick: crossing test, cut marks, tear law and sever of lattice edges.
#pragma once
#include "tissue_device.cuh"

namespace gbt {

// ---------------------------------------------------------------------------------------------
// blade ribbon tick on one lattice edge: CCD crossing, tear law, sever (V/cut.cu:486-746)
// ---------------------------------------------------------------------------------------------
static __constant__ int kStencilOff[3][4][3] = {{{0, 0, 0}, {0, -1, 0}, {0, -1, -1}, {0, 0, -1}},
                                         {{0, 0, 0}, {0, 0, -1}, {-1, 0, -1}, {-1, 0, 0}},
                                         {{0, 0, 0}, {-1, 0, 0}, {-1, -1, 0}, {0, -1, 0}}};
static __constant__ int kStencilEdge[3][4] = {{0, 2, 6, 4}, {3, 7, 5, 1}, {8, 9, 10, 11}};

__device__ __forceinline__ int nodeId(const DeviceMesh& m, int x, int y, int z) { return x + (m.dx + 1) * (y + (m.dy + 1) * z); }
__device__ __forceinline__ bool voxIn(const DeviceMesh& m, int x, int y, int z) {
    return x >= 0 && y >= 0 && z >= 0 && x < m.dx && y < m.dy && z < m.dz;
}
__device__ __forceinline__ int directedSlot(const DeviceMesh& m, int a, int b) {
    int d = b - a, ad = d < 0 ? -d : d;
    int axis = ad == 1 ? 0 : (ad == m.dx + 1 ? 1 : 2);
    return 6 * a + 2 * axis + (d > 0 ? 1 : 0);
}
static __device__ bool edgeIsCut(const DeviceMesh& m, const CutParams& cu, int4 g) {
    for (int s = 0; s < 4; s++) {
        int x = g.y + kStencilOff[g.x][s][0], y = g.z + kStencilOff[g.x][s][1], z = g.w + kStencilOff[g.x][s][2];
        if (voxIn(m, x, y, z) && ((cu.cutMask[x + m.dx * (y + m.dy * z)] >> kStencilEdge[g.x][s]) & 1u)) return true;
    }
    return false;
}
static __device__ bool cutHitsMaterial(float t, float skin, int ia, int ib) {
    if (ia && ib) return true;
    if (!ia && !ib) return false;
    if (!(skin >= 0.f && skin <= 1.f)) return false;
    return ia ? t <= skin : t >= skin;
}
// EmitCutPoint (V/cut.cu:186-215): the cut point of owner p on the undeformed edge (`along`) plus
// the half-kerf on p's side of the cut plane, and the outward cut normal, both in p's frame `rot`.
static __device__ void emitCutPoint(const DeviceMesh& m, const CutParams& cu, const float* rot, f3 hit, f3 along, int p, int slot, f3 ncut) {
    const f3 pp = xyz(m.pos[p]);
    const float sd = dot(pp - hit, ncut);
    float side = sd > 0.f ? 1.f : (sd < 0.f ? -1.f : 0.f);
    if (side == 0.f) side = 1.f;
    const float* q = rot + 9 * (size_t)p;
    const f3 r0 = mk(q[0], q[1], q[2]), r1 = mk(q[3], q[4], q[5]), r2 = mk(q[6], q[7], q[8]);
    const f3 g = ncut * (side * (cu.toolD * 0.5f)), n = ncut * side;
    const f3 local = along + ((r0 * g.x + r1 * g.y) + r2 * g.z);
    const f3 mat = (r0 * n.x + r1 * n.y) + r2 * n.z;
    cu.cutRec[2 * (size_t)slot] = make_float4(local.x, local.y, local.z, 1.f);
    cu.cutRec[2 * (size_t)slot + 1] = make_float4(mat.x, mat.y, mat.z, 0.f);
}

// MarkAndEmit (V/cut.cu:218-254): mark the edge in its occupied stencil voxels; on its first cut
// record the fractions and, for a crossing inside the material, the two cut points (the owners'
// frames `rot`; `hit` and `ncut` place the kerf).
static __device__ void markEdge(const DeviceMesh& m, const CutParams& cu, const float* rot, int4 g, int a, int b, float t, f3 hit, f3 ncut) {
    bool first = false, saw = false, occ = false;
    for (int s = 0; s < 4; s++) {
        int x = g.y + kStencilOff[g.x][s][0], y = g.z + kStencilOff[g.x][s][1], z = g.w + kStencilOff[g.x][s][2];
        if (!voxIn(m, x, y, z)) continue;
        int v = x + m.dx * (y + m.dy * z);
        if (cu.occupied[v] == 0u) continue;
        occ = true;
        unsigned bit = 1u << kStencilEdge[g.x][s];
        unsigned old = atomicOr(cu.cutMask + v, bit);
        if (!saw) { saw = true; first = (old & bit) == 0u; }
    }
    if (!(first && occ)) return;
    cu.edgeCutT[directedSlot(m, a, b)] = t;
    cu.edgeCutT[directedSlot(m, b, a)] = 1.f - t;
    if (!cutHitsMaterial(t, cu.skinT[directedSlot(m, a, b)], cu.inside[a], cu.inside[b])) return;
    atomicAdd(cu.counters + 1, 2u);
    if (cu.cutRec && rot) {
        const f3 rest = xyz(cu.rest[b]) - xyz(cu.rest[a]);
        emitCutPoint(m, cu, rot, hit, rest * t, a, 6 * a + 2 * g.x + 1, ncut);
        emitCutPoint(m, cu, rot, hit, rest * (t - 1.f), b, 6 * b + 2 * g.x, ncut);
    }
}

static __device__ void tickEdgeAt(const DeviceMesh& m, const CutParams& cu, int4 g, bool ccd, const float* rot) {
    int axis = g.x;                    // g = (axis, x, y, z) of the base node
    int a = nodeId(m, g.y, g.z, g.w);
    int b = nodeId(m, g.y + (axis == 0), g.z + (axis == 1), g.w + (axis == 2));
    int slotA = 6 * a + 2 * axis + 1;
    if (ccd && m.nbr[slotA] >= 0) {
        f3 S = mk(cu.sx, cu.sy, cu.sz), E = mk(cu.ex, cu.ey, cu.ez);
        f3 a0 = xyz(m.prev[a]), a1 = xyz(m.pos[a]), b0 = xyz(m.prev[b]), b1 = xyz(m.pos[b]);
        float pad = cu.voxelL;
        f3 sMin = mk(fminf(S.x, E.x) - pad, fminf(S.y, E.y) - pad, fminf(S.z, E.z) - pad);
        f3 sMax = mk(fmaxf(S.x, E.x) + pad, fmaxf(S.y, E.y) + pad, fmaxf(S.z, E.z) + pad);
        f3 eMin = mk(fminf(fminf(a0.x, a1.x), fminf(b0.x, b1.x)), fminf(fminf(a0.y, a1.y), fminf(b0.y, b1.y)),
                     fminf(fminf(a0.z, a1.z), fminf(b0.z, b1.z)));
        f3 eMax = mk(fmaxf(fmaxf(a0.x, a1.x), fmaxf(b0.x, b1.x)), fmaxf(fmaxf(a0.y, a1.y), fmaxf(b0.y, b1.y)),
                     fmaxf(fmaxf(a0.z, a1.z), fmaxf(b0.z, b1.z)));
        bool cull = eMax.x < sMin.x || eMin.x > sMax.x || eMax.y < sMin.y || eMin.y > sMax.y || eMax.z < sMin.z || eMin.z > sMax.z;
        if (!cull) {
            f3 D = E - S, P0 = a0 - S, Pv = a1 - a0, Q0 = b0 - S, Qv = b1 - b0;
            float c0 = dot(cross(P0, Q0), D), c1 = dot(cross(P0, Qv) + cross(Pv, Q0), D), c2 = dot(cross(Pv, Qv), D);
            float roots[2]; int nr = 0;
            if (fabsf(c2) < 1e-14f) {
                if (fabsf(c1) > 1e-14f) { float r = -c0 / c1; if (r >= 0.f && r <= 1.f) roots[nr++] = r; }
            } else {
                float disc = c1 * c1 - 4.f * c2 * c0;
                if (disc >= 0.f) {
                    float sq = sqrtf(disc), qq = -0.5f * (c1 + (c1 >= 0.f ? sq : -sq));
                    float r0 = qq / c2, r1 = fabsf(qq) > 1e-20f ? c0 / qq : r0;
                    if (r0 > r1) { float tmp = r0; r0 = r1; r1 = tmp; }
                    if (r0 >= 0.f && r0 <= 1.f) roots[nr++] = r0;
                    if (r1 >= 0.f && r1 <= 1.f && r1 != r0) roots[nr++] = r1;
                }
            }
            for (int ri = 0; ri < nr; ri++) {
                float tc = roots[ri];
                f3 pa = a0 + Pv * tc, pb = b0 + Qv * tc, e1 = pb - pa, n2 = cross(e1, D);
                float n2l = dot(n2, n2);
                if (n2l < 1e-16f) continue;
                f3 wv = S - pa;
                float u = dot(cross(wv, D), n2) / n2l, v = dot(cross(wv, e1), n2) / n2l;
                if (u <= 0.f || u > 1.f || v < -2e-2f || v > 1.f + 2e-2f) continue;
                // hit on the current edge; kerf normal = blade x relative tissue motion, else the
                // last valid blade normal (V/cut.cu:576-587)
                const f3 hit = a1 + (b1 - a1) * u;
                const f3 relV = (Pv + Qv) * 0.5f, nHit = cross(D, relV);
                const float nLen = len(nHit);
                const f3 nEmit = nLen > 1e-8f ? mk(nHit.x / nLen, nHit.y / nLen, nHit.z / nLen) : mk(cu.ncx, cu.ncy, cu.ncz);
                markEdge(m, cu, rot, g, a, b, u, hit, nEmit);
                break;
            }
        }
    }
    if (cu.tearLen2 > 0.f && m.nbr[slotA] >= 0 && m.active[a] != 0 && m.active[b] != 0 && !edgeIsCut(m, cu, g)) {
        bool anyOcc = false;
        for (int s = 0; s < 4 && !anyOcc; s++) {
            int x = g.y + kStencilOff[axis][s][0], y = g.z + kStencilOff[axis][s][1], z = g.w + kStencilOff[axis][s][2];
            anyOcc = voxIn(m, x, y, z) && cu.occupied[x + m.dx * (y + m.dy * z)] != 0u;
        }
        if (anyOcc) {
            f3 d = xyz(m.pos[b]) - xyz(m.pos[a]);
            float l2 = dot(d, d);
            f3 r = xyz(cu.rest[b]) - xyz(cu.rest[a]);
            float tl2 = cu.tearLen2 * (dot(r, r) / (cu.voxelL * cu.voxelL));
            if (l2 > tl2) {   // tear plane normal to the edge through its midpoint (V/cut.cu:674-683)
                atomicAdd(cu.counters + 2, 1u);
                const float l = sqrtf(l2);
                markEdge(m, cu, rot, g, a, b, 0.5f, xyz(m.pos[a]) + d * 0.5f, mk(d.x / l, d.y / l, d.z / l));
            }
        }
    }
    // SeverLinks (V/cut.cu:719-746): a cut mark on this edge parts the link and its bend pairs.
    bool valid = true;
    for (int s = 0; s < 4; s++)
        valid = valid && voxIn(m, g.y + kStencilOff[axis][s][0], g.z + kStencilOff[axis][s][1], g.w + kStencilOff[axis][s][2]);
    if (!valid || !edgeIsCut(m, cu, g)) return;
    // When every live bend pair's links exist (checked when the physics is set up, and kept: a
    // sever kills the pairs of the link it removes), an edge whose link is already gone has no live
    // pair left, and the pass below would change nothing.
    if (cu.skipSevered && m.nbr[slotA] < 0) return;
    if (m.nbr[slotA] >= 0) atomicAdd(cu.counters + 0, 1u);
    m.nbr[slotA] = -1;
    m.nbr[6 * b + 2 * axis] = -1;
    if (m.nBendPairs >= 15 * (max(a, b) + 1)) {
        for (int p = 0; p < 15; p++) {
            BendRecord* x = m.bendPairs + 15 * a + p;
            if (x->alive != 0 && (x->j == b || x->k == b)) x->alive = 0;
            BendRecord* y = m.bendPairs + 15 * b + p;
            if (y->alive != 0 && (y->j == a || y->k == a)) y->alive = 0;
        }
    }
}

__device__ __forceinline__ void tickEdge(const DeviceMesh& m, const CutParams& cu, int e, bool ccd, const float* rot) {
    tickEdgeAt(m, cu, cu.gridEdges[e], ccd, rot);
}

// Brick pre-cull of the ribbon tick: the lattice's base nodes in bricks of 4 x 4 x 4, each brick's
// box over the current and substep-start positions of its nodes and of the +1 layer that its edges
// reach.  An edge whose brick box misses the blade's padded box misses it too, so only the edges of
// listed bricks run the crossing test; the rest of the tick (the sever of marked edges) has nothing
// to do on the others: rod-phase marks are severed when made, tick marks are made on listed edges,
// and the tear law (which visits every edge) keeps the full pass.
constexpr int kBrick = 4, kBrickEdges = 3 * kBrick * kBrick * kBrick;
static __device__ void brickBounds(const DeviceMesh& m, const CutParams& cu, int b, int lane) {
    const int nbx = (m.dx + kBrick - 1) / kBrick, nby = (m.dy + kBrick - 1) / kBrick;
    const int bx = b % nbx, by = (b / nbx) % nby, bz = b / (nbx * nby);
    const int x0 = bx * kBrick, y0 = by * kBrick, z0 = bz * kBrick;
    const int x1 = min(x0 + kBrick, m.dx), y1 = min(y0 + kBrick, m.dy), z1 = min(z0 + kBrick, m.dz);
    // the (kBrick + 1)^3 = 125 node slots of the brick, four per lane (constant divisors), all loads
    // issued before any use; slots past the lattice's last layer are skipped
    constexpr int kSide = kBrick + 1;
    f3 lo = mk(3.0e38f, 3.0e38f, 3.0e38f), hi = mk(-3.0e38f, -3.0e38f, -3.0e38f);
    float4 P[4], Q[4];
    bool in[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const int k = lane + 32 * t;
        const int x = x0 + k % kSide, y = y0 + (k / kSide) % kSide, z = z0 + k / (kSide * kSide);
        in[t] = k < kSide * kSide * kSide && x <= x1 && y <= y1 && z <= z1;
        if (in[t]) { const int id = nodeId(m, x, y, z); P[t] = m.pos[id]; Q[t] = m.prev[id]; }
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
        if (!in[t]) continue;
        const f3 p = xyz(P[t]), q = xyz(Q[t]);
        lo = mk(fminf(lo.x, fminf(p.x, q.x)), fminf(lo.y, fminf(p.y, q.y)), fminf(lo.z, fminf(p.z, q.z)));
        hi = mk(fmaxf(hi.x, fmaxf(p.x, q.x)), fmaxf(hi.y, fmaxf(p.y, q.y)), fmaxf(hi.z, fmaxf(p.z, q.z)));
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = mk(fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o)), fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o)),
                fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o)));
        hi = mk(fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o)), fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o)),
                fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o)));
    }
    if (lane != 0) return;
    const float pad = cu.voxelL;
    const bool miss = hi.x < fminf(cu.sx, cu.ex) - pad || lo.x > fmaxf(cu.sx, cu.ex) + pad ||
                      hi.y < fminf(cu.sy, cu.ey) - pad || lo.y > fmaxf(cu.sy, cu.ey) + pad ||
                      hi.z < fminf(cu.sz, cu.ez) - pad || lo.z > fmaxf(cu.sz, cu.ez) + pad;
    if (!miss) {
        const unsigned slot = atomicAdd(cu.brickCount, 1u);
        if (slot < (unsigned)cu.nBricks) cu.brickList[slot] = b;
    }
}
// Edge `l` (0 .. kBrickEdges-1) of a listed brick as (axis, base node), or false when the lattice has
// no such interior edge (one whose four incident voxels exist, as the host's edge list holds).
__device__ __forceinline__ bool brickEdge(const DeviceMesh& m, int b, int l, int4& g) {
    const int nbx = (m.dx + kBrick - 1) / kBrick, nby = (m.dy + kBrick - 1) / kBrick;
    const int axis = l / (kBrick * kBrick * kBrick), o = l % (kBrick * kBrick * kBrick);
    const int x = (b % nbx) * kBrick + o % kBrick, y = ((b / nbx) % nby) * kBrick + (o / kBrick) % kBrick,
              z = (b / (nbx * nby)) * kBrick + o / (kBrick * kBrick);
    const int c[3] = {x, y, z}, d[3] = {m.dx, m.dy, m.dz};
    for (int a = 0; a < 3; a++)
        if (a == axis ? c[a] >= d[a] : (c[a] < 1 || c[a] >= d[a])) return false;
    g = make_int4(axis, x, y, z);
    return true;
}

}  // namespace gbt
