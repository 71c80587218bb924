// Contact model 0 on one node: the shaft capsule and the jaw slab of the substep's instrument frame.
#pragma once
#include "tissue_device.cuh"

namespace gbt {

// ---------------------------------------------------------------------------------------------
// contact model 0: shaft capsule + jaw slab CCD gate, k_SolveCCDContact (xpbd_solver.cu:1049-1123)
// ---------------------------------------------------------------------------------------------
// The substep's instrument frame (contactFrame) lives in tissue_device.cuh: batches evaluate it on
// the host, single meshes on the device, with the same operations.
// The contact of one mobile node (wc > 0) at p moving with the substep's predicted velocity v.
// Warp-level early-out of the capsule test: a node outside the box of the shaft segment grown by the
// radius (and a margin far above the rounding of the exact distance) cannot be inside the capsule,
// where the exact test would change nothing; a warp with no node inside that box skips the test
// (one ballot), the others run it exactly as before, so the result is the same bit for bit.
__device__ __forceinline__ bool nearCapsule(f3 p, const ContactFrame& f) {
    const float r = f.shaftR * 1.0001f + 1e-5f;
    return p.x >= fminf(f.sa.x, f.sb.x) - r && p.x <= fmaxf(f.sa.x, f.sb.x) + r && p.y >= fminf(f.sa.y, f.sb.y) - r &&
           p.y <= fmaxf(f.sa.y, f.sb.y) + r && p.z >= fminf(f.sa.z, f.sb.z) - r && p.z <= fmaxf(f.sa.z, f.sb.z) + r;
}
__device__ __forceinline__ f3 contactPoint(f3 p, float wc, f3 v, const ContactFrame& f, const ContactParams& cp) {
    const bool near = nearCapsule(p, f);
    if (__ballot_sync(__activemask(), near) != 0u && near) {
        f3 ab = f.sb - f.sa;
        float ab2 = dot(ab, ab);
        float tt = ab2 > 1e-12f ? dot(p - f.sa, ab) / ab2 : 0.f;
        tt = fmaxf(0.f, fminf(1.f, tt));
        f3 dv = p - (f.sa + ab * tt);
        float dist = len(dv), C = dist - f.shaftR;
        if (C < 0.f) {
            f3 n = dist > 1e-9f ? dv * (1.f / dist) : mk(0.f, 1.f, 0.f);
            if (-dot(v, n) > cp.ccdVelThresh) {
                float dl = (-C - f.alpha * 0.f) / (wc + f.alpha);
                float ap = cp.ccdOmega * dl;
                f3 corr = n * (wc * ap);
                float cl = len(corr);
                if (cl > cp.ccdMaxDisp) { float s = cp.ccdMaxDisp / cl; ap *= s; corr = corr * s; }
                p = p + corr;
            }
        }
    }
    {
        f3 rel = p - f.hinge;
        float u = dot(rel, f.axis), vv = dot(rel, f.w), n = dot(rel, f.normal);
        if (u >= 0.f && u <= f.jawLen && fabsf(vv) <= f.halfWidth) {
            float an = fabsf(n);
            if (an > f.gapHalf) {
                float C = f.gapHalf - an, sg = n >= 0.f ? 1.f : -1.f;
                f3 nOut = f.normal * sg;
                if (-dot(v, nOut) > cp.ccdVelThresh) {
                    float dl = (-C - f.alpha * 0.f) / (wc + f.alpha);
                    float ap = cp.ccdOmega * dl, cm = wc * ap;
                    if (fabsf(cm) > cp.ccdMaxDisp) { float s = cp.ccdMaxDisp / fabsf(cm); ap *= s; cm *= s; }
                    p = p - f.normal * (sg * cm);
                }
            }
        }
    }
    return p;
}

}  // namespace gbt
