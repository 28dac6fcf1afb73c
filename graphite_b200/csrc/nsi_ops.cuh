// Per-cell device math of the incompressible model, shared by the kernels of
// nsi.cu and the persistent loop of nsi_loop.cu.
#pragma once

#include "euler_ops.cuh"

namespace gb {

// The ghost state of one boundary face from its interior state (pi, ui) and
// outward normal n: type 0 slip, 1 inlet / outlet, 2 no-slip wall.
__device__ __forceinline__ void nsi_ghost_state(int type, float3 n, float pi, float3 ui, float3 vinf, float pinf,
                                                float& pg, float3& ug) {
    // explicitly rounded (xdot): the ghost kernel and the gradient kernel both
    // form these states and must agree bitwise
    if (type == 0) {
        const float s = __fmul_rn(2.f, xdot(n, ui));
        ug = make_float3(__fmaf_rn(-n.x, s, ui.x), __fmaf_rn(-n.y, s, ui.y), __fmaf_rn(-n.z, s, ui.z));
        pg = pi;
    } else if (type == 2) {
        ug = make_float3(-ui.x, -ui.y, -ui.z);
        pg = pi;
    } else if (xdot(vinf, n) < 0.f) {
        ug = vinf;
        pg = pi;
    } else {
        ug = ui;
        pg = pinf;
    }
}

struct NsiParams {
    float cfl, nu, beta2;
    int corrected;            // 1: compact correction of the face gradient
};

// Flux balance of one cell, summed over its faces.
struct NsiSum {
    float rp, sr;          // zero-initialised
    float3 ru;
    // a face with outward normal n and area / volume ds between the cell (pi,
    // ui, gradients + limiters gpi, gui, face offset d0) and its neighbour (d1
    // the face's offset from it); dw = (centroid offset, 1 / |.|^2).  Every
    // multiply-add is written out, as the compiler fused them in k_nsi_flux: it
    // fuses them differently from one loop to the next, and the kernels that
    // share this function must agree bitwise.
    __device__ __forceinline__ void face(const NsiParams& P, float pi, float3 ui, float4 gpi, const float4 gui[3],
                                         float pj, float3 uj, float4 gpj, const float4 guj[3], float3 n, float ds,
                                         float3 d0, float3 d1, float4 dw) {
        const float pL = __fmaf_rn(ydot(f3(gpi), d0), gpi.w, pi);
        const float pR = __fmaf_rn(xdot(f3(gpj), d1), gpj.w, pj);
        const float3 uL = make_float3(__fmaf_rn(ydot(f3(gui[0]), d0), gui[0].w, ui.x),
                                      __fmaf_rn(ydot(f3(gui[1]), d0), gui[1].w, ui.y),
                                      __fmaf_rn(ydot(f3(gui[2]), d0), gui[2].w, ui.z));
        const float3 uR = make_float3(__fmaf_rn(ydot(f3(guj[0]), d1), guj[0].w, uj.x),
                                      __fmaf_rn(ydot(f3(guj[1]), d1), guj[1].w, uj.y),
                                      __fmaf_rn(ydot(f3(guj[2]), d1), guj[2].w, uj.z));
        const float unL = ydot(uL, n), unR = ydot(uR, n);
        const float lam = fmaxf(fabsf(unL) + sqrtf(__fmaf_rn(unL, unL, P.beta2)),
                                fabsf(unR) + sqrtf(__fmaf_rn(unR, unR, P.beta2)));
        const float h = __fmul_rn(0.5f, ds), lh = __fmul_rn(lam, h);
        const float bs = __fmul_rn(P.beta2, __fadd_rn(unL, unR)), dp = __fadd_rn(pR, -pL);
        rp = __fadd_rn(rp, __fmaf_rn(bs, h, -__fmul_rn(lh, dp)));
        // viscous flux: face gradient of u dotted with n
        const float3 d = f3(dw);
        const float nds = __fmul_rn(P.nu, ds), dn = ydot(d, n);
        auto mom = [&](float r, float l, float rr, float nk) {
            float m = __fmaf_rn(nk, pL, __fmul_rn(l, unL));
            m = __fmaf_rn(rr, unR, m);
            m = __fmaf_rn(nk, pR, m);
            return __fmaf_rn(-__fadd_rn(rr, -l), lh, __fmaf_rn(m, h, r));
        };
        auto vis = [&](float4 gi, float4 gj, float u0, float u1) {
            const float3 ga = (f3(gi) + f3(gj)) * 0.5f;
            float gn = ydot(ga, n);
            if (P.corrected)
                gn = __fmaf_rn(__fmul_rn(__fadd_rn(__fadd_rn(u1, -u0), -ydot(ga, d)), dw.w), dn, gn);
            return gn;
        };
        ru = make_float3(__fmaf_rn(-vis(gui[0], guj[0], ui.x, uj.x), nds, mom(ru.x, uL.x, uR.x, n.x)),
                         __fmaf_rn(-vis(gui[1], guj[1], ui.y, uj.y), nds, mom(ru.y, uL.y, uR.y, n.y)),
                         __fmaf_rn(-vis(gui[2], guj[2], ui.z, uj.z), nds, mom(ru.z, uL.z, uR.z, n.z)));
        sr = __fmaf_rn(__fmaf_rn(__fmul_rn(2.f, P.nu), sqrtf(dw.w), lam), ds, sr);
    }
};

}  // namespace gb
