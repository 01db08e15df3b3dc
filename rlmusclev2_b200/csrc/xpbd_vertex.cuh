// Per-vertex substep boundary (push-out out of the bones' grid SDF, velocity,
// prediction, pin), shared by the per-vertex kernels (xpbd_core.cu) and the
// persistent frame (xpbd_frame.cu).
#pragma once
#include "xpbd_common.cuh"
#include "xpbd_device.cuh"

namespace xpbd {

// ---------------------------------------------------------------------------
// Trilinear grid SDF sample and gradient (phi at nodes origin + h*(i,j,k)).
__device__ __forceinline__ bool sdf_sample(const XpbdSdf& S, float3 x, float& phi, float3& grad) {
    const float inv_h = 1.f / S.h;
    const float gx = (x.x - S.origin[0]) * inv_h, gy = (x.y - S.origin[1]) * inv_h, gz = (x.z - S.origin[2]) * inv_h;
    if (!(gx >= 0.f && gy >= 0.f && gz >= 0.f && gx <= float(S.nx - 1) && gy <= float(S.ny - 1) && gz <= float(S.nz - 1)))
        return false;
    int ix = min(int(gx), S.nx - 2), iy = min(int(gy), S.ny - 2), iz = min(int(gz), S.nz - 2);
    const float fx = gx - float(ix), fy = gy - float(iy), fz = gz - float(iz);
    const size_t sx = 1, sy = size_t(S.nx), sz = size_t(S.nx) * size_t(S.ny);
    const float* b = S.phi + size_t(iz) * sz + size_t(iy) * sy + size_t(ix);
    const float c000 = __ldg(b), c100 = __ldg(b + sx), c010 = __ldg(b + sy), c110 = __ldg(b + sy + sx);
    const float c001 = __ldg(b + sz), c101 = __ldg(b + sz + sx), c011 = __ldg(b + sz + sy), c111 = __ldg(b + sz + sy + sx);
    const float c00 = c000 + fx * (c100 - c000), c10 = c010 + fx * (c110 - c010);
    const float c01 = c001 + fx * (c101 - c001), c11 = c011 + fx * (c111 - c011);
    const float c0 = c00 + fy * (c10 - c00), c1 = c01 + fy * (c11 - c01);
    phi = c0 + fz * (c1 - c0);
    // analytic gradient of the trilinear interpolant
    const float dx0 = (c100 - c000) + fy * ((c110 - c010) - (c100 - c000));
    const float dx1 = (c101 - c001) + fy * ((c111 - c011) - (c101 - c001));
    const float dy0 = (c010 - c000) + fx * ((c110 - c100) - (c010 - c000));
    const float dy1 = (c011 - c001) + fx * ((c111 - c101) - (c011 - c001));
    grad = make_float3((dx0 + fz * (dx1 - dx0)) * inv_h, (dy0 + fz * (dy1 - dy0)) * inv_h, (c1 - c0) * inv_h);
    return true;
}

// Push-out of one vertex (solve_mesh_contact_pos_kernel semantics with the
// bone mesh query replaced by the grid SDF): err = phi - offset; if err < 0
// (and depth <= max_push when max_push > 0) move along the outward normal.
__device__ __forceinline__ void sdf_push(const XpbdSdf& S, float4& p) {
    if (p.w == 0.f) return;
    float phi;
    float3 gr;
    if (!sdf_sample(S, f3(p), phi, gr)) return;
    const float gl = len(gr);
    if (!(gl > 1e-12f)) return;
    const float err = phi - S.contact_offset;
    if (err < 0.f && (S.max_push <= 0.f || -err <= S.max_push)) {
        const float3 n = gr / gl;
        p.x -= n.x * err;
        p.y -= n.y * err;
        p.z -= n.z * err;
    }
}

// One vertex's share of a substep boundary, on its registers: position p,
// velocity v (w: stopped), previous position q (read by OP_VELOCITY, replaced
// by OP_PREDICT).  Shared by the per-vertex kernels and the persistent frame.
__device__ __forceinline__ void vertex_step_regs(const XpbdParams& prm, const XpbdVerts& V, uint32_t ops,
                                                 const XpbdSdf& S, int g, float4& p, float4& v, float4& q) {
    const float dt = prm.dt;
    if (ops & XPBD_OP_SDF) sdf_push(S, p);
    if (ops & XPBD_OP_VELOCITY) {
        v.x = (p.x - q.x) / dt;
        v.y = (p.y - q.y) / dt;
        v.z = (p.z - q.z) / dt;
    }
    if (ops & XPBD_OP_PREDICT) {
        q = make_float4(p.x, p.y, p.z, 0.f);
        if (v.w != 0.f) {
            v.x = v.y = v.z = 0.f;
        } else {
            float3 ext = make_float3(prm.gravity[0], prm.gravity[1], prm.gravity[2]);
            if (V.force) {
                const float m = V.mass[g];
                if (m > 1.0e-12f) ext = ext + f3(reinterpret_cast<const float4*>(V.force)[g]) / m;
            }
            if (prm.quasi_static) {
                const float dt2 = dt * dt;
                p.x += dt2 * ext.x;
                p.y += dt2 * ext.y;
                p.z += dt2 * ext.z;
                v.x = v.y = v.z = 0.f;
            } else {
                const float damp = 1.f - prm.veldamping;
                v.x = damp * v.x + dt * ext.x;
                v.y = damp * v.y + dt * ext.y;
                v.z = damp * v.z + dt * ext.z;
                p.x += dt * v.x;
                p.y += dt * v.y;
                p.z += dt * v.z;
            }
        }
    }
}

__device__ __forceinline__ void vertex_step_at(const XpbdParams& prm, const XpbdVerts& V, uint32_t ops,
                                               const XpbdSdf& S, int g) {
    float4* pos4 = reinterpret_cast<float4*>(V.pos);
    float4* prev4 = reinterpret_cast<float4*>(V.pprev);
    float4* vel4 = reinterpret_cast<float4*>(V.vel);
    float4 p = pos4[g];
    float4 v = vel4[g];
    float4 q;
    if (ops & XPBD_OP_VELOCITY) q = prev4[g];
    vertex_step_regs(prm, V, ops, S, g, p, v, q);
    if (ops & XPBD_OP_PREDICT) prev4[g] = q;
    if ((ops & XPBD_OP_PIN) && V.vflags && (V.vflags[g] & XPBD_VF_PIN)) {
        const float4 t = reinterpret_cast<const float4*>(V.pin_target)[g];
        if (t.w != 0.f) {
            p.x = t.x;
            p.y = t.y;
            p.z = t.z;
        }
    }
    pos4[g] = p;
    if (ops & (XPBD_OP_VELOCITY | XPBD_OP_PREDICT)) vel4[g] = v;
}

// The grid of vertex g's instance; false: the vertex has none.
__device__ __forceinline__ bool instance_sdf(const XpbdSdfBatch& B, int g, XpbdSdf& S) {
    S.nx = B.nx;
    S.ny = B.ny;
    S.nz = B.nz;
    S.contact_offset = B.contact_offset;
    S.max_push = B.max_push;
    S.reserved = 0;
    S.phi = nullptr;
    S.origin[0] = S.origin[1] = S.origin[2] = 0.f;
    S.h = 1.f;
    const int inst = B.vert_inst[g];
    if (inst < 0 || inst >= B.n_inst) return false;
    const float4 fr = reinterpret_cast<const float4*>(B.frame)[inst];
    S.phi = B.phi + size_t(inst) * size_t(B.nx) * size_t(B.ny) * size_t(B.nz);
    S.origin[0] = fr.x;
    S.origin[1] = fr.y;
    S.origin[2] = fr.z;
    S.h = fr.w;
    return true;
}

}  // namespace xpbd
