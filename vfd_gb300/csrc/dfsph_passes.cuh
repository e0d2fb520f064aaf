// Device code shared by the neighbour-row kernels (dfsph_physics.cu) and the staged-tile
// kernels (dfsph_halo.cu): per-pair terms and what a pass does with a particle's sums.
#pragma once

#include "dfsph_common.cuh"

namespace vfd {

enum LoopId { kLoopDiv = 0, kLoopCG = 1, kLoopPres = 2 };

// kappa (or kappa_v) of particle p, mirrored into X[p].w for the neighbours' gathers.
// (Cell-relative positions keep their anchor in X.w; the neighbours then read kappa itself.)
__device__ __forceinline__ void set_kappa(const Dev& d, uint32_t p, float k) {
    if (!d.cellRel) reinterpret_cast<float*>(d.X)[4 * (size_t)p + 3] = k;
}

// A lane's partial sums of a neighbour loop with G lanes a particle. Four lanes keep two, of
// the even and of the odd rounds, which are those that eight lanes keep; total() adds them as
// the eight lanes' shuffle tree does, so either lane count gives the same bits.
template <uint32_t G, class T>
struct LaneSums {
    T s[2] = {};
    __device__ __forceinline__ T& at(uint32_t round) { return s[G == 4u ? round & 1u : 0u]; }
    __device__ __forceinline__ T total() {
        if (G == 4u) s[0] += s[1];
        return s[0];
    }
};

// One pair's terms, shared by the row and the tile kernels so that their bits agree: the sums
// of the density and factor (K2 - K4), ...
struct DensitySums {
    float w = 0.0f, g2 = 0.0f, div = 0.0f;
    float3 gi = {0.0f, 0.0f, 0.0f};
    __device__ __forceinline__ void add(float V, float wj, float gs, float3 r, bool withDiv, float3 dv) {
        w += wj;
        const float3 gj = mul3(-V * gs, r);
        g2 += dot3(gj, gj);
        gi -= gj;
        if (withDiv) div += dot3(dv, gs * r);
    }
    __device__ __forceinline__ void operator+=(const DensitySums& b) { w += b.w, g2 += b.g2, div += b.div, gi += b.gi; }
};
// ... the pressure acceleration (K5, K7, K18, K20) and the viscosity product (K14).
__device__ __forceinline__ void add_pressure(float3& a, float sum, float V, float gs, float3 r, bool ok) {
    if (ok && fabsf(sum) > kEps) a = fma3(sum * (-V * gs), r, a);
}
__device__ __forceinline__ void add_viscous(float3& acc, float cw, float3 dv, float eps2, float gs, float3 r, bool ok) {
    const float c = __fdividef(cw * dot3(dv, r), dot3(r, r) + eps2) * gs;
    if (ok) acc = fma3(c, r, acc);
}

// One particle's term of a CG dot product: the FP32 dot of its two vectors (no
// contraction, x + y then z, as the FP32 oracle forms it); the sum over particles is
// FP64-accurate (scene_accumulate). FP64 arithmetic runs at a small fraction of the
// FP32 rate on this GPU, so the per-particle terms stay FP32, as every per-particle sum
// of the reference does.
__device__ __forceinline__ float dot_term(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}

// W and gradW of one pair from one table position (GetW / GetGradientW keep their own
// range tests: |r|^2 <= R^2 for W, |r| <= R for gradW).
__device__ __forceinline__ void kernel_wg_r2(const Dev& d, float r2, float& w, float& gs) {
    const float rl = fast_sqrt(r2);
    if (d.analytic) {
        w = r2 <= d.radius2 ? spline_w(d, rl) : 0.0f;
        gs = rl <= d.radius ? spline_gs(d, rl) : 0.0f;
        return;
    }
    const uint32_t pos = table_pos(d, rl);
    w = r2 <= d.radius2 ? __ldg(d.WM + pos) : 0.0f;
    gs = rl <= d.radius ? __ldg(d.GM + pos) : 0.0f;
}
__device__ __forceinline__ void kernel_wg(const Dev& d, float3 r, float& w, float& gs) {
    kernel_wg_r2(d, dot3(r, r), w, gs);
}

struct Mat3 {
    float3 r0, r1, r2;
    __device__ __forceinline__ void operator+=(const Mat3& b) { r0 += b.r0, r1 += b.r1, r2 += b.r2; }
};
__device__ __forceinline__ float3 mul(const Mat3& m, float3 v) {
    return make_float3(dot3(m.r0, v), dot3(m.r1, v), dot3(m.r2, v));
}
__device__ __forceinline__ void add_outer(Mat3& m, float c, float3 a, float3 b) {  // m += c a b^T
    m.r0 = fma3(c * a.x, b, m.r0);
    m.r1 = fma3(c * a.y, b, m.r1);
    m.r2 = fma3(c * a.z, b, m.r2);
}
__device__ __forceinline__ Mat3 load_mat(const float4* M, size_t stride, uint32_t p) {
    Mat3 m;
    m.r0 = f3(M[p]);
    m.r1 = f3(M[stride + p]);
    m.r2 = f3(M[2 * stride + p]);
    return m;
}
__device__ __forceinline__ void store_mat(float4* M, size_t stride, uint32_t p, const Mat3& m) {
    M[p] = f4(m.r0, 0.f);
    M[stride + p] = f4(m.r1, 0.f);
    M[2 * stride + p] = f4(m.r2, 0.f);
}
__device__ __forceinline__ Mat3 inverse3(const Mat3& a) {  // cofactors / determinant
    const float c00 = a.r1.y * a.r2.z - a.r1.z * a.r2.y;
    const float c01 = a.r1.z * a.r2.x - a.r1.x * a.r2.z;
    const float c02 = a.r1.x * a.r2.y - a.r1.y * a.r2.x;
    const float det = a.r0.x * c00 + a.r0.y * c01 + a.r0.z * c02;
    const float id = 1.0f / det;
    Mat3 r;
    r.r0 = make_float3(c00 * id, (a.r0.z * a.r2.y - a.r0.y * a.r2.z) * id, (a.r0.y * a.r1.z - a.r0.z * a.r1.y) * id);
    r.r1 = make_float3(c01 * id, (a.r0.x * a.r2.z - a.r0.z * a.r2.x) * id, (a.r0.z * a.r1.x - a.r0.x * a.r1.z) * id);
    r.r2 = make_float3(c02 * id, (a.r0.y * a.r2.x - a.r0.x * a.r2.y) * id, (a.r0.x * a.r1.y - a.r0.y * a.r1.x) * id);
    return r;
}

// K2 + K3 (and K4 with `div`) after the pair sums: density, factor, boundary gradient.
__device__ __forceinline__ void density_finish(const Dev& d, uint32_t p, const SceneDev& S, float3 xi, float3 vi, bool div,
                                               DensitySums s, uint32_t flags) {
    const float V = S.volume;
    float rhoB = 0.0f;
    float3 gb = make_float3(0.f, 0.f, 0.f);
    if (flags & kHasBoundary) {
        for (uint32_t b = 0; b < S.bodyCount; b++) {
            const float4 xb = d.XB[(size_t)b * d.stride + p];
            if (xb.w > 0.0f) {
                const float3 r = xi - f3(xb);
                float w, gs;
                kernel_wg_r2(d, dot3_yx(r, r), w, gs);
                rhoB += xb.w * w;
                gb += (xb.w * gs) * r;
            }
        }
    }
    const float3 gi = s.gi + gb;
    d.RHO[p] = (__fmaf_rn(V, s.w, __fmul_rn(V, d.wZero)) + rhoB) * S.rho0;
    const float g2 = s.g2 + dot3_yx(gi, gi);
    const float alpha = g2 > kEps ? 1.0f / g2 : 0.0f;
    d.GB[p] = f4(gb, 0.0f);
    if (!div) {
        d.ALPHA[p] = alpha;
        return;
    }
    // K4 (:498-528)
    float rhoAdv = s.div * V;
    if (flags & kHasBoundary) rhoAdv += dot3_yx(vi, gb);
    rhoAdv = (flags & kCountMask) < 20u ? 0.0f : fmaxf(rhoAdv, 0.0f);
    d.RHOADV[p] = rhoAdv;
    const float alphaDt = alpha * S.dtInv;
    d.ALPHA[p] = alphaDt;
    d.KAPPAV[p] = rhoAdv * alphaDt;
    set_kappa(d, p, rhoAdv * alphaDt);
}

// K7 after the pair sum: the divergence solve's velocity.
__device__ __forceinline__ void div_finish_item(const Dev& d, uint32_t p, const SceneDev& S, float3 a) {
    d.AP[p] = f4(a, 0.0f);
    const float4 v = d.V[p];
    d.V[p] = f4(f3(v) + S.dt * a, v.w);
    d.ALPHA[p] *= S.dt;
}

// K12 + K13 after the pair sums: the preconditioner's inverse, the boundary viscosity matrix
// and the CG's right-hand side and first guess.
__device__ __forceinline__ void precond_finish(const Dev& d, uint32_t p, const SceneDev& S, float3 xi, Mat3 m,
                                               uint32_t flags) {
    const float eps2 = 0.01f * S.h2;
    Mat3 bv = {make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
    bool hasBV = false;
    if (S.dynBVisc != 0.0f && (flags & kHasBoundary)) {
        for (uint32_t b = 0; b < S.bodyCount; b++) {
            const float4 xb4 = d.XB[(size_t)b * d.stride + p];
            if (!(xb4.w > 0.0f)) continue;
            const float3 xb = f3(xb4);
            float3 normal = -(xi - xb);
            const float nl = sqrtf(dot3_yx(normal, normal));
            if (!(nl > 0.0001f)) continue;
            normal = make_float3(normal.x / nl, normal.y / nl, normal.z / nl);
            float3 t1, t2;
            orthogonal_vectors(normal, t1, t2);
            const float td = S.tangDist;
            const float3 pos[4] = {xb - t1 * td, xb + t1 * td, xb - t2 * td, xb + t2 * td};
            const float vol = 0.25f * xb4.w;
            const float3 d1 = xi - pos[0];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float3 dk = xi - pos[k];
                const float3 gk = kernel_grad(d, dk);
                const float c = 10.0f * S.dynBVisc * vol / (dot3(dk, dk) + eps2);
                add_outer(m, c, d1, gk);  // positionDirection1 in all four terms (:674-677)
                add_outer(bv, c, gk, dk);
            }
            hasBV = true;
        }
    }
    const float rho = d.RHO[p];
    const float f = S.dt / rho;
    Mat3 a;
    a.r0 = make_float3(1.0f - f * m.r0.x, -f * m.r0.y, -f * m.r0.z);
    a.r1 = make_float3(-f * m.r1.x, 1.0f - f * m.r1.y, -f * m.r1.z);
    a.r2 = make_float3(-f * m.r2.x, -f * m.r2.y, 1.0f - f * m.r2.z);
    store_mat(d.MINV, d.stride, p, inverse3(a));
    if (hasBV) {
        store_mat(d.BVM, d.stride, p, bv);
        d.NCNT[p] = flags | kHasBoundaryVisc;
    } else if (flags & kHasBoundaryVisc) {
        d.NCNT[p] = flags & ~kHasBoundaryVisc;
    }
    const float4 v = d.V[p];
    d.CB[p] = v;
    d.CG[p] = f4(f3(v) + f3(d.DV[p]), S.mass / rho);
}

// K6 / K19 after the pair sum `f` of the neighbours (ComputeDensityPressureForce, :280-315): the
// clamped residual and the kappa update. Returns the residual.
template <bool DIV>
__device__ __forceinline__ float jacobi_finish(const Dev& d, uint32_t p, const SceneDev& S, float3 ai, float f,
                                               uint32_t flags) {
    f *= S.volume;
    if (flags & kHasBoundary) f += dot3(ai, f3(d.GB[p]));
    float r;
    if (DIV) {
        r = (flags & kCountMask) < 20u ? 0.0f : fminf(-d.RHOADV[p] - __fmul_rn(f, S.dt), 0.0f);
        const float k = __fmaf_rn(-r, d.ALPHA[p], d.KAPPAV[p]);
        d.KAPPAV[p] = k;
        set_kappa(d, p, k);
    } else {
        r = fminf(__fmaf_rn(-f, S.dt2, 1.0f - d.RHOADV[p]), 0.0f);
        const float k = __fmaf_rn(-r, d.ALPHA[p], d.KAPPA[p]);
        d.KAPPA[p] = k;
        set_kappa(d, p, k);
    }
    d.RES[p] = r;
    return r;
}

// K14 after the pair sum: (A x)_p, of the first guess or (LOOP) of a direction of the loop.
template <bool LOOP>
__device__ __forceinline__ float3 visc_product(const Dev& d, uint32_t p, const SceneDev& S, float3 vi, float3 acc,
                                               uint32_t flags) {
    if (flags & kHasBoundaryVisc) acc += mul(load_mat(d.BVM, d.stride, p), vi);
    const float c = S.dt / d.RHO[p];
    return LOOP ? vi - mul3(c, acc) : fma3(-c, acc, vi);
}

// K17 after the pair sum: advected density, scaled factor, first kappa.
__device__ __forceinline__ void pres_init_finish(const Dev& d, uint32_t p, const SceneDev& S, float delta) {
    const float rhoAdv = d.RHO[p] / S.rho0 + S.dt * delta;
    d.RHOADV[p] = rhoAdv;
    const float alpha = d.ALPHA[p] * S.dt2Inv;
    d.ALPHA[p] = alpha;
    const float k = -fminf(1.0f - rhoAdv, 0.0f) * alpha;
    d.KAPPA[p] = k;
    set_kappa(d, p, k);
}

// K20 + K21 after the pair sum: velocity and position.
__device__ __forceinline__ void pres_finish_item(const Dev& d, uint32_t p, const SceneDev& S, float3 a) {
    d.AP[p] = f4(a, 0.0f);
    const float3 v = f3(d.V[p]) + S.dt * a;
    d.V[p] = f4(v, 0.0f);
    const float4 x4 = d.X[p];
    float3 x = f3(x4) + S.dt * v;
    if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z))) atomicOr(d.status, 0x10u);
    if (d.cellRel) {  // back into [0, h) of a (possibly new) anchor cell
        const float L = d.radius;
        int3 A = anchor_of(x4.w);
        const float fx = floorf(x.x / L), fy = floorf(x.y / L), fz = floorf(x.z / L);
        if (isfinite(x.x) && isfinite(x.y) && isfinite(x.z)) {
            A = make_int3(A.x + (int)fx, A.y + (int)fy, A.z + (int)fz);
            x = make_float3(x.x - fx * L, x.y - fy * L, x.z - fz * L);
            if (abs(A.x) > 511 || abs(A.y) > 511 || abs(A.z) > 511) atomicOr(d.status, 0x40u);
        }
        d.XN[p] = f4(x, anchor_pack(A));
    } else {
        d.XN[p] = f4(x, 0.0f);
    }
}

// K9 for one particle (:881-958): the Monte-Carlo samples are split over the group's lanes;
// at(j) is the vector to neighbour j.
template <uint32_t G, class F>
__device__ __forceinline__ void st_classify_item(const Dev& d, const Group<G>& grp, uint32_t p, const SceneDev& S,
                                                 uint32_t cnt, F&& at) {
    if (cnt == 0) {
        if (grp.lane == 0) d.STN[p] = make_float4(0.f, 0.f, 0.f, 1.0f / S.h);
        return;
    }
    LaneSums<G, float3> com3;
    for (uint32_t j = grp.lane; j < cnt; j += G) com3.at(j / G) += at(j);
    float3 com = grp.sum(com3.total());
    com = make_float3(com.x / S.h, com.y / S.h, com.z / S.h);
    const float input = sqrtf(dot3(com, com)) / (float)cnt;
    LaneSums<G, float3> nsum3;
    float3 nsum = make_float3(0.f, 0.f, 0.f);
    float curv = 0.0f;
    if ((float)cnt <= S.slope * input + S.constant + 0.0f) {
        const uint32_t samples = S.stSamples;
        const uint32_t s0 = d.PID[p] * samples / 3u * 3u;
        const float ratio = S.nbrRadius / S.r;
        const float lim = ratio * ratio * S.h2;
        uint32_t count = 0;
        for (uint32_t k = grp.lane; k < samples; k += G) {
            const uint32_t i3 = s0 + 3u * k;
            const float3 pt = S.h * make_float3(__ldg(d.halton + i3 % kHaltonCount),
                                                __ldg(d.halton + (i3 + 1u) % kHaltonCount),
                                                __ldg(d.halton + (i3 + 2u) % kHaltonCount));
            bool covered = false;
            for (uint32_t j = 0; j < cnt; j++) {
                const float3 v = pt - at(j);
                if (dot3(v, v) <= lim) { covered = true; break; }
            }
            if (!covered) { nsum3.at(k / G) += pt; count++; }
        }
        nsum = grp.sum(nsum3.total());
        count = grp.sum(count);
        if (count > 0) {
            if (dot3(nsum, nsum) > 0.0f) nsum = normalize3(nsum);
            curv = 1.0f / S.h * -2.0f * sqrtf(1.0f - S.nbrRadius * S.nbrRadius / (S.r * S.r)) *
                   cosf(acosf(1.0f - 2.0f * ((float)count / (float)samples)) + S.mcFactor);
        } else {
            nsum = make_float3(0.f, 0.f, 0.f);
        }
    }
    if (grp.lane == 0) d.STN[p] = f4(nsum, curv);
}

__device__ __forceinline__ bool nonzero3(float4 a) { return a.x != 0.0f || a.y != 0.0f || a.z != 0.0f; }

// K10 after the pair sums: smoothed normal and curvature.
__device__ __forceinline__ void st_smooth_finish(const Dev& d, uint32_t p, const SceneDev& S, float4 ni, float3 nc,
                                                 float cc, float cf) {
    if (dot3(nc, nc) > 0.0f) nc = normalize3(nc);
    const float sf = S.smoothing;
    float3 ns = (1.0f - sf) * f3(ni) + sf * nc;
    if (dot3(ns, ns) > 0.0f) ns = normalize3(ns);
    d.STNS[p] = f4(ns, ((1.0f - sf) * ni.w + sf * cc) / (1.0f - sf + sf * cf));
}

// K5 DivergenceSolveIterationKernel's force part / K18 (:388-432, :342-386): pressure
// acceleration a_p = -V sum_j (k_i + k_j) gradW_ij - k_i GB_i (kappa in X.w, or staged
// with cell-relative positions).
template <bool DIV, bool REL>
struct PressureAccelOp {
    static constexpr bool kField = REL;
    static constexpr bool kReduce = false;
    static constexpr int kSlot = 0;
    struct Own {
        float4 xi;
        float ki, V;
    };
    using Acc = float3;
    __device__ static bool active(const SceneDev& S) { return (DIV ? S.div.active : S.pres.active) != 0u; }
    __device__ static float4 field(const Dev& d, uint32_t q) {
        return make_float4((DIV ? d.KAPPAV : d.KAPPA)[q], 0.f, 0.f, 0.f);
    }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, Own& o) {
        o.xi = d.X[p];
        o.ki = (DIV ? d.KAPPAV : d.KAPPA)[p];
        o.V = S.volume;
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 fq, Acc& a) {
        const float sum = o.ki + (REL ? fq.x : xq.w);
        const float3 r = pair_r<REL>(d, o.xi, xq);
        const float gs = grad_factor(d, r);
        if (fabsf(sum) > kEps) a += (sum * (-o.V * gs)) * r;
    }
    __device__ static float finish(const Dev& d, uint32_t p, const SceneDev&, const Own& o, Acc a, uint32_t ncnt) {
        if (fabsf(o.ki) > kEps && (ncnt & kHasBoundary)) a += o.ki * (-f3(d.GB[p]));
        d.AP[p] = f4(a, 0.0f);
        return 0.0f;
    }
};

// K6 DivergenceSolveIterationKernel (:531-553) / K19 PressureSolveIterationKernel
// (:317-340), each with ComputeDensityPressureForce (:280-315): the density change of
// the pressure accelerations, the clamped residual, the kappa update, and the residual
// into the FP64-accurate sum.
template <bool DIV, bool REL>
struct JacobiOp {
    static constexpr bool kField = true;
    static constexpr bool kReduce = true;
    static constexpr int kSlot = 0;
    struct Own {
        float4 xi;
        float3 ai;
    };
    using Acc = float;
    __device__ static bool active(const SceneDev& S) { return (DIV ? S.div.active : S.pres.active) != 0u; }
    __device__ static float4 field(const Dev& d, uint32_t q) { return d.AP[q]; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev&, Own& o) {
        o.xi = d.X[p];
        o.ai = f3(d.AP[p]);
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 aq, Acc& f) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        const float gs = grad_factor(d, r);
        f += dot3(o.ai - f3(aq), gs * r);
    }
    __device__ static float finish(const Dev& d, uint32_t p, const SceneDev& S, const Own& o, Acc f, uint32_t ncnt) {
        return jacobi_finish<DIV>(d, p, S, o.ai, f, ncnt);
    }
};

// ComputeMatrixVecProdFunctionKernel (:758-842) on the CG direction p (p.w = m / rho) and
// the p . Ap term of the step length (:695-720).
template <bool REL>
struct SpmvOp {
    static constexpr bool kField = true;
    static constexpr bool kReduce = true;
    static constexpr int kSlot = 0;
    struct Own {
        float4 xi;
        float3 vi;
        float cmu, eps2;
    };
    using Acc = float3;
    __device__ static bool active(const SceneDev& S) { return S.cgActive != 0u; }
    __device__ static float4 field(const Dev& d, uint32_t q) { return d.CP[q]; }
    __device__ static void load(const Dev& d, uint32_t p, const SceneDev& S, Own& o) {
        o.xi = d.X[p];
        o.vi = f3(d.CP[p]);
        o.cmu = 10.0f * S.dynVisc;
        o.eps2 = 0.01f * S.h2;
    }
    __device__ static void pair(const Dev& d, const Own& o, float4 xq, float4 vq, Acc& acc) {
        const float3 r = pair_r<REL>(d, o.xi, xq);
        const float r2 = dot3(r, r);
        const float gs = grad_factor_r2(d, r2);
        acc += (__fdividef(o.cmu * vq.w * dot3(o.vi - f3(vq), r), r2 + o.eps2) * gs) * r;
    }
    __device__ static float finish(const Dev& d, uint32_t p, const SceneDev& S, const Own& o, Acc acc, uint32_t ncnt) {
        const float3 ap = visc_product<true>(d, p, S, o.vi, acc, ncnt);
        d.CAP[p] = f4(ap, 0.0f);
        return dot_term(o.vi, ap);
    }
};

// ---------------------------------------------------------------- control of the solver loops
__device__ __forceinline__ void set_condition(const Dev& d, int loop, uint32_t value) {
    if (d.condHandle[loop]) cudaGraphSetConditional((cudaGraphConditionalHandle)d.condHandle[loop], value);
    d.status[4 + loop] = value;
}

// Loop start: the reference's while condition evaluated with error 0, iteration 0
// (DFSPHImplementation.cu:461, :532). Returns whether the scene runs an iteration.
template <bool DIV>
__device__ __forceinline__ bool jacobi_begin(const Dev& d, SceneDev& S) {
    LoopState& L = DIV ? S.div : S.pres;
    L.it = 0;
    L.err = 0.0f;
    const uint32_t mn = DIV ? S.minIterD : S.minIterP, mx = DIV ? S.maxIterD : S.maxIterP;
    const bool enabled = (DIV ? S.enableDiv != 0 : true) && S.count > 0 && !is_aborted(d);
    const float eta = DIV ? S.dtInv * S.maxErrD * 0.0001f * S.rho0 : S.maxErrP * 0.0001f * S.rho0;
    L.active = (enabled && ((0.0f > eta) || 0u < mn) && 0u < mx) ? 1u : 0u;
    return L.active != 0u;
}
// A single scene's loop is started by the row pass before it, which reads nothing of LoopState: a
// launch less for each of the two loops. Not by the tile passes: the same lines take the density
// pass from 203 to 231 us at 1M particles. (A loop's later decisions stay launches: taken by the
// last block of a pass, with a fence and an arrival per block, a step of 64,000 particles went
// from 1,419 to 1,509 us and one of 33,401 from 1,170 to 1,221.)
inline bool start_apart(const Dev& d) { return d.nscenes > 1 || halo_on(d); }
template <bool DIV>
__device__ __forceinline__ void jacobi_start(const Dev& d) {
    if (d.nscenes == 1 && blockIdx.x == 0 && threadIdx.x == 0)
        set_condition(d, DIV ? kLoopDiv : kLoopPres, jacobi_begin<DIV>(d, d.scenes[0]) ? 1u : 0u);
}

}  // namespace vfd
