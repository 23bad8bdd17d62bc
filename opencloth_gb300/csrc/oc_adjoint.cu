// Adjoint of the implicit step (no counterpart in the reference): reverse-mode
// gradients of a trajectory with respect to per-spring Ks and Kd, the initial state and
// a per-vertex constant external force.
//
// Per step (REFERENCE Jacobian mode; vertex i takes spring i's Jacobians, IMP:737-798):
//   X' = X + dt V' (y clamped at 0), V' = V + dt dV, A dV = b,
//   A_i = m_i I - h Jv_i - h^2 J_i, b_i = h F_i + h^2 J_i V_i,
//   J = Ks n n^T - (Ks C + Kd Cdot) D, D = C diag(1 - dP*dP), Jv = -Kd n n^T,
//   f_s = (-Ks C + Kd (dV.dP)/L) n, F_i = m g + damping V_i + ext_i + sum_s +-f_s.
// The solve is differentiated as an exact solve: one extra CG on the same symmetric A
// gives lambda = A^-1 g_dV, then g_b = lambda and g_A = -lambda dV^T.  All sums are
// gathers in a fixed order (spring-ordered incidences, and per vertex the list of the
// vertices whose own spring touches it), so gradients are deterministic.  This unit is
// compiled with multiply-add contraction and approximate division and square root: the
// gradients are checked against finite differences and an FP64 adjoint, not against the
// reference's rounding sequence.
#include <cuda_runtime.h>

#include <algorithm>

#include "oc_device.cuh"
#include "oc_internal.h"

namespace oc {
namespace {

constexpr int kAdjThreads = 256;
constexpr int kAdjChunk = 128;  // vertices, and threads, of a CTA of k_adj_vertex and k_adj_springs

__device__ __forceinline__ float dot3f(float ax, float ay, float az, float bx, float by, float bz) {
    return ax * bx + ay * by + az * bz;
}

// A spring's geometry: dP = x_p1 - x_p2, its length L, 1/L and the elongation C = L - rest.
struct Geo {
    float dP[3];
    float L, iL, C;
};

// From positions.
__device__ __forceinline__ Geo geo_plain(const float4 p1, const float4 p2, float rest) {
    Geo g;
    g.dP[0] = p1.x - p2.x;
    g.dP[1] = p1.y - p2.y;
    g.dP[2] = p1.z - p2.z;
    g.L = sqrtf(dot3f(g.dP[0], g.dP[1], g.dP[2], g.dP[0], g.dP[1], g.dP[2]));
    g.iL = 1.0f / g.L;
    g.C = g.L - rest;
    return g;
}

// Displacement mode: base positions b and displacements u of the two ends, and the
// spring's constants k = {c0, L0} (c0 = |d0| - rest, L0 = |d0|, d0 = b1 - b2, rounded
// from FP64).  dP = d0 + (u1 - u2); the elongation is c0 + (|dP|^2 - |d0|^2) / (|dP| + |d0|)
// with |dP|^2 - |d0|^2 = 2 d0.du + du.du, so it keeps its relative precision when the
// elongation is small against the length (an FP32 L - rest would not).
__device__ __forceinline__ Geo geo_disp(const float4 b1, const float4 b2, const float4 u1, const float4 u2,
                                        const float2 k) {
    const float d0[3] = {b1.x - b2.x, b1.y - b2.y, b1.z - b2.z};
    const float du[3] = {u1.x - u2.x, u1.y - u2.y, u1.z - u2.z};
    Geo g;
#pragma unroll
    for (int c = 0; c < 3; ++c) g.dP[c] = d0[c] + du[c];
    g.L = sqrtf(dot3f(g.dP[0], g.dP[1], g.dP[2], g.dP[0], g.dP[1], g.dP[2]));
    g.iL = 1.0f / g.L;
    const float grow =
        2.0f * dot3f(d0[0], d0[1], d0[2], du[0], du[1], du[2]) + dot3f(du[0], du[1], du[2], du[0], du[1], du[2]);
    g.C = k.x + grow / (g.L + k.y);
    return g;
}

// Spring (p1, p2) with ends at x1, x2 (positions, or displacements in the displacement
// mode, where consts[at] holds its start constants).
__device__ __forceinline__ Geo spring_geo(const StepArgs& a, int32_t p1, int32_t p2, const float4 x1, const float4 x2,
                                          float rest, const float2* consts, int64_t at) {
    if (!a.gm) return geo_plain(x1, x2, rest);
    return geo_disp(__ldg(a.Xbase + p1), __ldg(a.Xbase + p2), x1, x2, __ldg(consts + at));
}

// The per-spring quantities of CalcForceDerivatives (IMP:719-724) from a geometry.
__device__ __forceinline__ void spring_eval(const Geo& G, const float4 v1, const float4 v2, SpringEval& e) {
    e.C = G.C;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        e.n[c] = G.dP[c] * G.iL;
        e.q[c] = G.dP[c] * G.dP[c];
    }
    e.Cdot = (v1.x * (-e.n[0]) + v1.y * (-e.n[1]) + v1.z * (-e.n[2])) + (v2.x * e.n[0] + v2.y * e.n[1] + v2.z * e.n[2]);
}

// Adjoint of one spring force f = (-Ks C + Kd u) n for dL/df = g.
__device__ __forceinline__ void spring_force_adj(const Geo& G, const float4 v1, const float4 v2, float ks, float kd,
                                                 const float g[3], float gdP[3], float gdV[3], float& gks,
                                                 float& gkd) {
    const float* dP = G.dP;
    const float dV[3] = {v1.x - v2.x, v1.y - v2.y, v1.z - v2.z};
    const float iL = G.iL;
    const float n[3] = {dP[0] * iL, dP[1] * iL, dP[2] * iL};
    const float C = G.C;
    const float u = dot3f(dV[0], dV[1], dV[2], dP[0], dP[1], dP[2]) * iL;
    const float m = -ks * C + kd * u;
    const float gm = dot3f(g[0], g[1], g[2], n[0], n[1], n[2]);
    const float gn[3] = {m * g[0], m * g[1], m * g[2]};
    const float ng = dot3f(n[0], n[1], n[2], gn[0], gn[1], gn[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        gdP[k] = gm * (-ks * n[k] + kd * (dV[k] - u * n[k]) * iL) + (gn[k] - n[k] * ng) * iL;
        gdV[k] = gm * kd * n[k];
    }
    gks = -C * gm;
    gkd = u * gm;
}

// Adjoint of spring i's (J, Jv) for G = dL/dJ, H = dL/dJv (full 3x3, row-major).
__device__ __forceinline__ void spring_jac_adj(const Geo& Gm, const float4 v1, const float4 v2, float ks, float kd,
                                               const float G[3][3], const float H[3][3], float gdP[3], float gdV[3],
                                               float& gks, float& gkd) {
    const float* dP = Gm.dP;
    const float dV[3] = {v1.x - v2.x, v1.y - v2.y, v1.z - v2.z};
    const float iL = Gm.iL;
    const float n[3] = {dP[0] * iL, dP[1] * iL, dP[2] * iL};
    const float C = Gm.C;
    const float Cd = -dot3f(n[0], n[1], n[2], dV[0], dV[1], dV[2]);
    const float w = ks * C + kd * Cd;
    float gS[3][3];
    gks = 0.0f;
    gkd = 0.0f;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float S = n[r] * n[c];
            gS[r][c] = ks * G[r][c] - kd * H[r][c];
            gks += G[r][c] * S;
            gkd += -H[r][c] * S;
        }
    float gw = 0.0f, gC = 0.0f, gq[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float D = C * (1.0f - dP[k] * dP[k]);
        gw += -G[k][k] * D;
        const float gD = -w * G[k][k];
        gC += gD * (1.0f - dP[k] * dP[k]);
        gq[k] = -C * gD;
    }
    gC += ks * gw;
    const float gCd = kd * gw;
    gks += C * gw;
    gkd += Cd * gw;
    float gn[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        gn[r] = (gS[r][0] + gS[0][r]) * n[0] + (gS[r][1] + gS[1][r]) * n[1] + (gS[r][2] + gS[2][r]) * n[2] -
                gCd * dV[r];
    const float ng = dot3f(n[0], n[1], n[2], gn[0], gn[1], gn[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        gdV[k] = -gCd * n[k];
        gdP[k] = 2.0f * dP[k] * gq[k] + gC * n[k] + (gn[k] - n[k] * ng) * iL;
    }
}

// Per vertex i: lambda -> g_F = h lambda, the terms of A_i and b_i: g_J = h^2 lambda (V +
// dV)^T, g_Jv = h lambda dV^T, g_V += h^2 J lambda + damping g_F, g_ext += g_F; spring
// i's Jacobian adjoint goes to the vertex's own-spring slots and to Ks_i, Kd_i.
// One vertex a thread with every load of a stage in flight together (the vertex's own entries, then
// spring i's ends and old gradient entries, then the arithmetic).  A CTA takes kAdjChunk of a block's
// vertices: measured, 24 cloths (231k vertices), 15.9 -> 10.6 us; a CTA of 256 threads for a whole
// block of 384 vertices leaves half its threads idle in a second pass.  Eight CTAs an SM; six 10.9,
// five 13.6.
__global__ void __launch_bounds__(kAdjChunk, 8) k_adj_vertex(const StepArgs a, const AdjArgs j) {
    const BlockInfo bi = a.blocks[blockIdx.x + a.blk_base];
    const InstParams& ip = a.inst[bi.inst];
    const float h = a.dt;
    const int64_t g = bi.v_begin + (int64_t)blockIdx.y * kAdjChunk + threadIdx.x;
    if (g >= bi.v_end) return;
    const float4 Vg = a.V[g];
    float lam[3], dv[3], gv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lam[k] = a.x[k][g];
        dv[k] = j.dV[k][g];
        gv[k] = j.gV[k][g];
    }
    OwnSpring os;
    os.ends = __ldg(a.own_ends + g);
    const int32_t sid = __ldg(j.own_sid + g);
    const bool pinned = Vg.w != 0.0f, own = os.ends.x >= 0 && !pinned;
    float gk_old = 0.0f, gd_old = 0.0f;
    if (own) {
        os.par = __ldg(a.own_par + g);
        os.E1 = __ldg(a.X + os.ends.x);
        os.E2 = __ldg(a.X + os.ends.y);
        os.W1 = __ldg(a.V + os.ends.x);
        os.W2 = __ldg(a.V + os.ends.y);
        gk_old = j.gKs[sid];
        gd_old = j.gKd[sid];
    }
    const float v[3] = {Vg.x, Vg.y, Vg.z};
    float gF[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) gF[k] = pinned ? 0.0f : h * lam[k];
    float gdP[3] = {0.f, 0.f, 0.f}, gdVs[3] = {0.f, 0.f, 0.f};
    if (own) {
        const Geo geo = spring_geo(a, os.ends.x, os.ends.y, os.E1, os.E2, os.par.x, a.gm_own, g);
        SpringEval e;
        spring_eval(geo, os.W1, os.W2, e);
        float J[6], Jv[6];
        jac_element(e, os.par.y, os.par.z, 0, 0, J[0], Jv[0]);
        jac_element(e, os.par.y, os.par.z, 0, 1, J[1], Jv[1]);
        jac_element(e, os.par.y, os.par.z, 0, 2, J[2], Jv[2]);
        jac_element(e, os.par.y, os.par.z, 1, 1, J[3], Jv[3]);
        jac_element(e, os.par.y, os.par.z, 1, 2, J[4], Jv[4]);
        jac_element(e, os.par.y, os.par.z, 2, 2, J[5], Jv[5]);
        float jl0, jl1, jl2;
        matvec(J, lam[0], lam[1], lam[2], jl0, jl1, jl2);
        gv[0] += h * h * jl0;
        gv[1] += h * h * jl1;
        gv[2] += h * h * jl2;
        float G[3][3], H[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                G[r][c] = h * h * lam[r] * (v[c] + dv[c]);
                H[r][c] = h * lam[r] * dv[c];
            }
        float gks, gkd;
        spring_jac_adj(geo, os.W1, os.W2, os.par.y, os.par.z, G, H, gdP, gdVs, gks, gkd);
        j.gKs[sid] = gk_old + gks;
        j.gKd[sid] = gd_old + gkd;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        gv[k] += ip.damping * gF[k];
        j.gV[k][g] = gv[k];
        j.gF[k][g] = gF[k];
        j.gOwn[k][g] = gdP[k];
        j.gOwn[3 + k][g] = gdVs[k];
        if (!pinned) j.gExt[k][g] += gF[k];
    }
}

// Per vertex v: every incident spring's force adjoint, in spring-id order (the spring's
// p1 side also adds to Ks_s, Kd_s), then the own-spring Jacobian terms of the vertices
// whose spring touches v.  The incidences are taken kAdjAhead at a time: their
// neighbours' states and gradient entries are all in flight before the first is used.
// An incidence comes from the vertex's record (neighbour | p2 flag, rest, Ks, Kd), or,
// for a grid cloth whose parameters fit its stencil slots (the forward's stencil
// condition), from its class's template entry: the neighbour offset and the parameter
// slot, no record read (rest lengths that vary from rest_inc, as the forward reads them).
// Both give the same incidences in the same order, so the same bits.  A spring's Ks / Kd
// gradient is written only by its p1 vertex, so its old value can be fetched early.
struct AdjInc {
    int32_t o;      // the other end
    bool p2;        // this vertex is the spring's p2
    float rest, ks, kd;
};

template <bool STENCIL, bool STAGED, bool GM, int kAdjAhead>
__device__ __forceinline__ void adj_springs_vertex(const StepArgs& a, const AdjArgs& j, const InstParams& ip,
                                                   int64_t g, const int4* s_rec, const int32_t* s_sid, int32_t kA) {
    const float4* __restrict__ X = a.X;
    const float4* __restrict__ V = a.V;
    const float* __restrict__ gF0 = j.gF[0];
    const float* __restrict__ gF1 = j.gF[1];
    const float* __restrict__ gF2 = j.gF[2];
    const float4 Xg = __ldg(X + g), Vg = __ldg(V + g);
    const float4 Bg = GM ? __ldg(a.Xbase + g) : Xg;
    const float gFg[3] = {__ldg(gF0 + g), __ldg(gF1 + g), __ldg(gF2 + g)};
    float gx[3] = {j.gX[0][g], j.gX[1][g], j.gX[2][g]};
    float gv[3] = {j.gV[0][g], j.gV[1][g], j.gV[2][g]};
    const int32_t k0 = __ldg(a.rowptr + g), k1 = __ldg(a.rowptr + g + 1);
    const int32_t o0 = __ldg(j.own_rowptr + g), o1 = __ldg(j.own_rowptr + g + 1);
    prefetch_l1(j.own_ent + o0);
    const int32_t* st = nullptr;
    const float4* par = nullptr;
    int32_t ebase = 0;
    const int32_t cols = ip.grid_cols;
    if constexpr (STENCIL) {
        const int32_t l = (int32_t)(g - ip.v_off);
        const int32_t r = l / cols, c = l - r * cols;
        st = a.st_data + ip.st_off;
        par = a.st_param + ip.st_par;
        ebase = __ldg(st + stencil_class_1d(r, ip.grid_rows) * 6 + stencil_class_1d(c, cols)) - k0;
    }
    for (int32_t kb = k0; kb < k1; kb += kAdjAhead) {
        AdjInc in[kAdjAhead];
        int32_t sid[kAdjAhead];
#pragma unroll
        for (int u = 0; u < kAdjAhead; ++u) {
            const int32_t k = kb + u;
            if (k >= k1) {
                in[u] = AdjInc{(int32_t)g, true, 0.0f, 0.0f, 0.0f};
            } else if constexpr (STENCIL) {
                const int32_t v = __ldg(st + ebase + k);
                const int32_t di = (v & 7) - 2, dj = ((v >> 3) & 7) - 2;
                const float4 p = __ldg(par + (v >> 7));
                in[u] = AdjInc{(int32_t)(g + (int64_t)di * cols + dj), (v & 64) != 0,
                               ip.st_rest ? __ldg(a.rest_inc + k) : p.x, p.y, p.z};
            } else {
                const int4 rec = STAGED ? s_rec[k - kA] : __ldg(a.inc + k);
                in[u] = AdjInc{rec.x & 0x7fffffff, rec.x < 0, __int_as_float(rec.y), __int_as_float(rec.z),
                               __int_as_float(rec.w)};
            }
            sid[u] = (k < k1 && !in[u].p2) ? (STAGED ? s_sid[k - kA] : __ldg(j.inc_sid + k)) : 0;
        }
        float4 Xo[kAdjAhead], Vo[kAdjAhead], Bo[GM ? kAdjAhead : 1];
        float2 Ko[GM ? kAdjAhead : 1];  // displacement mode: the other end's base and the constants
        float gFo[kAdjAhead][3], gk_old[kAdjAhead], gd_old[kAdjAhead];
#pragma unroll
        for (int u = 0; u < kAdjAhead; ++u) {
            const int32_t o = in[u].o;
            Xo[u] = __ldg(X + o);
            Vo[u] = __ldg(V + o);
            if constexpr (GM) {
                Bo[u] = __ldg(a.Xbase + o);
                Ko[u] = __ldg(a.gm_inc + min(kb + u, k1 - 1));
            }
            gFo[u][0] = __ldg(gF0 + o);
            gFo[u][1] = __ldg(gF1 + o);
            gFo[u][2] = __ldg(gF2 + o);
            const bool p1 = kb + u < k1 && !in[u].p2;
            gk_old[u] = p1 ? j.gKs[sid[u]] : 0.0f;
            gd_old[u] = p1 ? j.gKd[sid[u]] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kAdjAhead; ++u) {
            if (kb + u >= k1) break;
            const bool as_p2 = in[u].p2;
            // g_f = [p1 free] gF[p1] - [p2 free] gF[p2]; k_adj_vertex leaves gF = 0 at
            // pinned vertices.
            float gf[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) gf[c] = as_p2 ? gFo[u][c] - gFg[c] : gFg[c] - gFo[u][c];
            float gdP[3], gdV[3], gks, gkd;
            if (as_p2) {
                Geo geo;
                if constexpr (GM) geo = geo_disp(Bo[u], Bg, Xo[u], Xg, Ko[u]);
                else geo = geo_plain(Xo[u], Xg, in[u].rest);
                spring_force_adj(geo, Vo[u], Vg, in[u].ks, in[u].kd, gf, gdP, gdV, gks, gkd);
            } else {
                Geo geo;
                if constexpr (GM) geo = geo_disp(Bg, Bo[u], Xg, Xo[u], Ko[u]);
                else geo = geo_plain(Xg, Xo[u], in[u].rest);
                spring_force_adj(geo, Vg, Vo[u], in[u].ks, in[u].kd, gf, gdP, gdV, gks, gkd);
            }
            const float sgn = as_p2 ? -1.0f : 1.0f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                gx[c] += sgn * gdP[c];
                gv[c] += sgn * gdV[c];
            }
            if (!as_p2) {
                j.gKs[sid[u]] = gk_old[u] + gks;
                j.gKd[sid[u]] = gd_old[u] + gkd;
            }
        }
    }
    for (int32_t k = o0; k < o1; ++k) {
        const int32_t e = __ldg(j.own_ent + k);
        const int32_t i = e & 0x7fffffff;
        const float sgn = e < 0 ? -1.0f : 1.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            gx[c] += sgn * j.gOwn[c][i];
            gv[c] += sgn * j.gOwn[3 + c][i];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        j.gX[c][g] = gx[c];
        j.gV[c][g] = gv[c];
    }
}

// The chunk's incidence records (contiguous) and spring ids are copied to shared memory first
// (STAGE): read from memory by their threads they are 192 bytes apart, a line each, and the
// neighbours' loads wait for them.  T threads, a vertex each; AHEAD incidences in flight; grid.y CTAs
// take the chunks of a block of the table in turn (the grid's x-neighbours, which run together, are
// then a block apart: with adjacent chunks the same kernel took 67 us instead of 50).
// Measured, 24 cloths (231k vertices, a record a spring), us: 89 with <2, 256, 3, false> over whole
// blocks, 67 with <4, 128, 4, false> over chunks, 50 with <4, 128, 4, true>; two incidences and six
// CTAs an SM 78, three and four 62, six and three 59; 64 threads 56; four and three 57 (the copies
// and the gathered states share an SM's L1).  700 x 700 stencil 133 -> 101.  GM: the displacement
// mode, whose bases and constants are loaded with the neighbour's state: 257 x 257 32 -> 18, 600 x 600
// 139 -> 84 (loaded at their use 257 x 257 22; three incidences 28, four at three CTAs 24).
constexpr int kSpringStage = 13;  // records of a vertex that the copies have room for, on average

template <int AHEAD, int T, int MINB, bool STAGE, bool GM>
__global__ void __launch_bounds__(T, MINB) k_adj_springs(const StepArgs a, const AdjArgs j) {
    __shared__ int4 s_rec[STAGE ? T * kSpringStage : 1];
    __shared__ int32_t s_sid[STAGE ? T * kSpringStage : 1];
    const BlockInfo bi = a.blocks[blockIdx.x + a.blk_base];
    const InstParams& ip = a.inst[bi.inst];
    const bool stencil = ip.grid_cols > 0;
    for (int64_t base = bi.v_begin + (int64_t)blockIdx.y * T; base < bi.v_end; base += (int64_t)gridDim.y * T) {
        const int64_t g = base + threadIdx.x, end = min(base + T, bi.v_end);
        int32_t kA = 0;
        bool staged = false;
        if constexpr (STAGE) {
            kA = __ldg(a.rowptr + base);
            const int32_t n = __ldg(a.rowptr + end) - kA;
            staged = n <= T * kSpringStage;
            __syncthreads();  // the last copies have been read
            if (staged) {
                for (int i = threadIdx.x; i < n; i += T) {
                    if (!stencil) copy_async16(s_rec + i, a.inc + kA + i);
                    copy_async4(s_sid + i, j.inc_sid + kA + i);
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
            __syncthreads();
        }
        if (g >= end) continue;
        if (stencil) {
            if (staged) adj_springs_vertex<true, true, GM, AHEAD>(a, j, ip, g, s_rec, s_sid, kA);
            else adj_springs_vertex<true, false, GM, AHEAD>(a, j, ip, g, s_rec, s_sid, kA);
        } else {
            if (staged) adj_springs_vertex<false, true, GM, AHEAD>(a, j, ip, g, s_rec, s_sid, kA);
            else adj_springs_vertex<false, false, GM, AHEAD>(a, j, ip, g, s_rec, s_sid, kA);
        }
    }
}

// ---- displacement mode: the taped forward in X = Xbase + u --------------------------------
// An FP32 position near 5 resolves steps of about 5e-7, and an FP32 L - rest loses the
// bits of an elongation 1e-3 of the length, so an FP32 trajectory of a slow cloth drifts
// from the FP64 one by a good fraction of a small loss residual.  In this mode the state
// holds the displacement u from the tape's start and each spring's elongation is formed
// from its FP64-rounded start constants (geo_disp); the forward otherwise follows the
// step's arithmetic, the CG included.

// 0: Xbase = X.
__global__ void k_gm_base(const StepArgs a, int64_t nv) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nv; g += (int64_t)gridDim.x * blockDim.x)
        const_cast<float4*>(a.Xbase)[g] = a.X[g];
}

__device__ __forceinline__ float2 spring_consts(const float4 b1, const float4 b2, float rest) {
    const double dx = (double)b1.x - (double)b2.x, dy = (double)b1.y - (double)b2.y, dz = (double)b1.z - (double)b2.z;
    const double L0 = sqrt(dx * dx + dy * dy + dz * dz);
    return make_float2((float)(L0 - (double)rest), (float)L0);
}

// Threads of a vertex in k_gm_consts: its incidences are a root in FP64 each.  100 x 100 28 -> 15 us;
// four threads 16, and 257 x 257 55 against 50.
constexpr int kGmLanes = 2;

// 4: the spring constants from Xbase, and u = 0 (mass kept in w).
__global__ void k_gm_consts(const StepArgs a, int64_t nv) {
    const int64_t n = nv * kGmLanes, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += step) {
        const int64_t g = t / kGmLanes;
        const int q = (int)(t % kGmLanes);
        const float4 bg = __ldg(a.Xbase + g);
        const int32_t k0 = __ldg(a.rowptr + g), k1 = __ldg(a.rowptr + g + 1);
        for (int32_t k = k0 + q; k <= k1; k += kGmLanes) {  // the incidences, then spring i
            int2 e;
            float rest;
            if (k < k1) {
                const int4 rec = __ldg(a.inc + k);
                const int32_t o = rec.x & 0x7fffffff;
                e = rec.x < 0 ? make_int2(o, (int)g) : make_int2((int)g, o);
                rest = __int_as_float(rec.y);
            } else {
                e = __ldg(a.own_ends + g);
                rest = __ldg(a.own_par + g).x;
            }
            float2 c = make_float2(0.f, 0.f);
            if (e.x >= 0) c = spring_consts(__ldg(a.Xbase + e.x), __ldg(a.Xbase + e.y), rest);
            const_cast<float2*>(k < k1 ? a.gm_inc + k : a.gm_own + g)[0] = c;
        }
        if (q == 0) a.X[g] = make_float4(0.f, 0.f, 0.f, bg.w);
    }
}

// 3: X = Xbase + u.
__global__ void k_gm_leave(const StepArgs a, int64_t nv) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nv; g += (int64_t)gridDim.x * blockDim.x) {
        const float4 b = __ldg(a.Xbase + g), u = a.X[g];
        a.X[g] = make_float4(b.x + u.x, b.y + u.y, b.z + u.z, u.w);
    }
}

// The spring force on p1 (IMP:717-728) from a geometry.
__device__ __forceinline__ float3 spring_force_geo(const Geo& G, const float4 v1, const float4 v2, float ks, float kd) {
    const float dVx = v1.x - v2.x, dVy = v1.y - v2.y, dVz = v1.z - v2.z;
    const float left = (-ks) * G.C;
    const float right = kd * (dot3f(dVx, dVy, dVz, G.dP[0], G.dP[1], G.dP[2]) * G.iL);
    const float mag = left + right;
    return make_float3(mag * (G.dP[0] * G.iL), mag * (G.dP[1] * G.iL), mag * (G.dP[2] * G.iL));
}

// 1: the step's assembly in displacement mode (incidence-record gather in spring order,
// spring i's Jacobians, A and b, the CG set-up), one thread per vertex.
// Spring i's blocks of vertex g in the displacement mode (IMP:744-770 on geo_disp):
// A = M - h (Jv + h J) and h J.  The assembly and the reverse pass's seed both form them
// here.
__device__ __forceinline__ void gm_own_blocks(const StepArgs& a, int64_t g, float mass, float h, float A[6],
                                              float hJ[6]) {
    const OwnSpring os = load_own(a, g);
    float J[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, Jv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (os.ends.x >= 0) {
        SpringEval e;
        spring_eval(spring_geo(a, os.ends.x, os.ends.y, os.E1, os.E2, 0.0f, a.gm_own, g), os.W1, os.W2, e);
        jac_element(e, os.par.y, os.par.z, 0, 0, J[0], Jv[0]);
        jac_element(e, os.par.y, os.par.z, 0, 1, J[1], Jv[1]);
        jac_element(e, os.par.y, os.par.z, 0, 2, J[2], Jv[2]);
        jac_element(e, os.par.y, os.par.z, 1, 1, J[3], Jv[3]);
        jac_element(e, os.par.y, os.par.z, 1, 2, J[4], Jv[4]);
        jac_element(e, os.par.y, os.par.z, 2, 2, J[5], Jv[5]);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const float Mk = (k == 0 || k == 3 || k == 5) ? mass : 0.0f;
        A[k] = Mk - h * (Jv[k] + h * J[k]);
        hJ[k] = h * J[k];
    }
}

// Bound by the latency of an incidence's record, its neighbour and that one's state: two incidences in
// flight at four CTAs an SM, 100 x 100 14.9 -> 12.1 us, 600 x 600 60 -> 54 (four in flight 11.6 and
// 62, at three CTAs 12.8 and 82).
constexpr int kGmAhead = 2;

__global__ void __launch_bounds__(kAdjThreads, 4) k_gm_assemble(const StepArgs a) {
    const int blk = blockIdx.x + a.blk_base;
    const BlockInfo bi = a.blocks[blk];
    const InstParams& ip = a.inst[bi.inst];
    const float h = a.dt;
    Acc part = acc_zero();
    for (int64_t g = bi.v_begin + threadIdx.x; g < bi.v_end; g += blockDim.x) {
        const float4 Ug = a.X[g], Vg = a.V[g];
        const bool pinned = Vg.w != 0.0f;
        float Fx = 0.0f, Fy = 0.0f, Fz = 0.0f;
        if (!pinned) {
            Fx += Ug.w * ip.gravity[0];
            Fy += Ug.w * ip.gravity[1];
            Fz += Ug.w * ip.gravity[2];
        }
        Fx += ip.damping * Vg.x;
        Fy += ip.damping * Vg.y;
        Fz += ip.damping * Vg.z;
        if (!pinned) {
            if (ip.has_ext) {
                const float4 e = __ldg(a.fext + g);
                Fx += e.x;
                Fy += e.y;
                Fz += e.z;
            }
            const int32_t k0 = __ldg(a.rowptr + g), k1 = __ldg(a.rowptr + g + 1);
            const float4 Bg = __ldg(a.Xbase + g);
            for (int32_t kb = k0; kb < k1; kb += kGmAhead) {
                int4 rec[kGmAhead];
                float4 Uo[kGmAhead], Vo[kGmAhead], Bo[kGmAhead];
                float2 Ko[kGmAhead];
#pragma unroll
                for (int u = 0; u < kGmAhead; ++u) {
                    rec[u] = __ldg(a.inc + min(kb + u, k1 - 1));
                    Ko[u] = __ldg(a.gm_inc + min(kb + u, k1 - 1));
                }
#pragma unroll
                for (int u = 0; u < kGmAhead; ++u) {
                    const int32_t o = rec[u].x & 0x7fffffff;
                    Uo[u] = a.X[o];
                    Vo[u] = a.V[o];
                    Bo[u] = __ldg(a.Xbase + o);
                }
#pragma unroll
                for (int u = 0; u < kGmAhead; ++u) {
                    if (kb + u >= k1) break;
                    const float ks = __int_as_float(rec[u].z), kd = __int_as_float(rec[u].w);
                    if (rec[u].x < 0) {  // F[p2] -= f
                        const float3 f = spring_force_geo(geo_disp(Bo[u], Bg, Uo[u], Ug, Ko[u]), Vo[u], Vg, ks, kd);
                        Fx -= f.x;
                        Fy -= f.y;
                        Fz -= f.z;
                    } else {  // F[p1] += f
                        const float3 f = spring_force_geo(geo_disp(Bg, Bo[u], Ug, Uo[u], Ko[u]), Vg, Vo[u], ks, kd);
                        Fx += f.x;
                        Fy += f.y;
                        Fz += f.z;
                    }
                }
            }
        }
        // Spring i's Jacobians (IMP:744-770) and the vertex's system.
        VertexSystem sys;
        float hJ[6];
        gm_own_blocks(a, g, Ug.w, h, sys.A, hJ);
        float wx, wy, wz;
        matvec(hJ, Vg.x, Vg.y, Vg.z, wx, wy, wz);
        sys.b[0] = h * (Fx + wx);
        sys.b[1] = h * (Fy + wy);
        sys.b[2] = h * (Fz + wz);
        const CgInit c = cg_init(sys, a.x[0][g], a.x[1][g], a.x[2][g], pinned);
#pragma unroll
        for (int k = 0; k < 6; ++k) a.A[k][g] = sys.A[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a.x[k][g] = c.x[k];
            a.r[k][g] = c.r[k];
            a.d[k][g] = c.d[k];
        }
        acc_add(part, c.term);
    }
    finish<K_ASSEMBLE>(a, bi.gblk, bi.inst, true, part);
}

// The reverse pass's seed in the displacement mode: spring i's blocks rebuilt as the
// assembly formed them (A planes written), then adj_seed_vertex and the epilogue.
__global__ void __launch_bounds__(kAdjThreads) k_gm_seed_own(const StepArgs a, const AdjArgs j) {
    const int blk = blockIdx.x + a.blk_base;
    const BlockInfo bi = a.blocks[blk];
    Acc part = acc_zero();
    for (int64_t g = bi.v_begin + threadIdx.x; g < bi.v_end; g += blockDim.x) {
        const float4 Ug = a.X[g], Vg = a.V[g];
        float A[6], hJ[6];
        gm_own_blocks(a, g, Ug.w, a.dt, A, hJ);
#pragma unroll
        for (int k = 0; k < 6; ++k) a.A[k][g] = A[k];
        acc_add(part, adj_seed_vertex(a, j, g, Ug, Vg, A[0], A[3], A[5]));
    }
    finish<K_ASSEMBLE>(a, bi.gblk, bi.inst, true, part);
}

// 2: V += dV dt, u += dt V, ground clamp on the position (IMP:790-797).
__global__ void __launch_bounds__(kAdjThreads) k_gm_update(const StepArgs a) {
    const int blk = blockIdx.x + a.blk_base;
    const BlockInfo bi = a.blocks[blk];
    const float dt = a.dt;
    for (int64_t g = bi.v_begin + threadIdx.x; g < bi.v_end; g += blockDim.x) {
        float4 U = a.X[g], V = a.V[g];
        gm_advance(dt, a.x[0][g], a.x[1][g], a.x[2][g], __ldg(a.Xbase + g).y, U, V);
        a.X[g] = U;
        a.V[g] = V;
    }
}

// Per-spring Ks / Kd into the incidence records and spring i's parameters.
__global__ void k_set_spring_params(const StepArgs a, const AdjArgs j, const float* ks, const float* kd, int64_t n_rec,
                                    int64_t nv) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n_rec; k += stride) {
        const int32_t s = j.inc_sid[k];
        int4 rec = a.inc[k];
        rec.z = __float_as_int(ks[s]);
        rec.w = __float_as_int(kd[s]);
        const_cast<int4*>(a.inc)[k] = rec;
    }
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nv; g += stride) {
        const int32_t s = j.own_sid[g];
        if (s >= 0) {
            float4 p = a.own_par[g];
            p.y = ks[s];
            p.z = kd[s];
            const_cast<float4*>(a.own_par)[g] = p;
        }
    }
}

}  // namespace

cudaError_t launch_adjoint(int which, const StepArgs& a, const AdjArgs& j, int nblocks, int vpb, bool stencil,
                           cudaStream_t stream) {
    if (nblocks <= 0) return cudaSuccess;
    const int parts = (vpb + kAdjChunk - 1) / kAdjChunk;
    switch (which) {
        case 0: k_gm_seed_own<<<nblocks, kAdjThreads, 0, stream>>>(a, j); break;
        case 1: k_adj_vertex<<<dim3(nblocks, parts), kAdjChunk, 0, stream>>>(a, j); break;
        case 2:
            // Large handles of stencil cloths alone read no records to copy, and their whole blocks
            // make waves enough: 2 M vertices 327 us against 366, 4 M 624 against 741.
            if (stencil && (int64_t)nblocks * vpb >= 1500000) {
                if (a.gm) k_adj_springs<2, kAdjThreads, 2, false, true><<<nblocks, kAdjThreads, 0, stream>>>(a, j);
                else k_adj_springs<2, kAdjThreads, 3, false, false><<<nblocks, kAdjThreads, 0, stream>>>(a, j);
            } else {
                const dim3 grid(nblocks, std::min(parts, 3));
                if (a.gm) k_adj_springs<4, kAdjChunk, 4, true, true><<<grid, kAdjChunk, 0, stream>>>(a, j);
                else k_adj_springs<4, kAdjChunk, 4, true, false><<<grid, kAdjChunk, 0, stream>>>(a, j);
            }
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}


cudaError_t launch_gm(int which, const StepArgs& a, int n, cudaStream_t stream) {
    const int64_t nv = (int64_t)n;  // the per-vertex kernels (0, 3, 4) take the vertex count
    const int gs = (int)std::max<int64_t>(1, std::min<int64_t>((nv + kAdjThreads - 1) / kAdjThreads, 152 * 8));
    switch (which) {
        case 0: k_gm_base<<<gs, kAdjThreads, 0, stream>>>(a, nv); break;
        case 1: if (n > 0) k_gm_assemble<<<n, kAdjThreads, 0, stream>>>(a); break;
        case 2: if (n > 0) k_gm_update<<<n, kAdjThreads, 0, stream>>>(a); break;
        case 3: k_gm_leave<<<gs, kAdjThreads, 0, stream>>>(a, nv); break;
        case 4:
            k_gm_consts<<<(int)std::max<int64_t>(1, std::min<int64_t>((nv * kGmLanes + kAdjThreads - 1) / kAdjThreads, 152 * 8)),
                          kAdjThreads, 0, stream>>>(a, nv);
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_set_spring_params(const StepArgs& a, const AdjArgs& j, const float* ks, const float* kd,
                                     int64_t n_rec, int64_t nv, cudaStream_t stream) {
    k_set_spring_params<<<152 * 8, 256, 0, stream>>>(a, j, ks, kd, n_rec, nv);
    return cudaGetLastError();
}

}  // namespace oc
