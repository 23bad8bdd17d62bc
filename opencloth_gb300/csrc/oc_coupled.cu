// COUPLED Jacobian mode: Baraff-Witkin coupling of the per-spring blocks into one
// symmetric positive-definite block-sparse system per cloth, solved by a block-Jacobi
// preconditioned CG.  The reference has no such system (its vertex i takes spring i's
// blocks alone, IMP:782); the mode is defined on the reference's own force model:
//
//   (M' + sum_s [B_s, -B_s; -B_s, B_s]) dV = h (F - h sum_s Kt_s (v_i - v_j)),  V += dV
//
// with, for spring s and n = (x1 - x2) / |x1 - x2|,
//   Kt_s = kst I + (ksn - kst) n n^T,   ksn = max(ks, 0),  kst = ksn max(1 - L/l, 0)
//   B_s  = beta I + gamma n n^T,        beta = h^2 kst,  gamma = (h kdn + h^2 ksn) - beta,
//                                       kdn = max(-kd, 0)
//   M'   = (m + h max(-c, 0)) I,        c the velocity damping.
// The clamps keep every B_s positive semi-definite (the transverse term is dropped for a
// compressed spring), so the CG always sees an SPD system.  Pinned vertices are
// Dirichlet rows filtered out of the CG.
//
//   k_cpl_assemble  F (the reference's forces, bit for bit), each incidence's B_s into
//                   slot-major per-incidence planes (StepArgs::cpl_slice), the diagonal block and its inverse P^-1, b, and
//                   the CG set-up r = b - A x, z = P^-1 r, delta0 = r.z
//   k_cpl_dir       dn = z + beta d (first pass: z); q = A dn with the neighbours' dn
//                   rebuilt from their z and d; d.q
//   k_cpl_update    dn again; x += alpha dn; r -= alpha q; d = dn; z = P^-1 r; r.z
//   k_cpl_persist   all iterations of the two and the update of X and V in one cooperative
//                   launch, when every other cloth is resident and there are no more COUPLED
//                   cloths than SMs (else a WHILE loop of the two)
//
// The direction is never written during the matrix-vector pass, so a vertex's
// neighbours read its previous d and z while it runs: no second buffer is needed.
// Every per-vertex sum runs over the vertex's incidence records in spring-id order with
// a fixed operand order, the same expressions as the CPU restatement
// (oracle/oc_coupled_impl.h), and the CG scalars go through the streamed executor's
// deterministic per-instance reductions (finish in oc_device.cuh).
#include <cuda_runtime.h>

#include "oc_device.cuh"
#include "oc_exchange.cuh"
#include "oc_internal.h"

namespace oc {
namespace {

constexpr int kThreads = 256;

// What a spring gives the vertex at one of its ends, taken as its p1 whichever end it is: with the
// ends exchanged d, v and n are the exact negations, so the force is that of the other side (as in
// add_spring_forces) and every use of n below, which is even in it, gives the same float.
struct CplSpring {
    float3 f, n;
    float beta, gamma, ksn, kst;
};

__device__ __forceinline__ CplSpring spring_eval(const float3 d, const float3 v, float rest, float ks, float kd,
                                                   float h, float hh) {
    CplSpring c;
    const float sqr = d.x * d.x + d.y * d.y + d.z * d.z;
    const float dot = v.x * d.x + v.y * d.y + v.z * d.z;
    // The force's and the block's divisions by the length share its root and reciprocal.
    float l = sqrt_cr(sqr), inv = rcp_cr(l), q = div_cr(dot, l, inv), rl = div_cr(rest, l, inv);
    c.n = make_float3(div_cr(d.x, l, inv), div_cr(d.y, l, inv), div_cr(d.z, l, inv));
    if (!(cr_arg(sqr) && cr_num(dot) && cr_num(d.x) && cr_num(d.y) && cr_num(d.z) && cr_num(rest))) {
        l = __fsqrt_rn(sqr);
        inv = __frcp_rn(l);
        q = __fdiv_rn(dot, l);
        rl = __fdiv_rn(rest, l);
        c.n = make_float3(__fdiv_rn(d.x, l), __fdiv_rn(d.y, l), __fdiv_rn(d.z, l));
    }
    const float mag = (-ks) * (l - rest) + kd * q;
    c.f = make_float3(mag * (d.x * inv), mag * (d.y * inv), mag * (d.z * inv));
    c.ksn = ks > 0.0f ? ks : 0.0f;
    const float kdn = -kd > 0.0f ? -kd : 0.0f;
    const float t = 1.0f - rl;
    c.kst = c.ksn * (t > 0.0f ? t : 0.0f);
    c.beta = hh * c.kst;
    c.gamma = (h * kdn + hh * c.ksn) - c.beta;
    return c;
}

// acc += beta e + (gamma (n.e)) n
__device__ __forceinline__ void block_apply(float n0, float n1, float n2, float beta, float gamma, float e0, float e1,
                                            float e2, float& a0, float& a1, float& a2) {
    const float ne = n0 * e0 + n1 * e1 + n2 * e2;
    const float g = gamma * ne;
    a0 = a0 + (beta * e0 + g * n0);
    a1 = a1 + (beta * e1 + g * n1);
    a2 = a2 + (beta * e2 + g * n2);
}

// Bound by instructions and the registers that hide the gather's latency.  A spring's force and its
// block share one root, one reciprocal and the divisions by them, and neither branches on the side:
// 54 -> 41 us on a 513 x 511 cloth (12 incidences a vertex).  Three blocks an SM (no spills) 45,
// five 47.
__global__ void __launch_bounds__(kThreads, 4) k_cpl_assemble(const StepArgs a) {
    const int blk = blockIdx.x + a.blk_base;
    const BlockInfo bi = a.blocks[blk];
    const InstParams& ip = a.inst[bi.inst];
    const float h = a.dt, hh = h * h;
    const float nc = -ip.damping;
    const float mdamp = h * (nc > 0.0f ? nc : 0.0f);
    Acc part = acc_zero();
    for (int64_t g = bi.v_begin + threadIdx.x; g < bi.v_end; g += blockDim.x) {
        const float4 Xg = __ldg(a.X + g), Vg = __ldg(a.V + g);
        const bool pinned = Vg.w != 0.0f;
        const float mp = Xg.w + mdamp;
        float xi0 = a.x[0][g], xi1 = a.x[1][g], xi2 = a.x[2][g];
        if (pinned) xi0 = xi1 = xi2 = 0.0f;
        // Forces in the reference's order (IMP:701-734): gravity unless pinned, damping,
        // external force unless pinned, then the springs in spring-id order.
        float Fx = 0.0f, Fy = 0.0f, Fz = 0.0f;
        if (!pinned) {
            Fx += Xg.w * ip.gravity[0];
            Fy += Xg.w * ip.gravity[1];
            Fz += Xg.w * ip.gravity[2];
        }
        Fx += ip.damping * Vg.x;
        Fy += ip.damping * Vg.y;
        Fz += ip.damping * Vg.z;
        if (!pinned && ip.has_ext) {
            const float4 e = __ldg(a.fext + g);
            Fx += e.x;
            Fy += e.y;
            Fz += e.z;
        }
        float D[6] = {mp, 0.0f, 0.0f, mp, 0.0f, mp};
        float w0 = 0.0f, w1 = 0.0f, w2 = 0.0f;
        float ax0 = mp * xi0, ax1 = mp * xi1, ax2 = mp * xi2;
        const int64_t slot0 = __ldg(a.cpl_slice + (g >> 5)) + (g & 31);
        // Incidence e of the vertex (spring-id order): neighbour o and the spring's parameters.
        auto incidence = [&](int32_t e, int32_t o, float rest, float ks, float kd) {
            const int64_t sk = slot0 + 32 * (int64_t)e;
            const float4 Xo = __ldg(a.X + o), Vo = __ldg(a.V + o);
            float xo0 = a.x[0][o], xo1 = a.x[1][o], xo2 = a.x[2][o];
            // A x with the warm start filtered: a pinned neighbour's x counts as zero.
            if (Vo.w != 0.0f) xo0 = xo1 = xo2 = 0.0f;
            const float u0 = Vg.x - Vo.x, u1 = Vg.y - Vo.y, u2 = Vg.z - Vo.z;
            const CplSpring c = spring_eval(make_float3(Xg.x - Xo.x, Xg.y - Xo.y, Xg.z - Xo.z),
                                              make_float3(u0, u1, u2), rest, ks, kd, h, hh);
            if (!pinned) {  // pinned vertices take no spring force (IMP:730-733)
                Fx += c.f.x;
                Fy += c.f.y;
                Fz += c.f.z;
            }
            const float n0 = c.n.x, n1 = c.n.y, n2 = c.n.z;
            a.cpl_nb[sk] = make_float4(n0, n1, n2, c.beta);
            a.cpl_go[sk] = make_float2(c.gamma, __int_as_float(o));
            const float g0 = c.gamma * n0, g1 = c.gamma * n1, g2 = c.gamma * n2;
            D[0] = D[0] + (c.beta + g0 * n0);
            D[1] = D[1] + g0 * n1;
            D[2] = D[2] + g0 * n2;
            D[3] = D[3] + (c.beta + g1 * n1);
            D[4] = D[4] + g1 * n2;
            D[5] = D[5] + (c.beta + g2 * n2);
            const float nu = n0 * u0 + n1 * u1 + n2 * u2;
            const float kk = (c.ksn - c.kst) * nu;
            w0 = w0 + (c.kst * u0 + kk * n0);
            w1 = w1 + (c.kst * u1 + kk * n1);
            w2 = w2 + (c.kst * u2 + kk * n2);
            block_apply(n0, n1, n2, c.beta, c.gamma, xi0 - xo0, xi1 - xo1, xi2 - xo2, ax0, ax1, ax2);
        };
        if (ip.grid_cols > 0) {  // grid cloth: its class's stencil template, no records
            const int32_t cols = ip.grid_cols;
            const int32_t l = (int32_t)(g - ip.v_off), row = l / cols, col = l - row * cols;
            const int cl = stencil_class_1d(row, ip.grid_rows) * 6 + stencil_class_1d(col, cols);
            const int32_t* st = a.st_data + ip.st_off;
            const float4* par = a.st_param + ip.st_par;
            const int32_t e0 = __ldg(st + cl), e1 = __ldg(st + cl + 1);
            const float* rest_inc = ip.st_rest ? a.rest_inc + __ldg(a.rowptr + g) - e0 : nullptr;
            for (int32_t e = e0; e < e1; ++e) {
                const int32_t v = __ldg(st + e);
                const float4 p = __ldg(par + (v >> 7));
                const int32_t o = (int32_t)(g + (int64_t)((v & 7) - 2) * cols + (((v >> 3) & 7) - 2));
                incidence(e - e0, o, rest_inc ? __ldg(rest_inc + e) : p.x, p.y, p.z);
            }
        } else {
            const int32_t k0 = __ldg(a.rowptr + g), k1 = __ldg(a.rowptr + g + 1);
            for (int32_t k = k0; k < k1; ++k) {
                const int4 rec = __ldg(a.inc + k);
                incidence(k - k0, rec.x & 0x7fffffff, __int_as_float(rec.y), __int_as_float(rec.z),
                          __int_as_float(rec.w));
            }
        }
        const float c00 = D[3] * D[5] - D[4] * D[4], c01 = D[2] * D[4] - D[1] * D[5], c02 = D[1] * D[4] - D[2] * D[3];
        const float c11 = D[0] * D[5] - D[2] * D[2], c12 = D[1] * D[2] - D[0] * D[4], c22 = D[0] * D[3] - D[1] * D[1];
        const float det = D[0] * c00 + D[1] * c01 + D[2] * c02;
        const float inv = 1.0f / det;
        const float P[6] = {c00 * inv, c01 * inv, c02 * inv, c11 * inv, c12 * inv, c22 * inv};
        const float b0 = h * (Fx - h * w0), b1 = h * (Fy - h * w1), b2 = h * (Fz - h * w2);
        float r0 = 0.0f, r1 = 0.0f, r2 = 0.0f, z0 = 0.0f, z1 = 0.0f, z2 = 0.0f;
        if (!pinned) {
            r0 = b0 - ax0;
            r1 = b1 - ax1;
            r2 = b2 - ax2;
            matvec(P, r0, r1, r2, z0, z1, z2);
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) a.A[k][g] = P[k];
        a.cpl_m[g] = mp;
        a.r[0][g] = r0;
        a.r[1][g] = r1;
        a.r[2][g] = r2;
        a.cpl_z[g] = make_float4(z0, z1, z2, 0.0f);
        a.cpl_d[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (pinned) {
            a.x[0][g] = 0.0f;
            a.x[1][g] = 0.0f;
            a.x[2][g] = 0.0f;
        }
        acc_add(part, r0 * z0 + r1 * z1 + r2 * z2);
    }
    finish<K_ASSEMBLE>(a, bi.gblk, bi.inst, true, part);
}

__global__ void __launch_bounds__(kThreads) k_cpl_dir(const StepArgs a) {
    const int blk = blockIdx.x + a.blk_base;
    const BlockInfo bi = a.blocks[blk];
    const InstState& st = a.state[bi.inst];
    const bool active = st.active != 0;
    Acc part = acc_zero();
    if (active) {
        const bool first = st.iter == 0;
        const float beta = st.beta;
        const float4* __restrict__ Z = a.cpl_z;
        const float4* __restrict__ D = a.cpl_d;
        for (int64_t g = bi.v_begin + threadIdx.x; g < bi.v_end; g += blockDim.x) {
            float q0 = 0.0f, q1 = 0.0f, q2 = 0.0f;
            if (!__ldg(a.pinflag + g)) {
                const float4 zg = Z[g];
                float n0 = zg.x, n1 = zg.y, n2 = zg.z;
                if (!first) {
                    const float4 dg = D[g];
                    n0 = n0 + dg.x * beta;
                    n1 = n1 + dg.y * beta;
                    n2 = n2 + dg.z * beta;
                }
                const float mp = __ldg(a.cpl_m + g);
                q0 = mp * n0;
                q1 = mp * n1;
                q2 = mp * n2;
                const int32_t deg = __ldg(a.rowptr + g + 1) - __ldg(a.rowptr + g);
                const int64_t slot0 = __ldg(a.cpl_slice + (g >> 5)) + (g & 31);
                // The per-incidence planes are read once per pass (evict-first, .cs), so
                // the gathered z and d records stay in L2.
                for (int32_t e = 0; e < deg; ++e) {
                    const int64_t k = slot0 + 32 * (int64_t)e;
                    const float4 nb = __ldcs(a.cpl_nb + k);
                    const float2 go = __ldcs(a.cpl_go + k);
                    if (e + 1 < deg) {
                        prefetch_l1(a.cpl_nb + k + 32);
                        prefetch_l1(a.cpl_go + k + 32);
                    }
                    const int32_t o = __float_as_int(go.y);
                    const float4 zo = Z[o];
                    float m0 = zo.x, m1 = zo.y, m2 = zo.z;
                    if (!first) {
                        const float4 dd = D[o];
                        m0 = m0 + dd.x * beta;
                        m1 = m1 + dd.y * beta;
                        m2 = m2 + dd.z * beta;
                    }
                    block_apply(nb.x, nb.y, nb.z, nb.w, go.x, n0 - m0, n1 - m1, n2 - m2, q0, q1, q2);
                }
                acc_add(part, n0 * q0 + n1 * q1 + n2 * q2);
            }
            a.q[0][g] = q0;
            a.q[1][g] = q1;
            a.q[2][g] = q2;
        }
    }
    finish<K_CG_DIR>(a, bi.gblk, bi.inst, active, part);
}

__global__ void __launch_bounds__(kThreads) k_cpl_update(const StepArgs a) {
    const int blk = blockIdx.x + a.blk_base;
    const BlockInfo bi = a.blocks[blk];
    const InstState& st = a.state[bi.inst];
    const bool active = st.active != 0;
    Acc part = acc_zero();
    if (active) {
        const bool first = st.iter == 0;
        const float alpha = st.alpha, beta = st.beta;
        for (int64_t g = bi.v_begin + threadIdx.x; g < bi.v_end; g += blockDim.x) {
            float dn[3], r[3];
            const float4 zg = a.cpl_z[g], dg = a.cpl_d[g];
            const float zv[3] = {zg.x, zg.y, zg.z}, dv[3] = {dg.x, dg.y, dg.z};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float v = zv[k];
                if (!first) v = v + dv[k] * beta;
                dn[k] = v;
                a.x[k][g] = a.x[k][g] + dn[k] * alpha;
                r[k] = a.r[k][g] - a.q[k][g] * alpha;
                a.r[k][g] = r[k];
            }
            a.cpl_d[g] = make_float4(dn[0], dn[1], dn[2], 0.0f);
            const float P[6] = {a.A[0][g], a.A[1][g], a.A[2][g], a.A[3][g], a.A[4][g], a.A[5][g]};
            float z0, z1, z2;
            matvec(P, r[0], r[1], r[2], z0, z1, z2);
            a.cpl_z[g] = make_float4(z0, z1, z2, 0.0f);
            acc_add(part, r[0] * z0 + r[1] * z1 + r[2] * z2);
        }
    }
    finish<K_CG_UPDATE>(a, bi.gblk, bi.inst, active, part);
}

// The CG loop and the update of the COUPLED cloths in one cooperative launch.  A CTA keeps its
// vertices' x, r, dn, q, P^-1 and m' in shared memory (its first P.smem_rows vertices; the others
// stay in the planes) and writes only what the neighbours gather, z and d.  An iteration is the
// two passes above with one exchange behind each: the first so that every CTA has read z and d
// before they are written, the second so that they are written before they are read.  The
// exchange carries the pass's dot product as a tagged packet (oc_exchange.cuh), and every CTA
// applies the scalar rule itself to the same total.
//
// Measured on a 513 x 513 cloth (12 incidences a vertex, 4 iterations): 26 + 13.3 us an iteration
// in two kernels and about 13 us of gaps and graph conditions, now 22 us, 5 of them the
// exchanges.  What is left is the gather, 76 MB of blocks and neighbours a pass: a row is a chain
// of loads that depend on the neighbour's number, so the next incidence's block is requested into
// L1 meanwhile (109 -> 89 us for the launch), a block is one 16-byte and one 8-byte load (before,
// six planes), read evict-first (plain loads 98).  State in the planes instead: 98; 896 threads
// 86, 768 (three rows a thread) 100, two incidences at a time 87.
//
// Progress: all CTAs are co-resident, and a CTA sends its packet before it waits for the
// others'.  A wait gives up after a.barrier_polls polls or when another CTA has given up: it
// sets bit 0 of *err and the CTA leaves without its update.
constexpr int kCT = kCplThreads;

struct CplScalars {  // a cloth's, written by thread 0
    Acc dn, dq, thresh;  // delta_new, the last d.q, eps^2 delta0, each times the piece's scale
    float alpha, beta;
    int it;
    uint32_t fl;
};

__global__ void __launch_bounds__(kCT, 1) k_cpl_persist(const StepArgs a, const CplPlan P) {
    extern __shared__ float sm[];
    __shared__ Acc s_sums[kCT / 32];
    __shared__ float s_scal;
    __shared__ int s_ok, s_run;
    __shared__ CplScalars sc;
    const int tid = threadIdx.x, w = tid >> 5;
    const CplPiece pc = P.pieces[blockIdx.x];
    const int n = pc.n, S = P.smem_rows, in = min(n, S);
    const int64_t v = pc.v;
    const float scale = pc.scale;
    const InstParams& ip = a.inst[pc.inst];
    InstState& is = a.state[pc.inst];
    const uint32_t base = *(volatile uint32_t*)&P.ctl->base;
    uint32_t tag = base;
    float* const sx = sm;
    float* const sr = sm + 3 * S;
    float* const sd = sm + 6 * S;  // dn
    float* const sq = sm + 9 * S;
    float* const sP = sm + 12 * S;
    float* const sM = sm + 18 * S;
    if (tid == 0) {
        sc.dn = pair_from(__ldcg(&is.delta_new) * scale);
        sc.dq = acc_zero();
        sc.thresh = pair_from((double)ip.eps2 * __ldcg(&is.delta0) * scale);
        sc.alpha = sc.beta = 0.0f;
        sc.it = __ldcg(&is.iter);
        sc.fl = __ldcg(&is.flags);
        s_ok = 1;
        s_run = __ldcg(&is.active) != 0;
    }
    for (int i = tid; i < in; i += kCT) {
        const int64_t g = v + i;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sx[k * S + i] = a.x[k][g];
            sr[k * S + i] = a.r[k][g];
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) sP[k * S + i] = a.A[k][g];
        sM[i] = a.cpl_m[g];
    }
    __syncthreads();
    bool first = true;
    while (s_run) {
        if ((int)blockIdx.x == a.withhold_block) {
            if (tid == 0) s_ok = 0;
            __syncthreads();
            break;
        }
        // The direction pass; s_scal holds beta.
        float scal = s_scal;
        Acc part = acc_zero();
        for (int i = tid; i < n; i += kCT) {
            const int64_t g = v + i;
            if (__ldg(a.pinflag + g)) continue;
            const int deg = __ldg(a.rowptr + g + 1) - __ldg(a.rowptr + g);
            const int64_t slot0 = __ldg(a.cpl_slice + (g >> 5)) + (g & 31);
            const float4 zg = a.cpl_z[g];
            float n0 = zg.x, n1 = zg.y, n2 = zg.z;
            if (!first) {
                const float4 dg = a.cpl_d[g];
                n0 = n0 + dg.x * scal;
                n1 = n1 + dg.y * scal;
                n2 = n2 + dg.z * scal;
            }
            const float mp = i < S ? sM[i] : a.cpl_m[g];
            float q0 = mp * n0, q1 = mp * n1, q2 = mp * n2;
            for (int e = 0; e < deg; ++e) {
                const int64_t k = slot0 + 32 * (int64_t)e;
                const float4 nb = __ldcs(a.cpl_nb + k);
                const float2 go = __ldcs(a.cpl_go + k);
                if (e + 1 < deg) {
                    prefetch_l1(a.cpl_nb + k + 32);
                    prefetch_l1(a.cpl_go + k + 32);
                }
                const int32_t o = __float_as_int(go.y);
                const float4 zo = a.cpl_z[o];
                float m0 = zo.x, m1 = zo.y, m2 = zo.z;
                if (!first) {
                    const float4 dd = a.cpl_d[o];
                    m0 = m0 + dd.x * scal;
                    m1 = m1 + dd.y * scal;
                    m2 = m2 + dd.z * scal;
                }
                block_apply(nb.x, nb.y, nb.z, nb.w, go.x, n0 - m0, n1 - m1, n2 - m2, q0, q1, q2);
            }
            if (i < S) {
                sd[i] = n0;
                sd[S + i] = n1;
                sd[2 * S + i] = n2;
                sq[i] = q0;
                sq[S + i] = q1;
                sq[2 * S + i] = q2;
            } else {
                a.q[0][g] = q0;
                a.q[1][g] = q1;
                a.q[2][g] = q2;
            }
            acc_add(part, (n0 * q0 + n1 * q1 + n2 * q2) * scale);
        }
        Acc total = acc_zero();
        ++tag;
        bool ok = pull_sum<kCT / 32>(part, P.packets + (size_t)(tag & 1) * P.n_packets + pc.packet, pc.idx, pc.np, tag,
                                     false, a, P.err, s_sums, total);
        if (w == 0) {
            const bool fin = pair_finite(total), good = total.s > 0.0f && fin;
            const float alpha = good ? quotient(sc.dn, total) : 0.0f;
            if (tid == 0) {
                sc.dq = total;
                if (good) sc.alpha = alpha;
                else sc.fl |= fin ? OC_FLAG_BREAKDOWN : OC_FLAG_NON_FINITE;
                s_scal = alpha;
                s_run = ok && good;
                if (!ok) {
                    atomicOr(P.err, 1);
                    s_ok = 0;
                }
            }
        }
        __syncthreads();
        if (!s_run) break;
        // The update pass; s_scal holds alpha, scal still beta.
        const float al = s_scal;
        part = acc_zero();
        for (int i = tid; i < n; i += kCT) {
            const int64_t g = v + i;
            if (__ldg(a.pinflag + g)) continue;
            float m[3], r[3], Pi[6], z0, z1, z2;
            if (i < S) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    m[k] = sd[k * S + i];
                    sx[k * S + i] = sx[k * S + i] + m[k] * al;
                    r[k] = sr[k * S + i] - sq[k * S + i] * al;
                    sr[k * S + i] = r[k];
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) Pi[k] = sP[k * S + i];
            } else {
                const float4 zg = a.cpl_z[g], dg = a.cpl_d[g];
                const float zv[3] = {zg.x, zg.y, zg.z}, dv[3] = {dg.x, dg.y, dg.z};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    m[k] = zv[k];
                    if (!first) m[k] = m[k] + dv[k] * scal;
                    a.x[k][g] = a.x[k][g] + m[k] * al;
                    r[k] = a.r[k][g] - a.q[k][g] * al;
                    a.r[k][g] = r[k];
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) Pi[k] = a.A[k][g];
            }
            matvec(Pi, r[0], r[1], r[2], z0, z1, z2);
            a.cpl_d[g] = make_float4(m[0], m[1], m[2], 0.0f);
            a.cpl_z[g] = make_float4(z0, z1, z2, 0.0f);
            acc_add(part, (r[0] * z0 + r[1] * z1 + r[2] * z2) * scale);
        }
        ++tag;
        ok = pull_sum<kCT / 32>(part, P.packets + (size_t)(tag & 1) * P.n_packets + pc.packet, pc.idx, pc.np, tag, true,
                                a, P.err, s_sums, total);
        if (w == 0) {
            const bool fin = pair_finite(total);
            const float beta = quotient(total, sc.dn);
            __syncwarp();  // every lane has read sc.dn
            if (tid == 0) {
                const bool above = pair_gt(total, sc.thresh);
                const bool more = ++sc.it < ip.imax && above;
                sc.beta = beta;
                sc.dn = total;
                if (!fin) sc.fl |= OC_FLAG_NON_FINITE;
                else if (!more && above) sc.fl |= OC_FLAG_NOT_CONVERGED;
                s_scal = beta;
                s_run = ok && fin && more;
                if (!ok) {
                    atomicOr(P.err, 1);
                    s_ok = 0;
                }
            }
        }
        __syncthreads();
        first = false;
    }
    if (tid == 0) {
        leave_tags(P.ctl, base, tag - base + 1);
        if (s_ok && pc.idx == 0) {
            const double unit = 1.0f / scale;  // (a power of two)
            is.delta_new = ((double)sc.dn.s + (double)sc.dn.c) * unit;
            is.dq = ((double)sc.dq.s + (double)sc.dq.c) * unit;
            is.alpha = sc.alpha;
            is.beta = sc.beta;
            is.iter = sc.it;
            is.flags = sc.fl;
            is.active = 0;
        }
    }
    if (!s_ok) return;
    for (int i = tid; i < n; i += kCT) {
        const int64_t g = v + i;
        float x[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[k] = i < S ? sx[k * S + i] : a.x[k][g];
            if (i < S) a.x[k][g] = x[k];
        }
        float4 X = a.X[g], V = a.V[g];
        update_vertex(ip, a.dt, x[0], x[1], x[2], X, V);
        a.X[g] = X;
        a.V[g] = V;
    }
}

}  // namespace

cudaError_t prepare_coupled(int device, int* max_rows) {
    int optin = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_cpl_persist);
    if (e != cudaSuccess) return e;
    const int room = optin - (int)fa.sharedSizeBytes;
    *max_rows = room / (int)(kCplRowFloats * sizeof(float)) / 32 * 32;
    return cudaFuncSetAttribute(k_cpl_persist, cudaFuncAttributeMaxDynamicSharedMemorySize, room);
}

cudaError_t launch_cpl_persist(const StepArgs& a, const CplPlan& plan, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)plan.grid);
    cfg.blockDim = dim3(kCT);
    cfg.dynamicSmemBytes = (size_t)plan.smem_rows * kCplRowFloats * sizeof(float);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_cpl_persist, a, plan);
}

const void* coupled_fn(KernelKind k) {
    switch (k) {
        case K_CPL_ASSEMBLE: return (const void*)k_cpl_assemble;
        case K_CPL_DIR: return (const void*)k_cpl_dir;
        case K_CPL_UPDATE: return (const void*)k_cpl_update;
        default: return nullptr;
    }
}

cudaError_t launch_coupled(KernelKind k, const StepArgs& a, int nblocks, cudaStream_t stream) {
    if (nblocks <= 0) return cudaSuccess;
    switch (k) {
        case K_CPL_ASSEMBLE: k_cpl_assemble<<<nblocks, kThreads, 0, stream>>>(a); break;
        case K_CPL_DIR: k_cpl_dir<<<nblocks, kThreads, 0, stream>>>(a); break;
        case K_CPL_UPDATE: k_cpl_update<<<nblocks, kThreads, 0, stream>>>(a); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace oc
