// k_sim: whole steps of small REFERENCE cloths, any number of steps in one launch: the forces,
// spring i's Jacobians, the assembly, the CG and the update (IMP:698-798), then EllipsoidCollision
// and ApplyProvotDynamicInverse (IMP:800-848) where a cloth has them.
//
// One cluster of up to 16 CTAs of 256 threads per cloth; a thread owns VPT vertices.  Every
// vertex's system and CG state live in registers (with VPT > 1 they pass through shared memory
// between the assembly's loop and the CG's), the warm start across steps too, and the CTA's
// window of positions and velocities (its own vertices and, of a grid cloth, those on either side
// that its stencil reaches: 2 cols in the reference's order) in shared memory: a step reads global memory only for
// the window's halo, which the neighbouring CTAs wrote at the end of the step before, and for the
// springs' constants, which stay in L1.  Neighbours outside the window (a general mesh on more
// than one CTA) are read through L2.
//
// A step of a small cloth is bound by latencies, not by bytes: before, it was three graph nodes
// (a memset, the assembly with its last-block epilogue, the resident CG) whose gaps alone cost
// 4 us, the assembly's twelve incidences were six rounds of dependent L2 loads (11.5 us for 441
// vertices), and delta0 cost a grid-wide ticket.  Here delta0 travels with the first d.(A d), the
// incidences are shared-memory loads, and the dot products are exchanged as tagged packets
// (oc_exchange.cuh), one barrier an exchange.  Measured per step: 21 x 21 cloth, two iterations,
// 22.7 -> 7.7 us; 100 x 75, four iterations, 33 -> 15.4 us.  What is left is the instructions of a
// thread's own vertex (about 900 for its springs, 400 for spring i and the system, at 4 to 5 cycles
// each with two to four warps a scheduler) and 1,500 to 2,200 cycles an exchange.  256 vertices
// on 256 threads measured 5% better than 512 on 512 for the small cloth and level for the other.
// With 512 cloths (3 M vertices) it took 1.65 ms for what the separate launches do in 0.99: the
// plan takes it only while all CTAs fit on the SMs at once (plan_sim).
//
// The arithmetic is the streamed executor's expression for expression (--fmad=false); sums run in
// float pairs in a fixed order, as in oc_persist.cu.
#include <cuda_runtime.h>

#include <algorithm>

#include "oc_device.cuh"
#include "oc_exchange.cuh"
#include "oc_internal.h"

namespace oc {
namespace {

constexpr int kStage = 15;  // A, r, d, x of a vertex staged in shared memory when VPT > 1

// One vertex's incidences from the window: B of them fetched ahead of their forces, added in
// spring-id order (stencil_gather's and thread_gather's arithmetic and order).
struct Window {
    const float4* X;
    const float4* V;
    int lo;       // its first vertex (of the cloth)
    unsigned n;   // its vertices
};

__device__ __forceinline__ void window_at(const StepArgs& a, const InstParams& ip, const Window& w, int l, float4& X,
                                          float4& V) {
    const unsigned i = (unsigned)(l - w.lo);
    if (i < w.n) {
        X = w.X[i];
        V = w.V[i];
    } else {
        X = __ldcg(a.X + ip.v_off + l);
        V = __ldcg(a.V + ip.v_off + l);
    }
}

// A grid cloth's stencil in shared memory: the first entry of each class, and per entry the
// neighbour's offset, the side and the parameters.  The window's halo is the stencil's own reach, so
// its neighbours are indexed without a test.
struct Stencil {
    const int32_t* first;  // kStencilClasses + 1
    const float4* entry;   // {offset << 1 | is_p2, rest, ks, kd}
};

template <int B>
__device__ __forceinline__ float3 window_forces(const StepArgs& a, const InstParams& ip, const Window& w,
                                                const Stencil& st, int l, int cls, const float* rest_of, int stride,
                                                const float4 Xg, const float4 Vg) {
    const int64_t g = ip.v_off + l;
    float3 F = base_force(a, ip, g, Xg, Vg);
    if (Vg.w != 0.0f) return F;  // pinned vertices take no spring force (IMP:730-733)
    if (ip.grid_cols > 0) {
        const int32_t e0 = st.first[cls], n = st.first[cls + 1] - e0;
        const float4* ent = st.entry + e0;
        const float4 *wX = w.X + (l - w.lo), *wV = w.V + (l - w.lo);
        for (int32_t e = 0; e < n; e += B) {
            float4 Xo[B], Vo[B];
            float rest[B], ks[B], kd[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const float4 p = e + u < n ? ent[e + u] : make_float4(0.f, 0.f, 0.f, 0.f);  // past the end: itself
                const int o = __float_as_int(p.x) >> 1;
                rest[u] = rest_of && e + u < n ? rest_of[(e + u) * stride] : p.y;
                ks[u] = p.z;
                kd[u] = p.w;
                Xo[u] = wX[o];
                Vo[u] = wV[o];
            }
            add_spring_forces<B>(F, Xg, Vg, Xo, Vo, rest, ks, kd, n - e);
        }
    } else {
        const int32_t k0 = __ldg(a.rowptr + g), k1 = __ldg(a.rowptr + g + 1);
        for (int32_t k = k0; k < k1; k += B) {
            float4 Xo[B], Vo[B];
            float rest[B], ks[B], kd[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int4 rec = k + u < k1 ? __ldg(a.inc + k + u) : make_int4((int)g, 0, 0, 0);
                rest[u] = __int_as_float(rec.y);
                ks[u] = __int_as_float(rec.z);
                kd[u] = __int_as_float(rec.w);
                window_at(a, ip, w, (int)((rec.x & 0x7fffffff) - ip.v_off), Xo[u], Vo[u]);
            }
            add_spring_forces<B>(F, Xg, Vg, Xo, Vo, rest, ks, kd, k1 - k);
        }
    }
    return F;
}

// ApplyProvotDynamicInverse for one vertex, its incidences in spring order (k_provot).
__device__ __forceinline__ void window_provot(const StepArgs& a, const InstParams& ip, const Window& w,
                                              const Stencil& st, int l, int cls, int32_t k0, const float4 Xg,
                                              float4& Vg) {
    const int64_t g = ip.v_off + l;
    const bool pin_self = a.pinflag[g] != 0;
    if (ip.grid_cols > 0) {
        const int32_t e0 = st.first[cls], n = st.first[cls + 1] - e0;
        for (int32_t e = 0; e < n; ++e) {
            const float4 p = st.entry[e0 + e];
            const int o = l + (__float_as_int(p.x) >> 1);
            const float rest = ip.st_rest ? __ldg(a.rest_inc + k0 + e) : p.y;
            provot_pair(a, ip.provot_ratio, Xg, w.X[o - w.lo], pin_self, ip.v_off + o, (__float_as_int(p.x) & 1) != 0,
                        rest, Vg);
        }
    } else {
        const int32_t k1 = __ldg(a.rowptr + g + 1);
        for (int32_t k = k0; k < k1; ++k) {
            const int4 rec = __ldg(a.inc + k);
            const int64_t o = rec.x & 0x7fffffff;
            const unsigned i = (unsigned)((int)(o - ip.v_off) - w.lo);
            provot_pair(a, ip.provot_ratio, Xg, i < w.n ? w.X[i] : __ldcg(a.X + o), pin_self, o, rec.x < 0,
                        __int_as_float(rec.y), Vg);
        }
    }
}

template <int kST, int VPT>
__global__ void __launch_bounds__(kST, 1) k_sim(const StepArgs a, const SimLaunch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kSW = kST / 32, kCap = kST * VPT;
    // Packets by parity and value: of the CTA's warps (or of all warps of a cluster of up to
    // kDirect CTAs, by rank and warp), and of the CTAs of a larger cluster.
    constexpr int kDirect = 32 / kSW;
    __shared__ __align__(16) ulonglong2 s_box[2][2][32], s_cbox[2][2][kSimMaxCluster];
    __shared__ float s_scal;
    __shared__ int s_run, s_ok;
    __shared__ int s_gone[2];  // a CTA of the cluster gave up, by the parity of the barriers inside the steps
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int C = L.cluster, rank = (int)blockIdx.x % C;
    const int inst = L.inst_ids[blockIdx.x / C];
    const InstParams& ip = a.inst[inst];
    const int nv = ip.nv, chunk = (nv + C - 1) / C;
    const int lb = rank * chunk, n = max(0, min(nv, lb + chunk) - lb);
    const int halo = ip.grid_cols > 0 ? ip.st_reach : 0;
    const int wlo = max(0, lb - halo), whi = n > 0 ? min(nv, lb + n + halo) : wlo;
    float4* const wX = reinterpret_cast<float4*>(smem_raw);
    float4* const wV = wX + L.window;
    float4* const s_ent = wV + L.window;
    float* const s_st = reinterpret_cast<float*>(s_ent + L.entries);  // staging planes of kCap floats
    float* const s_rest = s_st + (VPT > 1 ? kStage * kCap : 0);       // rest lengths by entry, L.rest planes
    __shared__ int32_t s_first[kStencilClasses + 1];
    const Window win{wX, wV, wlo, (unsigned)(whi - wlo)};
    const Stencil sten{s_first, s_ent};
    const int64_t vo = ip.v_off;

    if (tid == 0) {
        s_ok = 1;
        s_gone[0] = s_gone[1] = 0;
    }
    if (tid < 2 * 2 * 32) (&s_box[0][0][0])[tid] = make_ulonglong2(0, 0);
    if (tid < 2 * 2 * kSimMaxCluster) (&s_cbox[0][0][0])[tid] = make_ulonglong2(0, 0);
    if (C > 1) cluster_arrive();  // every CTA's boxes are clear before a packet is sent
    for (int i = wlo + tid; i < whi; i += kST) {
        wX[i - wlo] = a.X[vo + i];
        wV[i - wlo] = a.V[vo + i];
    }
    if (ip.grid_cols > 0) {
        const int32_t* st = a.st_data + ip.st_off;
        for (int i = tid; i <= kStencilClasses; i += kST) s_first[i] = __ldg(st + i) - (kStencilClasses + 1);
        const int m = __ldg(st + kStencilClasses);
        for (int i = kStencilClasses + 1 + tid; i < m; i += kST) {
            const int32_t v = __ldg(st + i);
            const int off = ((v & 7) - 2) * ip.grid_cols + (((v >> 3) & 7) - 2);
            const float4 p = __ldg(a.st_param + ip.st_par + (v >> 7));
            s_ent[i - (kStencilClasses + 1)] = make_float4(__int_as_float(off * 2 | (v >> 6 & 1)), p.x, p.y, p.z);
        }
    }
    // A vertex's class.
    auto class_of = [&](int l) {
        if (ip.grid_cols <= 0) return 0;
        const int row = l / ip.grid_cols, col = l - row * ip.grid_cols;
        return stencil_class_1d(row, ip.grid_rows) * 6 + stencil_class_1d(col, ip.grid_cols);
    };
    const bool rest_planes = ip.grid_cols > 0 && ip.st_rest;
    if (rest_planes) {
        __syncthreads();
        for (int j = tid; j < n; j += kST) {
            const int cls = class_of(lb + j), m = s_first[cls + 1] - s_first[cls];
            const float* src = a.rest_inc + __ldg(a.rowptr + vo + lb + j);
            for (int e = 0; e < m; ++e) s_rest[e * kCap + j] = __ldg(src + e);
        }
    }
    float A[VPT][6], r[VPT][3], d[VPT][3], x[VPT][3];
    bool own[VPT];
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
        const int j = tid + u * kST;
        own[u] = j < n;
#pragma unroll
        for (int k = 0; k < 6; ++k) A[u][k] = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            r[u][k] = d[u][k] = 0.0f;
            x[u][k] = own[u] ? a.x[k][vo + lb + j] : 0.0f;
            if constexpr (VPT > 1) s_st[(12 + k) * kCap + j] = x[u][k];
        }
    }
    // Warp 0's scalars (every lane).
    Acc dn = acc_zero(), dn0 = acc_zero(), thresh = acc_zero();  // delta_new, delta0, eps^2 delta0
    int it = 0;
    uint32_t fl = 0u;
    const int imax = ip.imax;
    const float eps2 = ip.eps2;
    unsigned tag = 0;

    // The partial sums of a thread's p (and p2) sent off by every warp, and their totals over the
    // cluster, in every lane of warp 0; receive is false when the wait gave up.  With at most 32
    // warps in the cluster the warps' packets go to every CTA; in a larger one warp 0 sums its
    // CTA's first.
    auto send = [&](Acc p, int value) {
        p = lanes_sum<16>(p);
        if (C > kDirect || C == 1) {
            if (lane == 0) put_local(&s_box[tag & 1][value][w], p, tag);
        } else if (lane < C) {
            put_cluster(&s_box[tag & 1][value][rank * kSW + w], lane, p, tag);
        }
    };
    auto send2 = [&](Acc p, Acc p2) {  // two values, their lane sums interleaved
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const Acc u = make_acc(__shfl_xor_sync(0xffffffffu, p.s, o), __shfl_xor_sync(0xffffffffu, p.c, o));
            const Acc u2 = make_acc(__shfl_xor_sync(0xffffffffu, p2.s, o), __shfl_xor_sync(0xffffffffu, p2.c, o));
            p = acc_merge(p, u);
            p2 = acc_merge(p2, u2);
        }
        if (C > kDirect || C == 1) {
            if (lane < 2) put_local(&s_box[tag & 1][lane][w], lane == 0 ? p : p2, tag);
        } else if (lane < C) {
            put_cluster(&s_box[tag & 1][0][rank * kSW + w], lane, p, tag);
            put_cluster(&s_box[tag & 1][1][rank * kSW + w], lane, p2, tag);
        }
    };
    const bool mine = lane < (C > kDirect ? kSW : C * kSW);
    auto receive = [&](int value, Acc& total) -> bool {
        Acc t = acc_zero();
        const ulonglong2* box = &s_box[tag & 1][value][lane];
        bool ok = poll<1>(mine ? 1u : 0u, a, L.err, [&](int) { return get_cluster(box, tag, t); });
        if (!ok) {
            // Nothing of this exchange may be decided before the CTA's other warps, which have read the
            // last one's decision when they send, have sent (they wait for nothing on the way).
            const int from = C > kDirect ? 0 : rank * kSW;
            const bool theirs = lane >= from && lane < from + kSW;
            for (unsigned i = 0; i < 1u << 22; ++i)
                if (__all_sync(0xffffffffu, !theirs || get_cluster(box, tag, t))) break;
        }
        if (!mine) t = acc_zero();
        total = lanes_sum<16>(t);
        if (C > kDirect && ok) {
            if (lane < C) put_cluster(&s_cbox[tag & 1][value][rank], lane, total, tag);
            t = acc_zero();
            const ulonglong2* cbox = &s_cbox[tag & 1][value][lane % kSimMaxCluster];
            ok = poll<1>(lane < C ? 1u : 0u, a, L.err, [&](int) { return get_cluster(cbox, tag, t); });
            if (lane >= C) t = acc_zero();
            total = lanes_sum<16>(t);
        }
        total = pair_norm(total);
        return ok;
    };
    auto decide = [&](bool ok, bool run, float scal) {  // by warp 0, for the CTA
        if (lane == 0) {
            s_scal = scal;
            s_run = run && ok ? 1 : 0;
            if (!ok) {
                s_ok = 0;
                atomicOr(L.err, 1);
            }
        }
    };
    // After d.(A d): alpha, or a breakdown.
    auto alpha_rule = [&](bool ok, const Acc& dq) {
        bool run = true;
        float scal = 0.0f;
        const bool fin = pair_finite(dq);
        if (!(dq.s > 0.0f) || !fin) {
            fl |= fin ? OC_FLAG_BREAKDOWN : OC_FLAG_NON_FINITE;
            run = false;
        } else {
            scal = quotient(dn, dq);
        }
        decide(ok, run, scal);
    };

    // The cluster's barrier inside a step: true when no CTA's wait has given up.  One whose has takes the
    // barrier like the others, having told them first, and all of them leave behind the same barrier: a
    // CTA that left alone would be missing at the others' next barrier, and their packets would go to
    // shared memory that is no longer its own.  Two flags, by the parity of these barriers, as a CTA may be
    // one barrier ahead of another that has not read its flag yet, but not two.
    auto together = [&](int parity) -> bool {
        int* const gone = &s_gone[parity];
        if (!s_ok && tid < C) flag_cluster(gone, tid);
        cluster_arrive();
        cluster_wait();
        return *(volatile int*)gone == 0;
    };
    const int n_steps = L.n_steps;
    int step = 0;

    __syncthreads();
    if (C > 1) cluster_wait();
    if ((int)blockIdx.x == a.withhold_block) {  // (a testing aid) sends no packets, meets the others at their first barrier
        if (tid == 0) s_ok = 0;
        __syncthreads();
        if (C > 1 && (n_steps > 1 || (ip.passes & OC_PASS_PROVOT))) together(0);
        step = n_steps;
    }
    for (; step < n_steps; ++step) {
        // The assembly of the CTA's vertices, with the first direction's dot product.
        Acc p0 = acc_zero(), p1 = acc_zero();
#pragma unroll 1
        for (int u = 0; u < VPT; ++u) {
            const int j = tid + u * kST;
            if (j >= n) break;
            const int l = lb + j;
            const int64_t g = vo + l;
            const float4 Xg = wX[l - wlo], Vg = wV[l - wlo];
            OwnSpring os;
            os.ends = __ldg(a.own_ends + g);
            os.par = make_float4(0.f, 0.f, 0.f, 0.f);
            os.E1 = os.E2 = os.W1 = os.W2 = make_float4(0.f, 0.f, 0.f, 0.f);
            const float3 F = window_forces<4>(a, ip, win, sten, l, class_of(l), rest_planes ? s_rest + j : nullptr, kCap,
                                              Xg, Vg);
            if (os.ends.x >= 0) {
                os.par = __ldg(a.own_par + g);
                window_at(a, ip, win, (int)(os.ends.x - vo), os.E1, os.W1);
                window_at(a, ip, win, (int)(os.ends.y - vo), os.E2, os.W2);
            }
            const VertexSystem sys = vertex_system(a.dt, Xg, Vg, F, os);
            float x0, x1, x2;
            if constexpr (VPT == 1) {
                x0 = x[0][0];
                x1 = x[0][1];
                x2 = x[0][2];
            } else {
                x0 = s_st[12 * kCap + j];
                x1 = s_st[13 * kCap + j];
                x2 = s_st[14 * kCap + j];
            }
            const CgInit c = cg_init(sys, x0, x1, x2, Vg.w != 0.0f);
            acc_add(p0, c.term);
            float q0, q1, q2;
            matvec(sys.A, c.d[0], c.d[1], c.d[2], q0, q1, q2);
            acc_add(p1, c.d[0] * q0 + c.d[1] * q1 + c.d[2] * q2);
            if constexpr (VPT == 1) {
#pragma unroll
                for (int k = 0; k < 6; ++k) A[0][k] = sys.A[k];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    r[0][k] = c.r[k];
                    d[0][k] = c.d[k];
                    x[0][k] = c.x[k];
                }
            } else {
#pragma unroll
                for (int k = 0; k < 6; ++k) s_st[k * kCap + j] = sys.A[k];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    s_st[(6 + k) * kCap + j] = c.r[k];
                    s_st[(9 + k) * kCap + j] = c.d[k];
                    s_st[(12 + k) * kCap + j] = c.x[k];
                }
            }
        }
        ++tag;
        send2(p0, p1);
        if constexpr (VPT > 1) {
#pragma unroll
            for (int u = 0; u < VPT; ++u)
                if (own[u]) {
                    const float* p = s_st + tid + u * kST;
#pragma unroll
                    for (int k = 0; k < 6; ++k) A[u][k] = p[k * kCap];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        r[u][k] = p[(6 + k) * kCap];
                        d[u][k] = p[(9 + k) * kCap];
                        x[u][k] = p[(12 + k) * kCap];
                    }
                }
        }
        if (w == 0) {
            Acc dq;
            bool ok = receive(0, dn);
            ok = receive(1, dq) && ok;
            // delta0 and the decision to iterate, as the assembly's epilogue takes them.
            // eps^2 delta0 as a pair: the head product exactly, as an FMA gives its error.
            dn0 = dn;
            const float th = __fmul_rn(eps2, dn.s);
            thresh = pair_norm(make_acc(th, __fmaf_rn(eps2, dn.s, -th) + __fmul_rn(eps2, dn.c)));
            it = 0;
            fl = pair_finite(dn) ? 0u : OC_FLAG_NON_FINITE;
            if (pair_finite(dn) && 0 < imax && pair_gt(dn, thresh))
                alpha_rule(ok, dq);
            else
                decide(ok, false, 0.0f);
        }
        __syncthreads();
        while (s_run) {
            // x += alpha d; r -= alpha A d; r.r, IMP:322-325.
            const float alpha = s_scal;
            Acc part = acc_zero();
#pragma unroll
            for (int u = 0; u < VPT; ++u) res_vertex(A[u], r[u], d[u], alpha, 1.0f, part);
            ++tag;
            send(part, 0);
#pragma unroll
            for (int u = 0; u < VPT; ++u)
#pragma unroll
                for (int k = 0; k < 3; ++k) x[u][k] = x[u][k] + d[u][k] * alpha;
            if (w == 0) {
                Acc rr;
                const bool ok = receive(0, rr);
                const bool fin = pair_finite(rr), above = pair_gt(rr, thresh);
                bool run = true;
                const float beta = quotient(rr, dn);
                dn = rr;
                ++it;
                if (!fin) {
                    fl |= OC_FLAG_NON_FINITE;
                    run = false;
                } else if (!(it < imax && above)) {
                    if (above) fl |= OC_FLAG_NOT_CONVERGED;
                    run = false;
                }
                decide(ok, run, beta);
            }
            __syncthreads();
            if (!s_run) break;
            // d = r + beta d; d.(A d), IMP:320-321, 327.
            const float beta = s_scal;
            part = acc_zero();
#pragma unroll
            for (int u = 0; u < VPT; ++u) dir_vertex(A[u], r[u], d[u], false, beta, 1.0f, part);
            ++tag;
            send(part, 0);
            if (w == 0) {
                Acc dq;
                const bool ok = receive(0, dq);
                alpha_rule(ok, dq);
            }
            __syncthreads();
        }
        // A wait that gave up: no update; the CTAs of a cluster go on to their next barrier.
        if (C == 1 && !s_ok) break;
        // The update (IMP:790-797) and the ellipsoid; the window's own part, and, for the other
        // CTAs and at the end, global memory.
        const bool last = step + 1 == n_steps;
        const bool prov = (ip.passes & OC_PASS_PROVOT) != 0;
#pragma unroll
        for (int u = 0; u < VPT; ++u)
            if (own[u] && s_ok) {
                const int j = tid + u * kST, i = lb + j - wlo;
                float4 X = wX[i], V = wV[i];
                update_vertex(ip, a.dt, x[u][0], x[u][1], x[u][2], X, V);
                wX[i] = X;
                wV[i] = V;
                if (C > 1 || last) {
                    a.X[vo + lb + j] = X;
                    if (!prov) a.V[vo + lb + j] = V;
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if constexpr (VPT > 1) s_st[(12 + k) * kCap + j] = x[u][k];
                    if (last) a.x[k][vo + lb + j] = x[u][k];
                }
            }
        if (prov) {
            if (C > 1) {
                if (!together(0)) break;
                for (int i = wlo + tid; i < whi; i += kST)
                    if (i < lb || i >= lb + n) wX[i - wlo] = __ldcg(a.X + vo + i);
            }
            __syncthreads();
#pragma unroll 1
            for (int u = 0; u < VPT; ++u) {
                const int j = tid + u * kST;
                if (j >= n) break;
                const int l = lb + j;
                float4 V = wV[l - wlo];
                window_provot(a, ip, win, sten, l, class_of(l), __ldg(a.rowptr + vo + l), wX[l - wlo], V);
                wV[l - wlo] = V;
                if (C > 1 || last) a.V[vo + l] = V;
            }
        }
        if (!last) {
            if (C > 1) {  // the neighbouring CTAs' new state into the halo
                if (!together(prov ? 1 : step & 1)) break;
                for (int i = wlo + tid; i < whi; i += kST)
                    if (i < lb || i >= lb + n) {
                        if (!prov) wX[i - wlo] = __ldcg(a.X + vo + i);
                        wV[i - wlo] = __ldcg(a.V + vo + i);
                    }
            }
            __syncthreads();
        }
    }
    if (rank == 0 && tid == 0 && s_ok && step == n_steps) {
        InstState& st = a.state[inst];
        st.delta0 = (double)dn0.s + (double)dn0.c;
        st.delta_new = (double)dn.s + (double)dn.c;
        st.dq = 0.0;
        st.iter = it;
        st.flags = fl;
        st.active = 0;
        st.ticket = 0;
        st.alpha = st.beta = 0.0f;
    }
    // A CTA's shared memory must outlive the packets sent to it.
    if (C > 1) {
        cluster_arrive();
        cluster_wait();
    }
}

typedef void (*SimFn)(StepArgs, SimLaunch);
SimFn sim_fn(int threads, int vpt) {
    if (threads == 256) return k_sim<256, 1>;
    return vpt == 1 ? k_sim<512, 1> : k_sim<512, 2>;
}
constexpr int kShapes[][2] = {{256, 1}, {512, 1}, {512, 2}};

}  // namespace

size_t sim_smem_bytes(const SimLaunch& L) {
    const size_t cap = (size_t)L.threads * L.vpt;
    return ((size_t)2 * L.window + L.entries) * sizeof(float4) +
           ((L.vpt > 1 ? kStage : 0) + (size_t)L.rest) * cap * sizeof(float);
}

cudaError_t prepare_sim(int device, int* max_smem) {
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    *max_smem = optin;
    for (const auto& sh : kShapes) {
        const SimFn fn = sim_fn(sh[0], sh[1]);
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
        if (e != cudaSuccess) return e;
        const int room = optin - (int)fa.sharedSizeBytes;
        *max_smem = std::min(*max_smem, room);
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, room);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    return e;
}

cudaError_t sim_max_clusters(const SimLaunch& L, int* n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.cluster);
    cfg.blockDim = dim3((unsigned)L.threads);
    cfg.dynamicSmemBytes = sim_smem_bytes(L);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)L.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(n, sim_fn(L.threads, L.vpt), &cfg);
}

cudaError_t launch_sim(const StepArgs& a, const SimLaunch& L, int n_clusters, cudaStream_t stream) {
    if (n_clusters <= 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_clusters * L.cluster));
    cfg.blockDim = dim3((unsigned)L.threads);
    cfg.dynamicSmemBytes = sim_smem_bytes(L);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)L.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = L.cluster > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, sim_fn(L.threads, L.vpt), a, L);
}

}  // namespace oc
