// k_cg_persist: the whole CG loop of the streamed REFERENCE cloths (IMP:308-330), any number
// of them, and their update (IMP:790-797), in one cooperative launch of at most one CTA per SM.
//
// The system is block-diagonal, so the only thing a CTA needs of the others in an iteration
// is the two dot products.  Each CTA therefore keeps its vertices' A, r and d (48 bytes a
// vertex) on chip for the whole loop: the first kRegSlots vertices of every thread in
// registers, the next ones in shared memory, and only what is left over (cloths beyond about
// a million vertices) in the planes in L2.  x is read and written in L2, while the dot
// product of the update pass travels.
//
// The concatenated vertices of the streamed cloths are cut into one contiguous range per CTA.
// The part of a cloth that lies in a CTA's range is a piece; a piece is cut into slots of
// kPersistThreads vertices, one vertex per thread.  Phase q of a cloth is the direction pass
// (q even) or the update pass (q odd) of iteration q / 2.  At the end of a phase the CTAs of a
// cloth exchange their partial sums and every one of them applies the scalar rule itself to
// the same total, so all take identical decisions.
//
// The exchange.  A partial travels as a packet of two 8-byte words, each a float of the pair
// and the phase's tag: the data is its own flag, so a hop is a store and the polls that see
// it, without a fence, an atomic or a counter.  Among CTAs of one cluster packets go through
// distributed shared memory; between clusters (CTAs, with clusters of one) through L2, where
// one CTA of a cluster writes a copy for every rank and rank r polls copy r.  Measured on GB300
// (a cooperative probe of 512-thread CTAs, with the block's sum and the quotient): 1,400
// cycles among 16 CTAs of a cluster, 3,300 over 7 clusters of 16, 5,100 to 5,900 over 152 CTAs
// without clusters, 6,600 with FP64 sums and quotient instead of float pairs.  So the plan takes
// clusters of 16 where their CTAs (a cluster needs 16 free SMs of one GPC, so only 7 fit) hold
// all the vertices on chip, and every SM without clusters for larger cloths.
// Packets are double buffered by the phase's parity: a CTA writes phase q + 1's only after it
// has read all of phase q's, which its cloths' CTAs write after reading all of phase q - 1's.
// Tags run on from launch to launch (PersistCtl::base; the last CTA to leave moves it past the
// tags that were used), so the packets in memory are never cleared between launches.  They wrap after
// 2^32, some hours of stepping: a launch's own boxes therefore start with the tag `base`, the one
// that none of its phases has, and not with a fixed one.
//
// Measured (time of the launch, a wave of arrival counts over memory-resident planes before):
// 257 x 257 cloth, 4 iterations, 51 -> 20 us; 120,000-vertex mesh, 22 iterations, 317 -> 92 us;
// 385 x 385, 66 -> 29 us; 1025 x 1025, 105 -> 80 us, which moves 63 MB in and 80 MB out at about
// 5.8 TB/s (25 us) and whose phases are 5,000 cycles of arithmetic and 6,000 of exchange and x.
//
// Progress: a CTA waits in phase q only for cloths that it still runs, whose CTAs publish their
// phase-q packets before their phase-q waits, and all CTAs are co-resident.  A wait gives up
// after a.barrier_polls polls or when another CTA has given up: it sets bit 0 of *err and the
// CTA leaves without its update.  The CTA a.withhold_block (a testing aid; normally -1) leaves
// before its first packets, so the waits on its cloths run out.  The CTAs of a cluster leave
// together, so no packet meets the shared memory of a CTA that has gone.  Whether a wait has given
// up is kept by the phase's parity, like the scalars: the warp that gives up in one phase need not wait
// for the others, which may have yet to read what the phase before decided.
//
// Compiled with --fmad=false; the dot terms are FP32, summed in error-free pairs at every
// level (about 48 bits, as the resident kernel's), in a fixed order; alpha and beta are the
// pairs' quotients rounded to float, which are the two-kernel loop's bits (its sums above a
// warp are FP64) unless a quotient lies within about 2^-46 of a rounding boundary.
#include <cuda_runtime.h>

#include <algorithm>

#include "oc_device.cuh"
#include "oc_exchange.cuh"
#include "oc_internal.h"

namespace oc {
namespace {

constexpr int kPT = kPersistThreads;
constexpr int kWarps = kPT / 32;
constexpr int kRegSlots = 12;     // of k_cg_persist
constexpr int kOneRegSlots = 15;  // of k_cg_persist_one when not FULL
constexpr int kFullSlots = 7;  // the largest piece held in registers with x, X and V
constexpr int kSlotFloats = 12;  // A, r, d of a slot in shared memory
constexpr int kMaxCluster = kPersistMaxCluster;

// Whether the launch has the plan's clusters: without them a packet would go to a CTA that does not
// exist, which is a fault, so a launch that lost them (a tool's own replay) sets the error word instead.
__device__ __forceinline__ bool clusters_as_planned(const PersistPlan& P) {
    uint32_t n;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    if (n == (uint32_t)P.cluster) return true;
    if (threadIdx.x == 0) atomicOr(P.err, 1);
    return false;
}

// Shared memory of a piece: its warps' packets by parity (a piece that shares no cluster with
// another CTA), and the scalars of its cloth.
struct PieceState {
    ulonglong2 box[2][kWarps];
    Acc dn, thresh;  // delta_new, eps^2 delta0, each times the piece's scale
    Acc dq;          // the last d.(A d), likewise
    double d0;
    float scal[2];   // beta or alpha of the phase of that parity
    float alpha, beta;
    int32_t run[2];  // whether the cloth runs in the phase of that parity
    int32_t it, imax;
    uint32_t fl;
    int32_t pad_;
};
static_assert(sizeof(PieceState) == kPersistPieceBytes, "persist_state_bytes");

// The update (IMP:790-797) of a piece's slots [b, e), four vertices of a thread in flight; x out
// of shared memory where it was kept there.
__device__ __forceinline__ void persist_update(const StepArgs& a, const InstParams& ip, int64_t v, int n, int b, int e,
                                               int x_slots, const float* sx) {
    for (int s0 = b; s0 < e; s0 += 4) {
        float4 X[4], V[4];
        float x[4][3];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int s = s0 + u;
            const int64_t g = v + (s - b) * kPT;
            ok[u] = s < e && (s - b) * kPT + (int)threadIdx.x < n;
            if (ok[u]) {
                if (!a.cg_only) {
                    X[u] = a.X[g];
                    V[u] = a.V[g];
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) x[u][k] = s < x_slots ? sx[(s * 3 + k) * kPT] : a.x[k][g];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (!ok[u]) continue;
            const int64_t g = v + (s0 + u - b) * kPT;
            if (s0 + u < x_slots) {
#pragma unroll
                for (int k = 0; k < 3; ++k) a.x[k][g] = x[u][k];
            }
            if (a.cg_only) continue;
            update_vertex(ip, a.dt, x[u][0], x[u][1], x[u][2], X[u], V[u]);
            a.X[g] = X[u];
            a.V[g] = V[u];
        }
    }
}

__global__ void __launch_bounds__(kPT, 1) k_cg_persist(const StepArgs a, const PersistPlan P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_ok[2];  // 0: a wait gave up in the phase before the one of that parity
    // Packets of the warps of the cluster's CTAs, for the CTA's first and last piece (no other
    // piece has vertices in another CTA): by parity, piece, and sender's rank and warp.
    __shared__ __align__(16) ulonglong2 s_box[2][2][kMaxCluster * kWarps];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int CS = P.cluster, rank = (int)blockIdx.x % CS;
    if (!clusters_as_planned(P)) return;
    const int pc0 = P.cta_piece[blockIdx.x], np = P.cta_piece[blockIdx.x + 1] - pc0;
    const PersistPiece* __restrict__ pieces = P.pieces + pc0;
    PieceState* const st = reinterpret_cast<PieceState*>(smem_raw);
    float* const sm = reinterpret_cast<float*>(smem_raw + persist_state_bytes(P.max_pieces)) + tid;
    float* const sx = sm + (size_t)P.smem_slots * kSlotFloats * kPT;  // x of the first P.x_slots slots
    const int s_end = kRegSlots + P.smem_slots;                       // slots from here on stay in the planes
    const uint32_t base = *(volatile uint32_t*)&P.ctl->base;

    if (tid < 2) s_ok[tid] = 1;
    const ulonglong2 none = empty_packet(base);
    for (int i = tid; i < 2 * 2 * kMaxCluster * kWarps; i += kPT) (&s_box[0][0][0])[i] = none;
    for (int j = tid; j < np; j += kPT) {
        const InstState& is = a.state[pieces[j].inst];
        const InstParams& ip = a.inst[pieces[j].inst];
        const double d0 = __ldcg(&is.delta0);
#pragma unroll
        for (int i = 0; i < kWarps; ++i) st[j].box[0][i] = st[j].box[1][i] = none;
        st[j].d0 = d0;
        st[j].dn = pair_from(__ldcg(&is.delta_new) * pieces[j].scale);
        st[j].thresh = pair_from((double)ip.eps2 * d0 * pieces[j].scale);
        st[j].dq = acc_zero();
        st[j].alpha = st[j].beta = 0.0f;
        st[j].it = __ldcg(&is.iter);
        st[j].fl = __ldcg(&is.flags);
        st[j].imax = ip.imax;
        st[j].run[0] = __ldcg(&is.active) ? 1 : 0;
        st[j].scal[0] = 0.0f;
    }
    // Every CTA's boxes are clear before a packet is sent (waited for before the first phase).
    if (CS > 1) cluster_arrive();
    // The CG state the assembly left in the planes: into shared memory by asynchronous copies
    // (all of a thread's in flight together), and into registers.
    float A[kRegSlots][6], r[kRegSlots][3], d[kRegSlots][3];
#pragma unroll
    for (int u = 0; u < kRegSlots; ++u) {
#pragma unroll
        for (int k = 0; k < 6; ++k) A[u][k] = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) r[u][k] = d[u][k] = 0.0f;
    }
    for (int j = 0; j < np; ++j) {
        const int b = pieces[j].slot0, e = pieces[j].slot1, n = pieces[j].n;
        const int64_t v = pieces[j].v + tid;
        for (int s = max(b, kRegSlots); s < min(e, s_end); ++s) {
            if ((s - b) * kPT + tid >= n) break;
            float* p = sm + (s - kRegSlots) * kSlotFloats * kPT;
            const int64_t g = v + (s - b) * kPT;
#pragma unroll
            for (int k = 0; k < 6; ++k) copy_async4(p + k * kPT, a.A[k] + g);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                copy_async4(p + (6 + k) * kPT, a.r[k] + g);
                copy_async4(p + (9 + k) * kPT, a.d[k] + g);
            }
        }
        for (int s = b; s < min(e, P.x_slots); ++s) {
            if ((s - b) * kPT + tid >= n) break;
#pragma unroll
            for (int k = 0; k < 3; ++k) copy_async4(sx + (s * 3 + k) * kPT, a.x[k] + v + (s - b) * kPT);
        }
#pragma unroll
        for (int u = 0; u < kRegSlots; ++u) {
            if (u < b || u >= e || (u - b) * kPT + tid >= n) continue;
            const int64_t g = v + (u - b) * kPT;
#pragma unroll
            for (int k = 0; k < 6; ++k) A[u][k] = a.A[k][g];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                r[u][k] = a.r[k][g];
                d[u][k] = a.d[k][g];
            }
        }
    }
    __syncthreads();
    if (a.persist_d0) {
        // The strip-swept cloths' delta0 and the decision to iterate, formed here as
        // k_assemble_finish forms them (the step then launches that kernel only for the
        // strip-swept cloths this launch does not run).
        for (int j = 0; j < np; ++j) {
            const InstParams& ip = a.inst[pieces[j].inst];
            if (!ip.strip) continue;
            const double total = strip_delta0<kWarps>(a, ip);
            if (tid == 0) {
                uint32_t fl = 0u;
                bool run = (0 < ip.imax) && (total > (double)ip.eps2 * total);
                if (!isfinite(total)) {
                    fl |= OC_FLAG_NON_FINITE;
                    run = false;
                }
                st[j].dn = pair_from(total * pieces[j].scale);
                st[j].thresh = pair_from((double)ip.eps2 * total * pieces[j].scale);
                st[j].d0 = total;
                st[j].it = 0;
                st[j].fl = fl;
                st[j].run[0] = run ? 1 : 0;
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // a thread reads back only its own copies
    __syncthreads();
    if (CS > 1) cluster_wait();
    bool whole = true;  // no wait of this CTA has given up
    unsigned q = 0;
    for (;; ++q) {
        const int cur = q & 1, nxt = cur ^ 1;
        const bool dir = cur == 0, first = q == 0;
        const uint32_t tag = base + q + 1;
        int any = 0;
        for (int j = 0; j < np; ++j) any |= st[j].run[cur];
        if (!any) break;
        if ((int)blockIdx.x == a.withhold_block) {
            whole = false;
            break;
        }
        // The pass of every running piece; each warp sends its partial to the cloth's CTAs of
        // this cluster.
        for (int j = 0; j < np; ++j) {
            if (!st[j].run[cur]) continue;
            const int b = pieces[j].slot0, e = pieces[j].slot1, n = pieces[j].n;
            const float scal = st[j].scal[cur], scale = pieces[j].scale;
            Acc part = acc_zero();
#pragma unroll
            for (int u = 0; u < kRegSlots; ++u) {
                if (u < b || u >= e) continue;  // a slot's lanes past its end hold zeros, whose terms are zeros
                if (dir)
                    dir_vertex(A[u], r[u], d[u], first, scal, scale, part);
                else
                    res_vertex(A[u], r[u], d[u], scal, scale, part);
            }
#pragma unroll 2
            for (int s = max(b, kRegSlots); s < min(e, s_end); ++s) {
                if ((s - b) * kPT + tid >= n) break;
                float* p = sm + (s - kRegSlots) * kSlotFloats * kPT;
                float As[6], rs[3], ds[3];
#pragma unroll
                for (int k = 0; k < 6; ++k) As[k] = p[k * kPT];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    rs[k] = p[(6 + k) * kPT];
                    ds[k] = p[(9 + k) * kPT];
                }
                if (dir) {
                    dir_vertex(As, rs, ds, first, scal, scale, part);
                    if (!first) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) p[(9 + k) * kPT] = ds[k];
                    }
                } else {
                    res_vertex(As, rs, ds, scal, scale, part);
#pragma unroll
                    for (int k = 0; k < 3; ++k) p[(6 + k) * kPT] = rs[k];
                }
            }
            for (int s = max(b, s_end); s < e; ++s) {
                if ((s - b) * kPT + tid >= n) break;
                const int64_t g = pieces[j].v + (s - b) * kPT + tid;
                float As[6], rs[3], ds[3];
#pragma unroll
                for (int k = 0; k < 6; ++k) As[k] = a.A[k][g];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    rs[k] = a.r[k][g];
                    ds[k] = a.d[k][g];
                }
                if (dir) {
                    dir_vertex(As, rs, ds, first, scal, scale, part);
                    if (!first) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) a.d[k][g] = ds[k];
                    }
                } else {
                    res_vertex(As, rs, ds, scal, scale, part);
#pragma unroll
                    for (int k = 0; k < 3; ++k) a.r[k][g] = rs[k];
                }
            }
            part = lanes_sum<16>(part);
            const int r0 = pieces[j].rank0, nr = pieces[j].ranks;
            if (nr == 1) {
                if (lane == 0) put_local(&st[j].box[cur][w], part, tag);
            } else if (lane >= r0 && lane < r0 + nr) {
                // The cloth is the first piece of its CTAs, but the last of the one it starts in.
                put_cluster(&s_box[cur][pieces[j].tail && lane == r0 ? 1 : 0][rank * kWarps + w], lane, part, tag);
            }
        }
        // While the packets travel: x = x + alpha d (IMP:322).
        if (!dir) {
            for (int j = 0; j < np; ++j) {
                if (!st[j].run[cur]) continue;
                const int b = pieces[j].slot0, e = pieces[j].slot1, n = pieces[j].n;
                const int64_t v = pieces[j].v + tid;
                const float alpha = st[j].scal[cur];
#pragma unroll
                for (int u = 0; u < kRegSlots; ++u) {
                    if (u < b || u >= min(e, P.x_slots)) continue;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        float* xp = sx + (u * 3 + k) * kPT;
                        *xp = *xp + d[u][k] * alpha;
                    }
                }
                for (int s = max(b, kRegSlots); s < min(e, P.x_slots); ++s) {
                    const float* p = sm + ((s - kRegSlots) * kSlotFloats + 9) * kPT;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        float* xp = sx + (s * 3 + k) * kPT;
                        *xp = *xp + p[k * kPT] * alpha;
                    }
                }
                if (e <= P.x_slots) continue;
                // The rest in the planes: four slots' loads in flight, then their stores.
#pragma unroll
                for (int u0 = 0; u0 < kRegSlots; u0 += 4) {
                    if (u0 + 4 <= max(b, P.x_slots) || u0 >= e) continue;
                    float y[4][3];
                    bool ok[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int s = u0 + u;
                        ok[u] = s >= max(b, P.x_slots) && s < e && (s - b) * kPT + tid < n;
                        if (ok[u]) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) y[u][k] = a.x[k][v + (s - b) * kPT];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (ok[u]) {
#pragma unroll
                            for (int k = 0; k < 3; ++k)
                                a.x[k][v + (u0 + u - b) * kPT] = y[u][k] + d[u0 + u][k] * alpha;
                        }
                }
                for (int s0 = max(max(b, kRegSlots), P.x_slots); s0 < e; s0 += 4) {
                    float y[4][3], ds[4][3];
                    bool ok[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int s = s0 + u;
                        ok[u] = s < e && (s - b) * kPT + tid < n;
                        if (ok[u]) {
                            const float* p = sm + ((s - kRegSlots) * kSlotFloats + 9) * kPT;
                            const int64_t g = v + (s - b) * kPT;
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                y[u][k] = a.x[k][g];
                                ds[u][k] = s < s_end ? p[k * kPT] : a.d[k][g];
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (ok[u]) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) a.x[k][v + (s0 + u - b) * kPT] = y[u][k] + ds[u][k] * alpha;
                        }
                }
            }
        }
        // The totals of the phase and the scalar rule: warp w takes the pieces w, w + kWarps, ...
        // First the sums of this cluster's CTAs (its first CTA sends them to the other clusters),
        // then those of all clusters.
        ulonglong2* const packets = P.packets + (size_t)cur * P.n_packets;
        bool ok = true;
        for (int j = w; j < np && ok; j += kWarps) {
            if (!st[j].run[cur]) {
                if (lane == 0) st[j].run[nxt] = 0;
                continue;
            }
            const PersistPiece pc = pieces[j];
            PieceState& ps = st[j];
            Acc total;
            if (pc.ranks == 1) {
                Acc v = acc_zero();
                // Every eight lanes read the eight warps' packets, so every lane has the sum.
                ok = poll<1>(1u, a, P.err, [&](int) { return get_cluster(&ps.box[cur][lane % kWarps], tag, v); });
                total = lanes_sum<kWarps / 2>(v);
            } else {
                const ulonglong2* box = s_box[cur][pc.tail && rank == pc.rank0 ? 1 : 0] + lane;
                constexpr int U = kMaxCluster * kWarps / 32;
                Acc v[U];
                unsigned want = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    v[u] = acc_zero();
                    const int from = (u * 32 + lane) / kWarps;
                    if (from >= pc.rank0 && from < pc.rank0 + pc.ranks) want |= 1u << u;
                }
                ok = poll<U>(want, a, P.err, [&](int u) { return get_cluster(box + u * 32, tag, v[u]); });
                total = v[0];
#pragma unroll
                for (int u = 1; u < U; ++u) total = acc_merge(total, v[u]);
                total = lanes_sum<16>(total);
            }
            if (ok && pc.clusters > 1) {  // the other clusters
                if (rank == pc.rank0 && lane < CS)
                    put_global(packets + pc.packet + lane * pc.clusters + pc.k, total, tag);
                const ulonglong2* from = packets + pc.packet + rank * pc.clusters + lane;
                if (pc.clusters <= 8) {
                    Acc v = acc_zero();
                    ok = poll<1>(lane < pc.clusters ? 1u : 0u, a, P.err, [&](int) { return get_global(from, tag, v); });
                    total = lanes_sum<4>(v);
                } else {
                    Acc sum = acc_zero();
                    for (int k0 = 0; k0 < pc.clusters && ok; k0 += 5 * 32) {
                        Acc v[5];
                        unsigned want = 0;
#pragma unroll
                        for (int u = 0; u < 5; ++u) {
                            v[u] = acc_zero();
                            if (k0 + u * 32 + lane < pc.clusters) want |= 1u << u;
                        }
                        ok = poll<5>(want, a, P.err, [&](int u) { return get_global(from + k0 + u * 32, tag, v[u]); });
#pragma unroll
                        for (int u = 0; u < 5; ++u) sum = acc_merge(sum, v[u]);
                    }
                    total = lanes_sum<16>(sum);
                }
            }
            if (lane == 0 && ok) {
                total = pair_norm(total);
                const bool fin = pair_finite(total);
                bool run = true;
                float scal = 0.0f;
                if (dir) {  // d.(A d) -> alpha
                    if (!(total.s > 0.0f) || !fin) {
                        ps.fl |= fin ? OC_FLAG_BREAKDOWN : OC_FLAG_NON_FINITE;
                        run = false;
                    } else {
                        scal = quotient(ps.dn, total);
                    }
                    ps.scal[nxt] = scal;
                    ps.run[nxt] = run ? 1 : 0;
                    ps.dq = total;
                    if (run) ps.alpha = scal;
                } else {  // r.r -> beta, the stop test
                    const int it = ps.it + 1;
                    const bool above = pair_gt(total, ps.thresh);
                    if (!fin) {
                        ps.fl |= OC_FLAG_NON_FINITE;
                        run = false;
                    } else if (!(it < ps.imax && above)) {
                        if (above) ps.fl |= OC_FLAG_NOT_CONVERGED;
                        run = false;
                    }
                    scal = quotient(total, ps.dn);
                    ps.scal[nxt] = scal;
                    ps.run[nxt] = run ? 1 : 0;
                    ps.beta = scal;
                    ps.dn = total;
                    ps.it = it;
                }
            }
        }
        if (!ok && lane == 0) {
            atomicOr(P.err, 1);
            s_ok[nxt] = 0;
        }
        __syncthreads();
        whole = s_ok[nxt] != 0;
        if (!whole) break;
    }
    if (CS > 1) cluster_arrive();
    if (tid == 0) leave_tags(P.ctl, base, q + 2);
    if (whole) {
        // The cloths' scalars for the host, by each cloth's first piece.
        for (int j = tid; j < np; j += kPT) {
            if (!pieces[j].head) continue;
            const PieceState& ps = st[j];
            InstState& is = a.state[pieces[j].inst];
            is.delta0 = ps.d0;
            const double unit = 1.0f / pieces[j].scale;  // (a power of two)
            is.delta_new = ((double)ps.dn.s + (double)ps.dn.c) * unit;
            is.dq = ((double)ps.dq.s + (double)ps.dq.c) * unit;
            is.alpha = ps.alpha;
            is.beta = ps.beta;
            is.iter = ps.it;
            is.flags = ps.fl;
            is.active = 0;
            is.ticket = 0;
        }
        for (int j = 0; j < np; ++j)
            persist_update(a, a.inst[pieces[j].inst], pieces[j].v + tid, pieces[j].n, pieces[j].slot0, pieces[j].slot1,
                           P.x_slots, sx);
    }
    if (CS > 1) cluster_wait();
}

// The same with one piece per CTA (or none, n = 0), the plan whenever there are no more cloths
// than CTAs: its slots start at 0, and warp 0 keeps its cloth's scalars in its registers.  The passes are
// straight-line code over KR register slots (a slot past the piece holds zeros, whose terms are
// zeros): with 8 warps an SM, a phase's length is its instructions and their fetches, so the
// plan takes the smallest KR that holds the piece.  FULL: KR slots hold the whole piece, x, X
// and V in registers too, and memory is touched once at either end.
template <int KR, bool FULL>
__global__ void __launch_bounds__(kPT, 1) k_cg_persist_one(const StepArgs a, const PersistPlan P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_ok[2];
    __shared__ float s_scal[2];
    __shared__ int s_run[2];
    __shared__ __align__(16) ulonglong2 s_box[2][kMaxCluster * kWarps];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int CS = P.cluster, rank = (int)blockIdx.x % CS;
    if (!clusters_as_planned(P)) return;
    const PersistPiece pc = P.pieces[blockIdx.x];
    const uint32_t base = *(volatile uint32_t*)&P.ctl->base;
    float* const sm = reinterpret_cast<float*>(smem_raw) + tid;
    float* const sx = sm + (size_t)P.smem_slots * kSlotFloats * kPT;
    const int s_end = KR + P.smem_slots;
    const int n = pc.n, e = pc.slot1;
    const int64_t v = pc.v + tid;
    const bool upd = !a.cg_only;
    const float scale = pc.scale;

    if (tid < 2) s_ok[tid] = 1;
    for (int i = tid; i < 2 * kMaxCluster * kWarps; i += kPT) (&s_box[0][0])[i] = empty_packet(base);
    if (CS > 1) cluster_arrive();
    float A[KR][6], r[KR][3], d[KR][3];
    float x[FULL ? KR : 1][3];
    float4 X[FULL ? KR : 1], V[FULL ? KR : 1];
    if constexpr (!FULL) {
        for (int s = KR; s < min(e, s_end); ++s) {
            if (s * kPT + tid >= n) break;
            float* p = sm + (s - KR) * kSlotFloats * kPT;
            const int64_t g = v + s * kPT;
#pragma unroll
            for (int k = 0; k < 6; ++k) copy_async4(p + k * kPT, a.A[k] + g);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                copy_async4(p + (6 + k) * kPT, a.r[k] + g);
                copy_async4(p + (9 + k) * kPT, a.d[k] + g);
            }
        }
        for (int s = 0; s < min(e, P.x_slots); ++s) {
            if (s * kPT + tid >= n) break;
#pragma unroll
            for (int k = 0; k < 3; ++k) copy_async4(sx + (s * 3 + k) * kPT, a.x[k] + v + s * kPT);
        }
    }
#pragma unroll
    for (int u = 0; u < KR; ++u) {
        const bool own = u * kPT + tid < n;
        const int64_t g = v + u * kPT;
#pragma unroll
        for (int k = 0; k < 6; ++k) A[u][k] = own ? a.A[k][g] : 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            r[u][k] = own ? a.r[k][g] : 0.0f;
            d[u][k] = own ? a.d[k][g] : 0.0f;
            if constexpr (FULL) x[u][k] = own ? a.x[k][g] : 0.0f;
        }
        if constexpr (FULL)
            if (own && upd) {
                X[u] = a.X[g];
                V[u] = a.V[g];
            }
    }
    // Warp 0's scalars (every lane): delta_new, the threshold, the last d.(A d), each times scale.
    Acc dn = acc_zero(), thresh = acc_zero(), dq = acc_zero();
    double d0 = 0.0;
    float alpha = 0.0f, beta = 0.0f;
    int it = 0, imax = 0;
    uint32_t fl = 0u;
    bool go = false;
    if (n > 0) {
        const InstParams& ip = a.inst[pc.inst];
        if (a.persist_d0 && ip.strip) {  // as in k_cg_persist
            const double total = strip_delta0<kWarps>(a, ip);
            if (w == 0) {
                d0 = __shfl_sync(0xffffffffu, total, 0);
                dn = pair_from(d0 * scale);
                go = (0 < ip.imax) && (d0 > (double)ip.eps2 * d0);
                if (!isfinite(d0)) {
                    fl |= OC_FLAG_NON_FINITE;
                    go = false;
                }
            }
        } else if (w == 0) {
            const InstState& is = a.state[pc.inst];
            d0 = __ldcg(&is.delta0);
            dn = pair_from(__ldcg(&is.delta_new) * scale);
            it = __ldcg(&is.iter);
            fl = __ldcg(&is.flags);
            go = __ldcg(&is.active) != 0;
        }
        thresh = pair_from((double)ip.eps2 * d0 * scale);
        imax = ip.imax;
    }
    if (tid == 0) {
        s_run[0] = go ? 1 : 0;
        s_scal[0] = 0.0f;
    }
    if constexpr (!FULL) asm volatile("cp.async.wait_all;" ::: "memory");  // a thread reads back only its own copies
    __syncthreads();
    if (CS > 1) cluster_wait();
    // The packets that this lane waits for, and where they are.
    constexpr int U = kMaxCluster * kWarps / 32;
    unsigned want_box = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int from = (u * 32 + lane) / kWarps;
        if (from >= pc.rank0 && from < pc.rank0 + pc.ranks) want_box |= 1u << u;
    }
    bool whole = true;  // no wait of this CTA has given up
    unsigned q = 0;
    for (;; ++q) {
        const int cur = q & 1, nxt = cur ^ 1;
        const bool dir = cur == 0;
        const uint32_t tag = base + q + 1;
        if (!s_run[cur]) break;
        if ((int)blockIdx.x == a.withhold_block) {
            whole = false;
            break;
        }
        const float scal = s_scal[cur];
        Acc part = acc_zero();
        if (dir) {
            const bool first = q == 0;
#pragma unroll
            for (int u = 0; u < KR; ++u) dir_vertex(A[u], r[u], d[u], first, scal, scale, part);
        } else {
#pragma unroll
            for (int u = 0; u < KR; ++u) res_vertex(A[u], r[u], d[u], scal, scale, part);
        }
        if constexpr (!FULL) {
#pragma unroll 2
            for (int s = KR; s < min(e, s_end); ++s) {
                if (s * kPT + tid >= n) break;
                float* p = sm + (s - KR) * kSlotFloats * kPT;
                float As[6], rs[3], ds[3];
#pragma unroll
                for (int k = 0; k < 6; ++k) As[k] = p[k * kPT];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    rs[k] = p[(6 + k) * kPT];
                    ds[k] = p[(9 + k) * kPT];
                }
                if (dir) {
                    dir_vertex(As, rs, ds, q == 0, scal, scale, part);
                    if (q > 0) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) p[(9 + k) * kPT] = ds[k];
                    }
                } else {
                    res_vertex(As, rs, ds, scal, scale, part);
#pragma unroll
                    for (int k = 0; k < 3; ++k) p[(6 + k) * kPT] = rs[k];
                }
            }
            for (int s = s_end; s < e; ++s) {
                if (s * kPT + tid >= n) break;
                const int64_t g = v + s * kPT;
                float As[6], rs[3], ds[3];
#pragma unroll
                for (int k = 0; k < 6; ++k) As[k] = a.A[k][g];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    rs[k] = a.r[k][g];
                    ds[k] = a.d[k][g];
                }
                if (dir) {
                    dir_vertex(As, rs, ds, q == 0, scal, scale, part);
                    if (q > 0) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) a.d[k][g] = ds[k];
                    }
                } else {
                    res_vertex(As, rs, ds, scal, scale, part);
#pragma unroll
                    for (int k = 0; k < 3; ++k) a.r[k][g] = rs[k];
                }
            }
        }
        part = lanes_sum<16>(part);
        if (pc.ranks == 1) {
            if (lane == 0) put_local(&s_box[cur][rank * kWarps + w], part, tag);
        } else if (lane >= pc.rank0 && lane < pc.rank0 + pc.ranks) {
            put_cluster(&s_box[cur][rank * kWarps + w], lane, part, tag);
        }
        // Warp 0 sums this cluster's partials and sends the sum to the other clusters.
        Acc total = acc_zero();
        bool ok = true;
        ulonglong2* const packets = P.packets + (size_t)cur * P.n_packets + pc.packet;
        if (w == 0) {
            Acc t[U];
#pragma unroll
            for (int u = 0; u < U; ++u) t[u] = acc_zero();
            const ulonglong2* box = s_box[cur] + lane;
            ok = poll<U>(want_box, a, P.err, [&](int u) { return get_cluster(box + u * 32, tag, t[u]); });
            total = lanes_sum<16>(acc_merge(acc_merge(t[0], t[1]), acc_merge(t[2], t[3])));
            if (ok && pc.clusters > 1) {
                if (pc.full) {  // every rank of every cluster holds a piece: rank r sends copy r
                    if (lane == 0) put_global(packets + rank * pc.clusters + pc.k, total, tag);
                } else if (rank == pc.rank0 && lane < CS) {
                    put_global(packets + lane * pc.clusters + pc.k, total, tag);
                }
            }
        }
        if (!dir) {  // while the packets travel: x = x + alpha d (IMP:322)
            if constexpr (FULL) {
#pragma unroll
                for (int u = 0; u < KR; ++u)
#pragma unroll
                    for (int k = 0; k < 3; ++k) x[u][k] = x[u][k] + d[u][k] * scal;
            } else {
                const int xs = min(e, P.x_slots);
#pragma unroll
                for (int u = 0; u < KR; ++u)
                    if (u < xs) {
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            float* xp = sx + (u * 3 + k) * kPT;
                            *xp = *xp + d[u][k] * scal;
                        }
                    }
                for (int s = KR; s < xs; ++s) {
                    const float* p = sm + ((s - KR) * kSlotFloats + 9) * kPT;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        float* xp = sx + (s * 3 + k) * kPT;
                        *xp = *xp + p[k * kPT] * scal;
                    }
                }
                // The rest in the planes: four slots' loads in flight, then their stores.
                constexpr int B = 4;
#pragma unroll
                for (int u0 = 0; u0 < KR; u0 += B) {
                    if (u0 + B <= P.x_slots) continue;
                    float y[B][3];
#pragma unroll
                    for (int u = 0; u < B; ++u)
                        if (u0 + u < KR && u0 + u >= P.x_slots && (u0 + u) * kPT + tid < n) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) y[u][k] = a.x[k][v + (u0 + u) * kPT];
                        }
#pragma unroll
                    for (int u = 0; u < B; ++u)
                        if (u0 + u < KR && u0 + u >= P.x_slots && (u0 + u) * kPT + tid < n) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) a.x[k][v + (u0 + u) * kPT] = y[u][k] + d[u0 + u][k] * scal;
                        }
                }
                for (int s0 = max(KR, P.x_slots); s0 < e; s0 += B) {
                    float y[B][3];
#pragma unroll
                    for (int u = 0; u < B; ++u)
                        if ((s0 + u) * kPT + tid < n) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) y[u][k] = a.x[k][v + (s0 + u) * kPT];
                        }
#pragma unroll
                    for (int u = 0; u < B; ++u)
                        if ((s0 + u) * kPT + tid < n) {
                            const int s = s0 + u;
                            const float* p = sm + ((s - KR) * kSlotFloats + 9) * kPT;
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                const float dk = s < s_end ? p[k * kPT] : a.d[k][v + s * kPT];
                                a.x[k][v + s * kPT] = y[u][k] + dk * scal;
                            }
                        }
                }
            }
        }
        if (w == 0) {
            if (ok && pc.clusters > 1) {
                const ulonglong2* from = packets + rank * pc.clusters + lane;
                if (pc.clusters <= 8) {
                    Acc y = acc_zero();
                    ok = poll<1>(lane < pc.clusters ? 1u : 0u, a, P.err, [&](int) { return get_global(from, tag, y); });
                    total = lanes_sum<4>(y);
                } else {
                    Acc sum = acc_zero();
                    for (int k0 = 0; k0 < pc.clusters && ok; k0 += 5 * 32) {
                        Acc y[5];
                        unsigned want = 0;
#pragma unroll
                        for (int u = 0; u < 5; ++u) {
                            y[u] = acc_zero();
                            if (k0 + u * 32 + lane < pc.clusters) want |= 1u << u;
                        }
                        ok = poll<5>(want, a, P.err, [&](int u) { return get_global(from + k0 + u * 32, tag, y[u]); });
                        sum = acc_merge(sum, acc_merge(acc_merge(acc_merge(y[0], y[1]), acc_merge(y[2], y[3])), y[4]));
                    }
                    total = lanes_sum<16>(sum);
                }
            }
            // Lane 0's total in every lane: the lanes past a short sum would send the quotient's
            // warp through its FP64 path too.
            total = pair_norm(make_acc(__shfl_sync(0xffffffffu, total.s, 0), __shfl_sync(0xffffffffu, total.c, 0)));
            const bool fin = pair_finite(total);
            bool run = ok;
            float next = 0.0f;
            if (dir) {  // d.(A d) -> alpha
                dq = total;
                if (!(total.s > 0.0f) || !fin) {
                    fl |= fin ? OC_FLAG_BREAKDOWN : OC_FLAG_NON_FINITE;
                    run = false;
                } else {
                    next = quotient(dn, total);
                    alpha = next;
                }
            } else {  // r.r -> beta, the stop test
                const bool above = pair_gt(total, thresh);
                next = quotient(total, dn);
                beta = next;
                dn = total;
                ++it;
                if (!fin) {
                    fl |= OC_FLAG_NON_FINITE;
                    run = false;
                } else if (!(it < imax && above)) {
                    if (above) fl |= OC_FLAG_NOT_CONVERGED;
                    run = false;
                }
            }
            if (lane == 0) {
                s_scal[nxt] = next;
                s_run[nxt] = run ? 1 : 0;
                if (!ok) {
                    atomicOr(P.err, 1);
                    s_ok[nxt] = 0;
                }
            }
        }
        __syncthreads();
        whole = s_ok[nxt] != 0;
        if (!whole) break;
    }
    if (CS > 1) cluster_arrive();
    if (tid == 0) {
        leave_tags(P.ctl, base, q + 2);
        if (whole && pc.head && n > 0) {
            InstState& is = a.state[pc.inst];
            is.delta0 = d0;
            const double unit = 1.0f / scale;  // (a power of two)
            is.delta_new = ((double)dn.s + (double)dn.c) * unit;
            is.dq = ((double)dq.s + (double)dq.c) * unit;
            is.alpha = alpha;
            is.beta = beta;
            is.iter = it;
            is.flags = fl;
            is.active = 0;
            is.ticket = 0;
        }
    }
    if (whole && n > 0) {
        const InstParams& ip = a.inst[pc.inst];
        if constexpr (FULL) {
#pragma unroll
            for (int u = 0; u < KR; ++u) {
                if (u * kPT + tid >= n) continue;
                const int64_t g = v + u * kPT;
#pragma unroll
                for (int k = 0; k < 3; ++k) a.x[k][g] = x[u][k];
                if (upd) {
                    update_vertex(ip, a.dt, x[u][0], x[u][1], x[u][2], X[u], V[u]);
                    a.X[g] = X[u];
                    a.V[g] = V[u];
                }
            }
        } else {
            persist_update(a, ip, v, n, 0, e, P.x_slots, sx);
        }
    }
    if (CS > 1) cluster_wait();
}

cudaLaunchConfig_t persist_config(int grid, int cluster, size_t smem, cudaStream_t stream, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)kPT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    int n = 0;
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    attr[n].id = cudaLaunchAttributeCooperative;
    attr[n].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = n + 1;
    return cfg;
}

// The kernel of a plan: with one piece per CTA, the smallest one whose register slots hold it.
typedef void (*PersistFn)(StepArgs, PersistPlan);
PersistFn persist_fn(const PersistPlan& plan) {
    if (!plan.one) return k_cg_persist;
    if (plan.max_slots <= 1) return k_cg_persist_one<1, true>;
    if (plan.max_slots <= 2) return k_cg_persist_one<2, true>;
    if (plan.max_slots <= 3) return k_cg_persist_one<3, true>;
    if (plan.max_slots <= 5) return k_cg_persist_one<5, true>;
    if (plan.max_slots <= kFullSlots) return k_cg_persist_one<kFullSlots, true>;
    return k_cg_persist_one<kOneRegSlots, false>;
}

}  // namespace

void persist_layout(PersistPlan* plan, int max_smem) {
    PersistPlan& P = *plan;
    const size_t slot = (size_t)kSlotFloats * kPT * sizeof(float), xs = (size_t)3 * kPT * sizeof(float);
    const size_t fixed = P.one ? 0 : persist_state_bytes(P.max_pieces), room = (size_t)max_smem;
    P.smem_slots = P.x_slots = 0;
    P.smem = fixed;
    P.on_chip = 1;
    P.chip_slots = P.chip_x = P.max_slots;
    if (P.one && P.max_slots <= kFullSlots) return;
    P.smem_slots = std::max(0, P.max_slots - (P.one ? kOneRegSlots : kRegSlots));
    if (fixed >= room) P.smem_slots = 0;
    else P.smem_slots = (int32_t)std::min<size_t>((size_t)P.smem_slots, (room - fixed) / slot);
    P.smem += P.smem_slots * slot;
    if (P.smem < room) P.x_slots = (int32_t)std::min<size_t>((size_t)P.max_slots, (room - P.smem) / xs);
    P.smem += P.x_slots * xs;
    P.on_chip = P.x_slots == P.max_slots && P.smem <= room;
    P.chip_slots = (P.one ? kOneRegSlots : kRegSlots) + P.smem_slots;
    P.chip_x = P.x_slots;
}

cudaError_t prepare_persist(int device, int* max_smem, int* max_clusters, int* max_pairs) {
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    const PersistFn fns[] = {k_cg_persist, k_cg_persist_one<1, true>, k_cg_persist_one<2, true>,
                             k_cg_persist_one<3, true>, k_cg_persist_one<5, true>, k_cg_persist_one<kFullSlots, true>,
                             k_cg_persist_one<kOneRegSlots, false>};
    *max_smem = optin;
    for (PersistFn f : fns) {
        cudaFuncAttributes fa;
        if ((e = cudaFuncGetAttributes(&fa, f)) != cudaSuccess) return e;
        *max_smem = std::min(*max_smem, optin - (int)fa.sharedSizeBytes);
    }
    for (PersistFn f : fns) {
        if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, *max_smem)) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    }
    const int sizes[2] = {kMaxCluster, 2};
    int* const counts[2] = {max_clusters, max_pairs};
    for (int i = 0; i < 2; ++i) {
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = persist_config(sizes[i], sizes[i], (size_t)*max_smem, nullptr, attr);
        cfg.numAttrs = 1;  // the cluster size alone
        *counts[i] = 0;
        if (cudaOccupancyMaxActiveClusters(counts[i], k_cg_persist, &cfg) != cudaSuccess) {
            cudaGetLastError();
            *counts[i] = 0;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_cg_persist(const StepArgs& a, const PersistPlan& plan, cudaStream_t stream) {
    if (plan.grid <= 0) return cudaErrorInvalidValue;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = persist_config(plan.grid, plan.cluster, plan.smem, stream, attr);
    return cudaLaunchKernelEx(&cfg, persist_fn(plan), a, plan);
}

}  // namespace oc
