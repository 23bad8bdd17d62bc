// What the kernels that run whole CG loops share (oc_persist.cu, oc_sim.cu, oc_bsr.cu,
// oc_coupled.cu): the packets by
// which CTAs exchange partial sums, the bounded polls that wait for them, the quotient of the
// scalar rule, and the two passes of one vertex.
//
// A packet is a float pair in two 8-byte words, each with the exchange's tag beside its float:
// a word is one access, so the data is its own flag and needs no fence.
#pragma once

#include <cuda_runtime.h>

#include "oc_device.cuh"
#include "oc_internal.h"

namespace oc {
namespace {

__device__ __forceinline__ int load_relaxed(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long word_of(float v, uint32_t tag) {
    return (unsigned long long)tag << 32 | __float_as_uint(v);
}

// What a box holds before its first packet in a launch whose tags are base + 1, base + 2, ...
__device__ __forceinline__ ulonglong2 empty_packet(uint32_t base) {
    const unsigned long long w = word_of(0.0f, base);
    return make_ulonglong2(w, w);
}

__device__ __forceinline__ void put_global(ulonglong2* p, Acc v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(word_of(v.s, tag)), "l"(word_of(v.c, tag))
                 : "memory");
}

__device__ __forceinline__ bool get_global(const ulonglong2* p, uint32_t tag, Acc& v) {
    unsigned long long s, c;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(s), "=l"(c) : "l"(p) : "memory");
    v = make_acc(__uint_as_float((uint32_t)s), __uint_as_float((uint32_t)c));
    return (uint32_t)(s >> 32) == tag && (uint32_t)(c >> 32) == tag;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The same words in this CTA's shared memory, and in that of CTA `rank` of the cluster (at
// this CTA's address p).
__device__ __forceinline__ void put_local(ulonglong2* p, Acc v, uint32_t tag) {
    asm volatile("st.relaxed.cta.shared::cta.v2.b64 [%0], {%1, %2};" ::"r"(smem_addr(p)), "l"(word_of(v.s, tag)),
                 "l"(word_of(v.c, tag))
                 : "memory");
}

__device__ __forceinline__ void put_cluster(ulonglong2* p, int rank, Acc v, uint32_t tag) {
    asm volatile("{ .reg .b32 a; mapa.shared::cluster.u32 a, %0, %1;\n\t"
                 "st.relaxed.cluster.shared::cluster.v2.b64 [a], {%2, %3}; }" ::"r"(smem_addr(p)),
                 "r"(rank), "l"(word_of(v.s, tag)), "l"(word_of(v.c, tag))
                 : "memory");
}

// 1 into the word of CTA `rank` of the cluster at this CTA's address p.
__device__ __forceinline__ void flag_cluster(int* p, int rank) {
    asm volatile("{ .reg .b32 a; mapa.shared::cluster.u32 a, %0, %1;\n\t"
                 "st.relaxed.cluster.shared::cluster.b32 [a], %2; }" ::"r"(smem_addr(p)),
                 "r"(rank), "r"(1)
                 : "memory");
}

__device__ __forceinline__ bool get_cluster(const ulonglong2* p, uint32_t tag, Acc& v) {
    unsigned long long s, c;
    asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];" : "=l"(s), "=l"(c) : "r"(smem_addr(p)) : "memory");
    v = make_acc(__uint_as_float((uint32_t)s), __uint_as_float((uint32_t)c));
    return (uint32_t)(s >> 32) == tag && (uint32_t)(c >> 32) == tag;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// A pair's sum over the lanes, in every lane.
template <int FROM>
__device__ __forceinline__ Acc lanes_sum(Acc v) {
#pragma unroll
    for (int o = FROM; o > 0; o >>= 1)
        v = acc_merge(v, make_acc(__shfl_xor_sync(0xffffffffu, v.s, o), __shfl_xor_sync(0xffffffffu, v.c, o)));
    return v;
}

// Polls until get(u) has been true for every u < 5 of every lane (mask `want` of the ones that
// the lane waits for); false when the wait gave up.
template <int N, class Get>
__device__ __forceinline__ bool poll(unsigned want, const StepArgs& a, const int* err, Get get) {
    unsigned spins = 0;
    while (true) {
#pragma unroll
        for (int u = 0; u < N; ++u)
            if ((want >> u & 1u) && get(u)) want &= ~(1u << u);
        if (!__any_sync(0xffffffffu, want != 0)) return true;
        ++spins;
        if (spins > a.barrier_polls || ((spins & 63u) == 0 && __any_sync(0xffffffffu, load_relaxed(err) != 0)))
            return false;
    }
}

// The sum of `part` over the threads of `np` CTAs without clusters, in every lane of warp 0 (in
// the others `total` is not set): the CTA's own sum goes out as packet `idx` of `packets`, and
// warp 0 reads all of them.  With `publish`, what the CTA's threads stored before is visible to
// the other CTAs' loads after the barrier that the caller puts behind.  False (in warp 0) when a
// wait gave up.  Every thread of the CTA, of WARPS <= 32 warps, calls it.
template <int WARPS>
__device__ __forceinline__ bool pull_sum(Acc part, ulonglong2* packets, int idx, int np, uint32_t tag, bool publish,
                                         const StepArgs& a, const int* err, Acc* warp_sums, Acc& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    part = lanes_sum<16>(part);
    if (lane == 0) warp_sums[w] = part;
    __syncthreads();
    if (w != 0) return true;
    bool ok = true;
    total = lanes_sum<16>(lane < WARPS ? warp_sums[lane] : acc_zero());
    if (np > 1) {
        if (lane == 0) {
            if (publish) __threadfence();
            put_global(packets + idx, total, tag);
        }
        Acc sum = acc_zero();
        for (int k0 = 0; k0 < np && ok; k0 += 5 * 32) {
            Acc y[5];
            unsigned want = 0;
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                y[u] = acc_zero();
                if (k0 + u * 32 + lane < np) want |= 1u << u;
            }
            ok = poll<5>(want, a, err, [&](int u) { return get_global(packets + k0 + u * 32 + lane, tag, y[u]); });
            sum = acc_merge(sum, acc_merge(acc_merge(acc_merge(y[0], y[1]), acc_merge(y[2], y[3])), y[4]));
        }
        total = lanes_sum<16>(sum);
        if (publish) __threadfence();  // by every lane that has read packets, before the caller's barrier
        __syncwarp();
    }
    total = pair_norm(total);
    return ok;
}

// By one thread of a CTA that leaves: the last one moves the tags past those of this launch.
__device__ __forceinline__ void leave_tags(PersistCtl* ctl, uint32_t base, uint32_t used) {
    atomicMax(&ctl->used, used);
    __threadfence();
    if (atomicAdd(&ctl->left, 1u) == gridDim.x - 1) {
        ctl->base = base + *(volatile uint32_t*)&ctl->used;
        ctl->used = 0;
        ctl->left = 0;
    }
}

// a / b of two normalised pairs rounded to float; in FP64 where pair_div's remainder or the quotient
// would leave the float range.  The interval lies low because the sums are scaled down (sum_scale).
__device__ __forceinline__ float quotient(Acc a, Acc b) {
    const float ma = fabsf(a.s), mb = fabsf(b.s);
    if (ma >= 0x1p-80f && ma <= 0x1p40f && mb >= 0x1p-80f && mb <= 0x1p40f) return pair_div(a, b);
    return (float)(((double)a.s + (double)a.c) / ((double)b.s + (double)b.c));
}

// The dot products' terms are FP32, and a solve whose terms are finite goes on even where their
// total lies beyond FLT_MAX.  So each term is scaled by a power of two, at most one over the number of
// vertices (sum_scale), and no sum of finite terms overflows; the scalars that come from the sums
// (delta, threshold) carry the same factor, their quotients do not.  It is exact but for totals below
// about 2^-101 / scale, whose pairs reach below the smallest float.

// d = r + beta d (not in the first phase, IMP:327); the term of d.(A d) times scale.
__device__ __forceinline__ void dir_vertex(const float (&A)[6], const float (&r)[3], float (&d)[3], bool first,
                                           float beta, float scale, Acc& part) {
    if (!first) {
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = r[k] + d[k] * beta;
    }
    float q0, q1, q2;
    matvec(A, d[0], d[1], d[2], q0, q1, q2);
    acc_add(part, (d[0] * q0 + d[1] * q1 + d[2] * q2) * scale);
}

// r = r - alpha A d (IMP:323); the term of r.r times scale.
__device__ __forceinline__ void res_vertex(const float (&A)[6], float (&r)[3], const float (&d)[3], float alpha,
                                           float scale, Acc& part) {
    float q[3];
    matvec(A, d[0], d[1], d[2], q[0], q[1], q[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = r[k] - q[k] * alpha;
    acc_add(part, (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]) * scale);
}

}  // namespace
}  // namespace oc
