// Transforms over Fr spread over a thread-block cluster: C blocks (4 or 8) hold
// N = C S elements, block r the positions [r S, (r + 1) S) in its shared memory.
// The stages up to length S run inside a block (smem_dit4, smem_dif4); the outer
// ones run on distributed shared memory: with C = 8 the stage of length 2 S on
// pairs of blocks, then in both cases the last two stages as a radix-4 step.
#pragma once

#include "device_util.cuh"

#include <cooperative_groups.h>

namespace vkzg {

namespace cg = cooperative_groups;

// position p of the cluster's N elements
template <int S>
__device__ __forceinline__ Fr *cluster_at(cg::cluster_group &cl, Fr *s, int p) {
    return cl.map_shared_rank(s, p / S) + p % S;
}

// C = 8: the stage of length 2 S of an inverse DIT / a forward DIF; each block of
// a pair takes half of the pair's butterflies.  roots index stride: 8192 / (2 S).
template <int S, int NT>
__device__ __forceinline__ void cluster_pair_dit(cg::cluster_group &cl, Fr *s, const Fr *__restrict__ roots) {
    const int pair = (int)cl.block_rank() & ~1, half = (int)cl.block_rank() & 1;
    Fr *lo = cl.map_shared_rank(s, pair), *hi = cl.map_shared_rank(s, pair + 1);
    for (int i = threadIdx.x; i < S / 2; i += NT) {
        const int j = half * (S / 2) + i;
        const Fr x = ld_vec(&lo[j]), y = fr_mul(ld_vec(&hi[j]), ldg_vec(&roots[j * (4096 / S)]));
        st_vec(&lo[j], fr_add(x, y));
        st_vec(&hi[j], fr_sub(x, y));
    }
}
template <int S, int NT>
__device__ __forceinline__ void cluster_pair_dif(cg::cluster_group &cl, Fr *s, const Fr *__restrict__ roots) {
    const int pair = (int)cl.block_rank() & ~1, half = (int)cl.block_rank() & 1;
    Fr *lo = cl.map_shared_rank(s, pair), *hi = cl.map_shared_rank(s, pair + 1);
    for (int i = threadIdx.x; i < S / 2; i += NT) {
        const int j = half * (S / 2) + i;
        const Fr x = ld_vec(&lo[j]), y = ld_vec(&hi[j]);
        st_vec(&lo[j], fr_add(x, y));
        st_vec(&hi[j], fr_mul(fr_sub(x, y), ldg_vec(&roots[j * (4096 / S)])));
    }
}

// The last two stages of an inverse DIT of N = C S points on the elements k,
// k + N/4, k + N/2, k + 3N/4: a0..a3 in place.
template <int N>
__device__ __forceinline__ void radix4_dit_last(Fr &a0, Fr &a1, Fr &a2, Fr &a3, int k, const Fr *__restrict__ roots) {
    constexpr int st = 8192 / N;
    // length N/2: (k, k + N/4) and (k + N/2, k + 3N/4), one twiddle
    const Fr w = ldg_vec(&roots[2 * st * k]);
    Fr t = fr_mul(a1, w);
    a1 = fr_sub(a0, t);
    a0 = fr_add(a0, t);
    t = fr_mul(a3, w);
    a3 = fr_sub(a2, t);
    a2 = fr_add(a2, t);
    // length N: (k, k + N/2) and (k + N/4, k + 3N/4)
    t = fr_mul(a2, ldg_vec(&roots[st * k]));
    a2 = fr_sub(a0, t);
    a0 = fr_add(a0, t);
    t = fr_mul(a3, ldg_vec(&roots[st * (k + N / 4)]));
    a3 = fr_sub(a1, t);
    a1 = fr_add(a1, t);
}
// The first two stages of a forward DIF, likewise.
template <int N>
__device__ __forceinline__ void radix4_dif_first(Fr &a0, Fr &a1, Fr &a2, Fr &a3, int k, const Fr *__restrict__ roots) {
    constexpr int st = 8192 / N;
    Fr t = fr_sub(a0, a2);
    a0 = fr_add(a0, a2);
    a2 = fr_mul(t, ldg_vec(&roots[st * k]));
    t = fr_sub(a1, a3);
    a1 = fr_add(a1, a3);
    a3 = fr_mul(t, ldg_vec(&roots[st * (k + N / 4)]));
    const Fr v = ldg_vec(&roots[2 * st * k]);
    t = fr_sub(a0, a1);
    a0 = fr_add(a0, a1);
    a1 = fr_mul(t, v);
    t = fr_sub(a2, a3);
    a2 = fr_add(a2, a3);
    a3 = fr_mul(t, v);
}

// The outer stages of an inverse DIT, the pointwise factors shift(k), and the
// outer stages of a forward DIF, on blocks whose inner DIT stages are done; the
// inner DIF stages may follow.  Ends and begins with cluster barriers.
template <int C, int S, int NT, class Shift>
__device__ __forceinline__ void cluster_dit_shift_dif(cg::cluster_group &cl, Fr *s, const Fr *__restrict__ roots_fwd,
                                                      const Fr *__restrict__ roots_inv, Shift shift) {
    constexpr int N = C * S;
    cl.sync();
    if constexpr (C == 8) {
        cluster_pair_dit<S, NT>(cl, s, roots_inv);
        cl.sync();
    }
    const int first = (int)cl.block_rank() * (S / 4);
    for (int i = threadIdx.x; i < S / 4; i += NT) {
        const int k = first + i;
        Fr *p0 = cluster_at<S>(cl, s, k), *p1 = cluster_at<S>(cl, s, k + N / 4);
        Fr *p2 = cluster_at<S>(cl, s, k + N / 2), *p3 = cluster_at<S>(cl, s, k + 3 * N / 4);
        Fr a0 = ld_vec(p0), a1 = ld_vec(p1), a2 = ld_vec(p2), a3 = ld_vec(p3);
        radix4_dit_last<N>(a0, a1, a2, a3, k, roots_inv);
        a0 = shift(a0, k);
        a1 = shift(a1, k + N / 4);
        a2 = shift(a2, k + N / 2);
        a3 = shift(a3, k + 3 * N / 4);
        radix4_dif_first<N>(a0, a1, a2, a3, k, roots_fwd);
        st_vec(p0, a0);
        st_vec(p1, a1);
        st_vec(p2, a2);
        st_vec(p3, a3);
    }
    cl.sync();
    if constexpr (C == 8) {
        cluster_pair_dif<S, NT>(cl, s, roots_fwd);
        cl.sync();
    }
}

} // namespace vkzg
