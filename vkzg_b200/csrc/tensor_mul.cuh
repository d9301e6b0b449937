// Fp products whose Montgomery reduction runs on the tensor cores.
//
// T / R mod p is linear in the bytes of T, so for 128 threads at once it is one
// matrix product: row i of a constant matrix holds the 48 bytes of
// 2^(8 i) 2^32 / R mod p, the threads' bytes are the other operand (u8 x u8 into
// 32-bit sums, exact), and the sums come back as 48 columns of weight 2^(8 k).
// They add up to S = 2^32 T / R mod p with S < 144 * 255 * p, and one word-wise
// step, (S + m p) / 2^32, leaves T / R mod p below p + 2^365.
//
// The map being linear, the product is never put together: one Karatsuba level
// splits a = a0 + a1 2^191 (so that a0 + a1 still fits six words),
//   a b = z0 (1 - 2^191) + z2 (2^382 - 2^191) + zm 2^191,
//   z0 = a0 b0, z2 = a1 b1, zm = (a0 + a1)(b0 + b1),
// and the three 12-word products go to the tensor core as they are, with the
// factors in parentheses folded into their rows of the matrix: 108 word
// products and no recombination.
//
// What bounds it: issue slots.  A fused wide multiply-add holds a scheduler
// about four cycles and every other instruction one; the word-serial form spends
// 264 of the former per product, this one 120.  Measured on B200, two blocks of 256
// threads per SM (vkzg_b200_microbench 18 to 21, 4 and 6): products 42.2 G/s one after
// another and 45.0 in the pipeline below, against 29.2 for the scalar form; squares
// 48.9 and 53.7 against 33.7.  The matrix
// product takes 48 cycles of an SM per step of 32 rows.  Tried and slower: the
// reduction through mma.sync (26.8 G/s), products of 24-bit limbs on the FP64 pipe
// (25.9) or of 30-bit limbs without carries (29.8) in front of the same reduction.
#pragma once

#include "field.cuh"
#if defined(__CUDACC__)
#include "device_util.cuh"
#endif

namespace vkzg {

constexpr int kTmWords = 36;            // words of z0, z2, zm
constexpr int kTmRows = 4 * kTmWords;   // matrix rows in use
constexpr int kTmRowsPad = 160;         // padded to whole steps of 32 rows
constexpr int kTmCols = 48;             // result columns

struct TmMatrix {
    uint8_t b[kTmRows][kTmCols];
};

// ---- the matrix, at compile time
struct TmFp {
    uint32_t v[12];
};
constexpr TmFp tm_half(TmFp x) { // x / 2 mod p
    uint32_t top = 0;
    if (x.v[0] & 1u) {
        uint64_t t = 0;
        for (int i = 0; i < 12; i++) {
            t += (uint64_t)x.v[i] + fp_p(i);
            x.v[i] = (uint32_t)t;
            t >>= 32;
        }
        top = (uint32_t)t;
    }
    for (int i = 0; i < 12; i++) x.v[i] = (x.v[i] >> 1) | ((i < 11 ? x.v[i + 1] : top) << 31);
    return x;
}
constexpr TmFp tm_sub(TmFp x, TmFp y) { // x - y mod p
    uint64_t b = 0;
    for (int i = 0; i < 12; i++) {
        const uint64_t d = (uint64_t)x.v[i] - y.v[i] - b;
        x.v[i] = (uint32_t)d;
        b = (d >> 32) & 1u;
    }
    if (b) {
        uint64_t t = 0;
        for (int i = 0; i < 12; i++) {
            t += (uint64_t)x.v[i] + fp_p(i);
            x.v[i] = (uint32_t)t;
            t >>= 32;
        }
    }
    return x;
}
constexpr TmFp tm_dbl(TmFp x) { // 2 x mod p
    TmFp y{};
    uint32_t c = 0;
    for (int i = 0; i < 12; i++) {
        y.v[i] = (x.v[i] << 1) | c;
        c = x.v[i] >> 31;
    }
    TmFp s{};
    uint64_t b = 0;
    for (int i = 0; i < 12; i++) {
        const uint64_t d = (uint64_t)y.v[i] - fp_p(i) - b;
        s.v[i] = (uint32_t)d;
        b = (d >> 32) & 1u;
    }
    return b ? y : s;
}
constexpr TmMatrix tm_matrix() {
    TmMatrix m{};
    TmFp e0{}; // 2^32 / R
    e0.v[0] = 1;
    for (int e = 0; e < 352; e++) e0 = tm_half(e0);
    TmFp e191 = e0, e382 = e0;
    for (int e = 0; e < 191; e++) e191 = tm_dbl(e191);
    e382 = e191;
    for (int e = 0; e < 191; e++) e382 = tm_dbl(e382);
    const TmFp first[3] = {tm_sub(e0, e191), tm_sub(e382, e191), e191};
    for (int z = 0; z < 3; z++) {
        TmFp x = first[z];
        for (int i = 0; i < kTmCols; i++) {
            for (int k = 0; k < kTmCols; k++) m.b[z * kTmCols + i][k] = (uint8_t)(x.v[k / 4] >> (8 * (k & 3)));
            for (int h = 0; h < 8; h++) x = tm_dbl(x);
        }
    }
    return m;
}

// ---- an operand's Karatsuba parts: low 191 bits, the rest, and their sum.
// a < 2^382 (any value below 2p is).
struct TmPart {
    uint32_t lo[6], hi[6], sum[6];
};
VK_HD uint32_t tm_funnel(uint32_t lo, uint32_t hi, int s) { // bits [s, s + 32) of hi:lo
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
#endif
}
VK_HD TmPart tm_part(const uint32_t *a) {
    CARRY_DECL
    TmPart r;
#pragma unroll
    for (int i = 0; i < 5; i++) r.lo[i] = a[i];
    r.lo[5] = a[5] & 0x7fffffffu;
#pragma unroll
    for (int i = 0; i < 6; i++) r.hi[i] = tm_funnel(a[5 + i], a[6 + i], 31);
    ADD_CC(r.sum[0], r.lo[0], r.hi[0]);
#pragma unroll
    for (int i = 1; i < 5; i++) ADDC_CC(r.sum[i], r.lo[i], r.hi[i]);
    ADDC(r.sum[5], r.lo[5], r.hi[5]);
    return r;
}

// r = (S + m p) / 2^32 for S = sum_k w[k] 2^(16 k) < 2^396, m = -S / p mod 2^32.
// The even w (word-aligned) and the odd ones (half a word up) are kept as two
// numbers, which take the even and the odd products of m p: each array's wide
// multiply-adds fall on its own aligned register pairs, and one addition at the
// end joins them.
VK_HD void tm_join(uint32_t *r, const uint32_t *w) {
    CARRY_DECL
    uint32_t e[13], o[13];
#pragma unroll
    for (int k = 0; k < 12; k++) {
        e[k] = w[2 * k];
        o[k] = k ? tm_funnel(w[2 * k - 1], w[2 * k + 1], 16) : w[1] << 16;
    }
    o[12] = w[23] >> 16;
    ADD_CC(e[0], e[0], o[0]);
    const uint32_t m = e[0] * VK_FP_N0;
    MADC_LO_CC(o[1], m, fp_p(1), o[1]);
    MADC_HI_CC(o[2], m, fp_p(1), o[2]);
#pragma unroll
    for (int j = 3; j < 11; j += 2) {
        MADC_LO_CC(o[j], m, fp_p(j), o[j]);
        MADC_HI_CC(o[j + 1], m, fp_p(j), o[j + 1]);
    }
    MADC_LO_CC(o[11], m, fp_p(11), o[11]);
    MADC_HI(o[12], m, fp_p(11), o[12]);
    MAD_LO_CC(e[0], m, fp_p(0), e[0]);
    MADC_HI_CC(e[1], m, fp_p(0), e[1]);
#pragma unroll
    for (int j = 2; j < 12; j += 2) {
        MADC_LO_CC(e[j], m, fp_p(j), e[j]);
        MADC_HI_CC(e[j + 1], m, fp_p(j), e[j + 1]);
    }
    ADDC(e[12], 0u, 0u);
    ADD_CC(r[0], e[1], o[1]);
#pragma unroll
    for (int k = 1; k < 11; k++) ADDC_CC(r[k], e[k + 1], o[k + 1]);
    ADDC(r[11], e[12], o[12]);
}

// The matrix as it lies in shared memory: K-major core matrices of eight columns
// by 16 rows, [row / 16][column][row % 16], the padding rows zero.
struct alignas(16) TmImage {
    uint8_t b[kTmRowsPad * kTmCols];
};
constexpr TmImage tm_image() {
    const TmMatrix m = tm_matrix();
    TmImage im{};
    for (int row = 0; row < kTmRows; row++)
        for (int col = 0; col < kTmCols; col++) im.b[(row / 16 * kTmCols + col) * 16 + row % 16] = m.b[row][col];
    return im;
}

#if defined(__CUDACC__)
// ---- device side: groups of 128 threads (four warps, one row of the matrix
// product each) share a block's copy of the constant matrix.
constexpr int kTmGroup = 128;
// TMEM columns of a group: two areas for a product's bytes (one filled while the
// tensor core reads the other), then the sums
constexpr int kTmTmemCols = 128;
constexpr int kTmBytes = kTmRowsPad / 4;
constexpr int kTmSums = 2 * kTmBytes;
static_assert(kTmSums + kTmCols <= kTmTmemCols, "the areas fit a group's columns");
constexpr int kTmMatrixBytes = kTmRowsPad * kTmCols;
// a block's shared memory: the matrix, then one mbarrier per group (at most
// kTmMaxGroups) and one for tm_drain, the TMEM address, the flag that a wait gave
// up, and one count of arrived warps per group
constexpr int kTmMaxGroups = 2;
constexpr int kTmDrain = kTmMatrixBytes + 8 * kTmMaxGroups;
constexpr int kTmWords0 = kTmDrain + 8; // the TMEM address, then the flag
constexpr int kTmCounts = kTmWords0 + 8;
constexpr int kTmSmem = kTmCounts + 4 * kTmMaxGroups;
static_assert(kTmGroup == 128, "a count of four warps per product");
// polls of a wait for the tensor core (each suspends up to kTmPollNs) before it gives up
constexpr uint32_t kTmPolls = 20000, kTmPollNs = 2000;

__device__ const TmImage d_tm_image = tm_image();

struct Tm {
    uint32_t t;  // the warp's TMEM address
    uint32_t sm; // shared address of the block's area (128-byte aligned); bit 0: the
                 // mbarrier's phase, bit 1: the byte area of the next product
};
constexpr uint32_t kTmFlags = 3u;

__device__ __forceinline__ uint32_t tm_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Block set-up (all threads): the matrix, the mbarriers, TMEM for the block's
// groups.  area: kTmSmem bytes of shared memory, 128-byte aligned.
__device__ __forceinline__ Tm tm_begin(uint8_t *area) {
    const uint4 *im = reinterpret_cast<const uint4 *>(d_tm_image.b);
    for (int x = threadIdx.x; x < kTmMatrixBytes / 16; x += blockDim.x)
        reinterpret_cast<uint4 *>(area)[x] = __ldg(&im[x]);
    const uint32_t bars = tm_smem(area) + kTmMatrixBytes;
    uint32_t *word = reinterpret_cast<uint32_t *>(area + kTmWords0);
    if (threadIdx.x <= kTmMaxGroups) // tm_drain's takes an arrival from every warp
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8 * threadIdx.x),
                     "r"(threadIdx.x < kTmMaxGroups ? 1u : blockDim.x / 32)
                     : "memory");
    if (threadIdx.x <= kTmMaxGroups) word[1 + threadIdx.x] = 0; // the flag, the counts
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tm_smem(word)),
                     "n"(kTmMaxGroups * kTmTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    Tm g;
    g.t = *reinterpret_cast<volatile uint32_t *>(word) + (threadIdx.x / kTmGroup) * kTmTmemCols +
          ((threadIdx.x & 96u) << 16);
    g.sm = tm_smem(area);
    return g;
}

// After a wait gave up (all threads): waits, bounded like every wait, until no
// product that the block started is in flight any more, so that none reads TMEM or
// signals an mbarrier that the block no longer owns.  Each warp's first lane, which
// started that warp's products, commits them to one mbarrier.
static __device__ __noinline__ void tm_drain(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                     : "memory");
    uint32_t ok = 0;
    for (uint32_t polls = 0; !ok && polls <= kTmPolls; polls++)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0, %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "n"(kTmPollNs)
                     : "memory");
    __syncwarp();
}

// End of the block's products (all threads): frees the TMEM; if a wait gave up,
// waits for the products in flight first and marks the launch's error words like a
// grid barrier does.
__device__ __forceinline__ void tm_end(uint8_t *area, uint32_t *err, uint32_t n_err) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    volatile uint32_t *word = reinterpret_cast<volatile uint32_t *>(area + kTmWords0);
    const bool gave_up = word[1] != 0;
    if (gave_up) {
        tm_drain(tm_smem(area) + kTmDrain);
        __syncthreads();
    }
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(word[0]),
                     "n"(kTmMaxGroups * kTmTmemCols));
    if (gave_up)
        for (uint32_t b = threadIdx.x; b < n_err; b += blockDim.x) atomicOr(&err[b], kSyncFailed);
}

// 12 words of this thread's row to TMEM
__device__ __forceinline__ void tm_put(uint32_t t, const uint32_t *z) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t), "r"(z[0]),
                 "r"(z[1]), "r"(z[2]), "r"(z[3]), "r"(z[4]), "r"(z[5]), "r"(z[6]), "r"(z[7])
                 : "memory");
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t + 8), "r"(z[8]), "r"(z[9]),
                 "r"(z[10]), "r"(z[11])
                 : "memory");
}

// Starts the group's matrix product over the bytes put, once every warp of the
// group has put its rows and read the sums of the product before: each warp
// counts itself in and goes on, and the one that completes the count issues the
// product.  (A barrier of the group in its place is faster when warps do nothing
// but push, 47.3 against 44.9 G products/s; in the passes, whose warps drift apart
// over loads, it is slower: 20.98 against 20.52 ms for the proofs of 256 blobs.)
// Called by whole groups, as is everything below.
__device__ __forceinline__ void tm_start(uint32_t t, uint32_t ctl) {
    const uint32_t sm = ctl & ~kTmFlags, grp = threadIdx.x / kTmGroup;
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    uint32_t in = 0;
    if ((threadIdx.x & 31) == 0)
        asm volatile("atom.acq_rel.cta.shared.add.u32 %0, [%1], 1;"
                     : "=r"(in)
                     : "r"(sm + kTmCounts + 4 * grp)
                     : "memory");
    if ((threadIdx.x & 31) == 0 && (in & 3u) == 3u) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // S32 sums, U8 x U8, both K-major, 128 x kTmCols x 32 a step
        constexpr uint32_t idesc = (2u << 4) | ((kTmCols / 8) << 17) | ((kTmGroup / 16) << 24);
        // no swizzle: core matrices kTmCols * 16 bytes apart along K, 128 along N
        const uint64_t desc = (uint64_t)(sm >> 4) | ((uint64_t)kTmCols << 16) | ((uint64_t)8 << 32) | (1ull << 46);
        const uint32_t base = t & 0xffffu, bytes = base + (ctl & 2u) / 2 * kTmBytes;
#pragma unroll
        for (int s = 0; s < kTmRowsPad / 32; s++)
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                         "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(base + kTmSums),
                         "r"(bytes + 8 * s), "l"(desc + (uint64_t)(2 * kTmCols * s)), "r"(idesc), "r"(s)
                         : "memory");
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         sm + kTmMatrixBytes + 8 * grp)
                     : "memory");
    }
    __syncwarp();
}

// Waits for the matrix product started last and reads the sums of this thread's
// row: columns joined in pairs (weight 2^(16 k); each below 144 * 255^2 * 257 < 2^32).
__device__ __forceinline__ void tm_sums(uint32_t t, uint32_t ctl, uint32_t *w) {
    const uint32_t sm = ctl & ~kTmFlags, phase = ctl & 1u, grp = threadIdx.x / kTmGroup;
    const uint32_t bar = sm + kTmMatrixBytes + 8 * grp;
    uint32_t ok = 0, polls = 0;
    do {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(phase), "n"(kTmPollNs)
                     : "memory");
        if (!ok) { // bounded: after kTmPolls the block's flag is set and no wait of the block polls again
            uint32_t gave_up;
            const uint32_t flag = sm + kTmWords0 + 4;
            asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(flag) : "memory");
            if (gave_up) break;
            if (++polls > kTmPolls) asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(flag), "r"(1u) : "memory");
        }
    } while (!ok);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t c[kTmCols];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%48];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, "
        "%45, %46, %47}, [%49];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7]), "=r"(c[8]),
          "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]), "=r"(c[14]), "=r"(c[15]), "=r"(c[16]),
          "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]), "=r"(c[21]), "=r"(c[22]), "=r"(c[23]), "=r"(c[24]),
          "=r"(c[25]), "=r"(c[26]), "=r"(c[27]), "=r"(c[28]), "=r"(c[29]), "=r"(c[30]), "=r"(c[31]), "=r"(c[32]),
          "=r"(c[33]), "=r"(c[34]), "=r"(c[35]), "=r"(c[36]), "=r"(c[37]), "=r"(c[38]), "=r"(c[39]), "=r"(c[40]),
          "=r"(c[41]), "=r"(c[42]), "=r"(c[43]), "=r"(c[44]), "=r"(c[45]), "=r"(c[46]), "=r"(c[47])
        : "r"(t + kTmSums), "r"(t + kTmSums + 32)
        : "memory");
#pragma unroll
    for (int k = 0; k < kTmCols / 2; k++) w[k] = c[2 * k] + (c[2 * k + 1] << 8);
}

// The product, in [0, p + 2^365) for operands below 2^382.
__device__ __forceinline__ Fp tm_result(const uint32_t *w) {
    Fp r;
    tm_join(r.v, w);
    return r;
}
// a value below 2p in [0, p)
__device__ __forceinline__ Fp tm_canonical(const Fp &a) {
    CARRY_DECL
    Fp r;
    uint32_t s[12], borrow;
    SUB_CC(s[0], a.v[0], fp_p(0));
#pragma unroll
    for (int i = 1; i < 12; i++) SUBC_CC(s[i], a.v[i], fp_p(i));
    SUBC(borrow, 0u, 0u);
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = borrow ? a.v[i] : s[i];
    return r;
}
template <bool CANON>
__device__ __forceinline__ Fp tm_canonical_if(const Fp &a) {
    if constexpr (CANON) return tm_canonical(a);
    else return a;
}

// the three Karatsuba products of a b, or of a^2, to the product's byte area
__device__ __forceinline__ void tm_put_mul(const Fp &a, const Fp &b, uint32_t t, uint32_t ctl) {
    t += (ctl & 2u) / 2 * kTmBytes;
    const TmPart x = tm_part(a.v), y = tm_part(b.v);
    uint32_t z[12];
    mul_words<6>(z, x.lo, y.lo);
    tm_put(t, z);
    mul_words<6>(z, x.hi, y.hi);
    tm_put(t + 12, z);
    mul_words<6>(z, x.sum, y.sum);
    tm_put(t + 24, z);
}
__device__ __forceinline__ void tm_put_sqr(const Fp &a, uint32_t t, uint32_t ctl) {
    t += (ctl & 2u) / 2 * kTmBytes;
    const TmPart x = tm_part(a.v);
    uint32_t z[12];
    sqr_words<6>(z, x.lo);
    tm_put(t, z);
    sqr_words<6>(z, x.hi);
    tm_put(t + 12, z);
    sqr_words<6>(z, x.sum);
    tm_put(t + 24, z);
}
static __device__ __noinline__ Fp tm_mul_call(Fp a, Fp b, uint32_t t, uint32_t ctl) {
    tm_put_mul(a, b, t, ctl);
    tm_start(t, ctl);
    uint32_t w[kTmCols / 2];
    tm_sums(t, ctl, w);
    return tm_result(w);
}
static __device__ __noinline__ Fp tm_sqr_call(Fp a, uint32_t t, uint32_t ctl) {
    tm_put_sqr(a, t, ctl);
    tm_start(t, ctl);
    uint32_t w[kTmCols / 2];
    tm_sums(t, ctl, w);
    return tm_result(w);
}
static __device__ __noinline__ void tm_push_first_call(Fp a, Fp b, uint32_t t, uint32_t ctl) {
    tm_put_mul(a, b, t, ctl);
    tm_start(t, ctl);
}
static __device__ __noinline__ Fp tm_push_mul_call(Fp a, Fp b, uint32_t t, uint32_t ctl) {
    tm_put_mul(a, b, t, ctl);
    uint32_t w[kTmCols / 2];
    tm_sums(t, ctl, w);
    tm_start(t, ctl);
    return tm_result(w);
}
static __device__ __noinline__ Fp tm_push_sqr_call(Fp a, uint32_t t, uint32_t ctl) {
    tm_put_sqr(a, t, ctl);
    uint32_t w[kTmCols / 2];
    tm_sums(t, ctl, w);
    tm_start(t, ctl);
    return tm_result(w);
}
static __device__ __noinline__ Fp tm_pop_call(uint32_t t, uint32_t ctl) {
    uint32_t w[kTmCols / 2];
    tm_sums(t, ctl, w);
    return tm_result(w);
}

// a b and a^2, called by every thread of a group together (none in flight)
template <bool CANON>
__device__ __forceinline__ Fp tm_mul(Tm &g, const Fp &a, const Fp &b) {
    __syncwarp();
    const Fp r = tm_mul_call(a, b, g.t, g.sm);
    g.sm ^= 1u;
    return tm_canonical_if<CANON>(r);
}
template <bool CANON>
__device__ __forceinline__ Fp tm_sqr(Tm &g, const Fp &a) {
    __syncwarp();
    const Fp r = tm_sqr_call(a, g.t, g.sm);
    g.sm ^= 1u;
    return tm_canonical_if<CANON>(r);
}

// The same products in a pipeline of depth one: a push starts a product and
// returns the one pushed before it, whose trip through the tensor core has run
// while the new one's words were multiplied; CANON speaks of the one returned.
// tm_push_first starts the pipeline, tm_pop ends it.
__device__ __forceinline__ void tm_push_first(Tm &g, const Fp &a, const Fp &b) {
    __syncwarp();
    tm_push_first_call(a, b, g.t, g.sm);
    g.sm ^= 2u;
}
template <bool CANON>
__device__ __forceinline__ Fp tm_push(Tm &g, const Fp &a, const Fp &b) {
    __syncwarp();
    const Fp r = tm_push_mul_call(a, b, g.t, g.sm);
    g.sm ^= 3u;
    return tm_canonical_if<CANON>(r);
}
template <bool CANON>
__device__ __forceinline__ Fp tm_push_sqr(Tm &g, const Fp &a) {
    __syncwarp();
    const Fp r = tm_push_sqr_call(a, g.t, g.sm);
    g.sm ^= 3u;
    return tm_canonical_if<CANON>(r);
}
template <bool CANON>
__device__ __forceinline__ Fp tm_pop(Tm &g) {
    __syncwarp();
    const Fp r = tm_pop_call(g.t, g.sm);
    g.sm ^= 1u;
    return tm_canonical_if<CANON>(r);
}

// the same products by the scalar multiplier, for kernels that take either
struct ScalarMul {
    Fp last; // the product pushed last
};
template <bool CANON>
__device__ __forceinline__ Fp tm_mul(ScalarMul &, const Fp &a, const Fp &b) {
    return fp_mul(a, b);
}
template <bool CANON>
__device__ __forceinline__ Fp tm_sqr(ScalarMul &, const Fp &a) {
    return fp_sqr(a);
}
__device__ __forceinline__ void tm_push_first(ScalarMul &g, const Fp &a, const Fp &b) { g.last = fp_mul(a, b); }
template <bool CANON>
__device__ __forceinline__ Fp tm_push(ScalarMul &g, const Fp &a, const Fp &b) {
    const Fp r = g.last;
    g.last = fp_mul(a, b);
    return r;
}
template <bool CANON>
__device__ __forceinline__ Fp tm_push_sqr(ScalarMul &g, const Fp &a) {
    const Fp r = g.last;
    g.last = fp_sqr(a);
    return r;
}
template <bool CANON>
__device__ __forceinline__ Fp tm_pop(ScalarMul &g) {
    return g.last;
}
#endif

} // namespace vkzg
