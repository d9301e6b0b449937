// Cells of a blob: the 2x Reed-Solomon extension (EIP-7594 compute_cells), the
// half of compute_cells_and_kzg_proofs the reference leaves out
// (include/vkzg.h:16-18).  Its expected output is pinned by the cells in the
// reference's test vectors (tests/vectors/compute_cells_and_kzg_proofs_*,
// spans 1..128, which tests/vectors.h:88-95 skips).
//
// Per blob, one block.  The wire order of the 8192 extended evaluations is
// bit-reversed: position p holds the value at w_8192^brev13(p), and for p < 4096
// brev13(p) = 2 brev12(p), so the first 64 cells are the blob itself (its
// element p is the value at w_4096^brev12(p)); those bytes are copied.  The
// other 64 cells are the values on the coset w_8192 D_4096: the forward NTT-4096
// of f_k w_8192^k, f the blob's coefficients from an inverse NTT-4096
// (bit-reversed evaluations -> natural coefficients, as in the proof path), and
// that DIF transform's bit-reversed output is the cells' wire order.  The
// 1/4096 scale carries an extra 1/R, so the Montgomery limbs of every output
// are its canonical value.
#include "cluster_ntt.cuh"
#include "device_util.cuh"
#include "kernels.h"

namespace vkzg {

// A blob over a cluster of C blocks (cluster_ntt.cuh).  One 512-thread block per
// blob (128 KB, radix-2 stages) kept a single SM busy: 57 k products, 0.17 ms at
// the SM's rate, whatever the batch.  Four blocks a blob, or eight up to SMs / 8
// blobs (18), the line of recovery (recover_kernels.cu).  Measured, the call on
// page-locked buffers with eight and with four: 9 blobs 154 and 169 us, 18 blobs
// 201 and 214, 24 blobs (in parts, which take eight) 229 and 240, 32 blobs 280 and
// 281, 256 blobs 1528 and 1525.
constexpr int kCellsThreads = 256;

template <int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kCellsThreads, C == 4 ? 3 : 2)
    k_blob_to_cells(const uint8_t *__restrict__ blobs, uint8_t *cells, const Fr *__restrict__ roots_fwd,
                    const Fr *__restrict__ roots_inv, Fr scale, uint32_t *err) {
    constexpr int kSeg = kBlobElems / C, kLogSeg = C == 4 ? 10 : 9;
    static_assert(kSeg == 1 << kLogSeg, "whole segments");
    extern __shared__ uint4 smem_raw[];
    Fr *s = reinterpret_cast<Fr *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int b = blockIdx.x / C, first = (int)cl.block_rank() * kSeg;
    const uint8_t *src = blobs + (size_t)b * kBlobBytes + 32 * (size_t)first;
    uint8_t *dst = cells + (size_t)b * kExtElems * 32 + 32 * (size_t)first;
    bool bad = false;
    for (int i = threadIdx.x; i < kSeg; i += kCellsThreads) {
        const uint4 *p = reinterpret_cast<const uint4 *>(src + 32 * (size_t)i);
        const uint4 lo = p[0], hi = p[1];
        uint4 *w = reinterpret_cast<uint4 *>(dst + 32 * (size_t)i); // first half of the cells: the blob
        w[0] = lo;
        w[1] = hi;
        Fr v;
        v.v[7] = bswap32(lo.x); v.v[6] = bswap32(lo.y); v.v[5] = bswap32(lo.z); v.v[4] = bswap32(lo.w);
        v.v[3] = bswap32(hi.x); v.v[2] = bswap32(hi.y); v.v[1] = bswap32(hi.z); v.v[0] = bswap32(hi.w);
        bad |= !fr_is_canonical(v);
        st_vec(&s[i], fr_from_canonical(v));
    }
    if (bad) atomicOr(&err[b], 1u);
    __syncthreads();
    smem_dit4<kCellsThreads>(s, kLogSeg, 1, 2, kSeg, roots_inv);
    // f_k w_8192^k, f scaled by 1/(4096 R)
    cluster_dit_shift_dif<C, kSeg, kCellsThreads>(cl, s, roots_fwd, roots_inv, [&](const Fr &v, int k) {
        return fr_mul(fr_mul(v, scale), ldg_vec(&roots_fwd[k]));
    });
    smem_dif4<kCellsThreads>(s, kLogSeg, 1, kSeg, 2, roots_fwd);
    for (int q = threadIdx.x; q < kSeg; q += kCellsThreads) {
        const Fr v = ld_vec(&s[q]);
        uint4 *w = reinterpret_cast<uint4 *>(dst + 32 * (size_t)(kBlobElems + q));
        w[0] = make_uint4(bswap32(v.v[7]), bswap32(v.v[6]), bswap32(v.v[5]), bswap32(v.v[4]));
        w[1] = make_uint4(bswap32(v.v[3]), bswap32(v.v[2]), bswap32(v.v[1]), bswap32(v.v[0]));
    }
}

cudaError_t launch_cells(const DeviceTables &t, const uint8_t *blobs, uint8_t *cells, uint32_t *err, int n,
                         cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    // (1/4096) / R: the canonical integer of the Montgomery constant 1/4096
    static const Fr scale = fr_to_canonical(fr_inv(fr_from_u32(kBlobElems)));
    if (8 * n <= sm_count())
        k_blob_to_cells<8><<<8 * n, kCellsThreads, kBlobElems / 8 * sizeof(Fr), s>>>(blobs, cells, t.roots_fwd,
                                                                                    t.roots_inv, scale, err);
    else
        k_blob_to_cells<4><<<4 * n, kCellsThreads, kBlobElems / 4 * sizeof(Fr), s>>>(blobs, cells, t.roots_fwd,
                                                                                    t.roots_inv, scale, err);
    count_launches(1);
    return cudaGetLastError();
}

} // namespace vkzg
