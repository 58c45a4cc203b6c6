// Internal interface of the tensor-core GEMM (gemm.cu) for the other translation units.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace tb {

// A packed operand: [128-row block][32-wide k block][plane][128 rows][32 k], 16-bit elements
// (data_bytes).  fp32 sources (`scaled`) become two planes, fp16 hi / lo of the value times a
// per-row power of two; their tiles are followed by one 32-bit word per packed row, the bit
// pattern of the row's largest magnitude, which fixes that scale.
struct Packed {
    uint32_t rowblocks, kblocks, npl;
    bool scaled;
    size_t data_bytes, bytes;
};
inline uint32_t* packed_amax(const uint16_t* packed, const Packed& g) {
    return reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(const_cast<uint16_t*>(packed)) + g.data_bytes);
}

Packed packed_geometry(int dtype, int64_t rows, int64_t K);

// Packs `rows` x `K` operand elements from a row-major source (transposed when `trans`).  `beside`: on half of the SMs,
// where the stream of an inverse waits for the others.
int launch_pack(const void* src, int dtype, bool trans, uint64_t rows, uint64_t K, uint64_t ld,
                uint16_t* packed, const Packed& g, int sm_count, cudaStream_t stream, bool beside = false);

// The same for two fp32 operands in one launch (neither transposed).
int launch_pack_pair(const float* a, uint64_t rows_a, uint64_t K_a, uint64_t ld_a, uint16_t* packed_a, const Packed& ga,
                     const float* b, uint64_t rows_b, uint64_t K_b, uint64_t ld_b, uint16_t* packed_b, const Packed& gb,
                     int sm_count, cudaStream_t stream);

// The packed operand without its first `skip` row blocks: moves `packed` and returns the geometry of what is left.
Packed packed_tail(const uint16_t** packed, const Packed& g, uint32_t skip);

// How launch_gemm computes a product: CTA tile (2: 256 columns, 1: 128; as many rows, 128 where chunked), slices of the contraction, and the bytes
// of the slices' partial products, which the caller provides as `partial`.
struct GemmPlan {
    int tile;
    uint32_t splits, kb_per_split;
    size_t partial_bytes;
};
GemmPlan plan_gemm(uint32_t npl, bool chunked, bool symmetric, int64_t M, int64_t N, uint32_t kblocks);

// Which k of a product are known to be zero in one of its operands, so that a tile's contraction leaves them out
// (chunked products only).  m and n are rows of A and of B.
enum KRange : int {
    K_ALL,
    K_FROM_ROW,  // A[m][k] = 0 for k < m; symmetric: also for k < n
    K_TO_ROW,    // A[m][k] = 0 for k > m
    K_TO_COL,    // B[n][k] = 0 for k > n
};

// C[M x N] (+)= alpha * row_scale[m] * Apacked . Bpacked^T  (symmetric: A == B, mirrored stores;
// chunked: scaled fp32 operands only -- the tensor core accumulates 64 k at a time and the chunks are
// summed with rounded fp32 adds, for products whose error an inverse will amplify).  `early`: see launch_after; not where
// another stream waits for the SMs that the launch would hold.
int launch_gemm(int device, cudaStream_t stream, const uint16_t* pa, const Packed& ga, const uint16_t* pb,
                const Packed& gb, int dtype, int64_t M, int64_t N, float* C, int64_t ldc,
                const float* row_scale, float alpha, int accumulate, int symmetric, int chunked, float* partial,
                KRange range = K_ALL, bool early = true);

}  // namespace tb
