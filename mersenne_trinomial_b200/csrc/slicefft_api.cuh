// slicefft_api.cuh -- the bit-sliced product transform (slicefft.cu).
// Transform buffers hold 2^m words, 16-byte aligned, strides even; between
// slice_fwd and slice_inv their contents mean something to slice_pointwise
// only.
#pragma once

#include "gf2e_internal.cuh"

namespace gf2e {

constexpr int SLICE_MIN_M = 10, SLICE_MAX_M = 24;
// products keep 2^(m-16) <= 128 rows of the Taylor levels above 2^16 in a
// warp's registers
constexpr int SLICE_PRODUCT_MAX_M = 23;
constexpr int SLICE_SMALL_MAX_M = 14;        // whole products in one cluster of blocks

// operand i of a batch: nchunks 32-bit chunks from src + i * stride, chunk 0
// XORed with xor0; its transform goes to f + i * fstride words
struct SliceOp {
    const u32 *src;
    u64 stride, nchunks;
    u32 xor0;
    u64 *f;
};

// forward transforms of one or two operands, `batch` of each
int slice_fwd(int m, const SliceOp *ops, int nops, u64 fstride, int batch, cudaStream_t st);
// o = x1 y1 (+ x2 y2 unless null), n words each of `batch` transforms
int slice_pointwise(u64 *o, const u64 *x1, const u64 *y1, const u64 *x2, const u64 *y2, u64 n,
                    u64 fstride, int batch, cudaStream_t st);
// inverse transform of f (tmp: as large, used for m > 16) and overlap-add of
// its coefficients into out + i * ostride, ow words each
int slice_inv(int m, u64 *f, u64 *tmp, u64 fstride, int batch, u64 *out, u64 ostride, u64 ow,
              cudaStream_t st);
// out = x y, whole products of at most 2^m coefficients (10 <= m <= 14)
int slice_small(int m, const SliceOp &x, const SliceOp &y, int batch, u64 *out, u64 ostride,
                u64 ow, cudaStream_t st);
// the transform itself in place on 2^m words (16-byte aligned) in natural
// order, but for the Taylor levels above 2^16, which the caller runs on the
// words before (forward) or after it
int slice_transform(int m, bool forward, u64 *f, cudaStream_t st);
int slice_transform_passes(int m);
// the tower images of the Cantor basis agree with the basis itself
bool slice_selfcheck(const u64 *basis);

}  // namespace gf2e
