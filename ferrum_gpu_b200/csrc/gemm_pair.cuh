// Host interface of the CTA-pair products (gemm_pair.cu).
#pragma once
#include "common.cuh"

// The exact-class product of many rows of x on the tensor cores: y = epilogue(x . W^T), x in f32 (ep.norm: the raw
// residual stream, normalised on the way), any m, k in whole blocks of 32, any n.
bool qgemm_pair_takes(const QMat& w, uint32_t m);
// Workspace of one call: the fp16 terms of x and of a slice of the weight rows, and the sums of a split of K or before an
// activation. Depends on the device only through its SM count.
size_t qgemm_pair_scratch_bytes(const FcDevice* dev, uint32_t k, uint32_t n, uint32_t m, int act);
// Whether some cut of the product fits into a workspace of `bytes`. A workspace sized for one call need not hold a call
// with fewer rows: every caller passes the size that it has, and k_qgemm_pair cuts the product to it.
bool qgemm_pair_fits(const FcDevice* dev, uint32_t k, uint32_t n, uint32_t m, int act, size_t bytes);
int k_qgemm_pair(FcDevice* dev, const QMat& w, const float* x, uint32_t m, float* y, const Epilogue& ep, const Workspace& ws);
// x[m][k] as its two fp16 terms [mp][k] (rows m.. zero), each row times a power of two that brings its largest
// magnitude to [2^14, 2^15), the low term times 2^LOW_SHIFT; x_scale[mp] takes the power of two back, or is 0 for a row
// that the terms do not hold (infinities, NaNs, small elements that count beside far larger ones).
constexpr int LOW_SHIFT = 11;
int k_rows_split(FcDevice* dev, const float* x, uint32_t m, uint32_t mp, uint32_t k, __half* xh, __half* xl, float* x_scale);
