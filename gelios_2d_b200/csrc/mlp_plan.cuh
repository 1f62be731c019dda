// Split of the warm-start network's weight GEMMs over the rows of a batch
// (host arithmetic only; no CUDA types, so that a plain C++ compiler takes it).
//
// dW = dZ^T . H has the batch as its K: it is cut into slices whose partial
// sums are stored side by side and added in order.
#pragma once

namespace gelios {

constexpr int kGemmBK = 64;    // K stage of the GEMM kernels: a slice is a multiple of it
constexpr int kMaxSplit = 32;  // most slices of a weight GEMM

// K slice of a GEMM split `splits` ways
inline int tc_split_len(int K, int splits) {
    const int kc = (K + splits - 1) / splits;
    return kc > 0 ? (kc + kGemmBK - 1) / kGemmBK * kGemmBK : kGemmBK;
}
inline int split_count(int K, int kc) { return K > 0 ? (K + kc - 1) / kc : 1; }

// slices asked for of M rows: 256 rows each, at most kMaxSplit
inline int split_target(int M) {
    const int s = (M + 255) / 256;
    return s > kMaxSplit ? kMaxSplit : s < 1 ? 1 : s;
}
// slices of M rows
inline int splits_of(int M) { return split_count(M, tc_split_len(M, split_target(M))); }

// Slices a workspace that serves every batch of 1..max_batch rows holds.  Not
// splits_of(max_batch): rounding a slice up to the K stage makes that fall
// again as M grows (26 slices of 8193 rows, 32 of 8192).  splits_of(M) is at
// most split_target(M), which does not fall.
inline int reserved_splits(int max_batch) { return split_target(max_batch); }

}  // namespace gelios
