// Sizes and rules of the warm-start network's workspaces (host arithmetic
// only; no CUDA types, so that a plain C++ compiler takes it).
#pragma once
#include <cstddef>
#include <cstdint>

namespace gelios {

// ---- split of the weight GEMMs over the rows of a batch
// dW = dZ^T . H has the batch as its K: it is cut into slices whose partial
// sums are stored side by side and added in order.

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

// ---- one allocation of several workspaces
// (a cudaMalloc of 2 MB or more takes 340 us whatever its size)
struct Carve {
    size_t bytes = 0;
    size_t take(size_t n) {  // offset of the next workspace, 256-byte aligned
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    }
};

// ---- pinned staging of a network's predictions
// Rows per chunk: at most 16 MB of inputs and outputs.
inline int64_t stage_rows(int max_batch, int n_in, int n_out) {
    int64_t r = (int64_t(4) << 20) / (n_in + n_out);
    if (r < 1024) r = 1024;
    return r < max_batch ? r : max_batch;
}
// Whether it is worth its cost: `calls` predictions of io_bytes of inputs and
// outputs in all over the life of the network.  Pinning 0.8 MB (8192 rows, 7
// in, 5 out) takes 1.0-2.7 ms and 32 MB 18 ms.  A call of one row then takes 62
// us instead of 71 through the driver's own staging, one of 5400 rows (260 KB)
// 118 instead of 155, one of 86400 rows (4.1 MB) 1.13 ms instead of 1.6: 9 us a
// call and 115 a megabyte.  A network that is asked to predict once never pins.
inline bool staging_worth(int64_t calls, int64_t io_bytes, int64_t staging_bytes) {
    return 9.0 * calls + 115e-6 * io_bytes >= 1500.0 + 550e-6 * staging_bytes;
}

}  // namespace gelios
