// How a batch of plain instances runs (host arithmetic only; no CUDA types, so
// that a plain C++ compiler takes it).
#pragma once
#include <cstdint>

namespace gelios {

// A batch of n instances takes them one after the other, each on the whole
// chip (launch_stationary_persistent), instead of a cluster of `size` blocks
// per instance, where n steps of the one take no longer than a step of the
// other.  us per step, fitted to 40-step calls of 5k to 144k cells:
//   whole chip, lanes       4.7 + 0.055 per 1000 cells (5.4k 5.0, 21.6k 5.9)
//   whole chip, two phases  7.5 + 0.165 per 1000 cells (23.8k 11.3, 38.4k 13.9,
//                           86.4k 22.7, 144k 31.1)
//   clusters                8 + 43 per 1000 cells of a block, 31 where every
//                           block has an SM for itself (seven clusters of 16)
// us of 40 steps, one after the other against clusters: 90x60 cells, 2, 3
// instances 398 / 686, 597 / 756; 180x120, 8, 10, 12: 1881 / 2475, 2354 / 2722,
// 2825 / 2920; 186x128, 2, 4, 8: 920 / 1741, 1801 / 1820, 3596 / 2620; 240x160,
// 6, 12: 3346 / 3439, 6703 / 4820; 360x240, 8, 12, 16, 20, 29: 7241 / 9592,
// 10887 / 9879, 14527 / 18614, 18097 / 18512, 26256 / 20184.
inline bool plain_serial_faster(int64_t n_cells, int n, bool lanes, int size) {
    const double k = static_cast<double>(n_cells) / 1000.0;
    const double serial = n * (lanes ? 4.7 + 0.055 * k : 7.5 + 0.165 * k);
    const double cluster = 8.0 + (size >= 16 && n <= 7 ? 31.0 : 43.0) * k / size;
    return serial <= cluster;
}

}  // namespace gelios
