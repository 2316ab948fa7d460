// fcm_plan.cuh -- which grids take the transforms of fcm_fft.cuh, and in which
// stages.  Host code only.
#pragma once

#include <algorithm>
#include <vector>

namespace cufil {
namespace fftk {

constexpr int kMaxStages = 10;
constexpr int kMaxLen = 1024;  // y and z: three columns blocks of 1024 points fit the shared memory

// Radices of n (forward order, largest first); empty when n has a prime factor above 5.
inline std::vector<int> radices(int n) {
    std::vector<int> r;
    for (int p : {8, 5, 4, 3, 2})
        while (n % p == 0) {
            r.push_back(p);
            n /= p;
        }
    if (n != 1 || static_cast<int>(r.size()) > kMaxStages) return {};
    return r;
}

// Lengths with their own instantiation (fcm_fft.cuh: pick_x, with half of nx, pick_y and pick_z).
inline bool fixed_length(int n) { return n == 128 || n == 256 || n == 512 || n == 1024; }

// Whether a grid takes those transforms: every axis factors into the radices, the blocks fit the shared memory, and a
// call is not slower than with the library's transforms (within 4%) even where every row is used; with few rows used it
// is faster.  Where the line lies, by 150 shapes with particles everywhere (us of a call here, by the library):
// - three grids with their spectra (24 bytes a point) must outgrow the L2 cache: below that the library's passes stay
//   in it (128^3: 198 and 185 a solve), and its inverse transform is up to 1.6e-5 off FP64 there, by which results
//   would move.  180^3 530, 601; 200^3 595, 711; 256^3 902, 896; 320^3 1721, 2296; 512^3 5775, 6189.
// - no axis above five times another: a short axis leaves a block little work between its barriers, a long row few warps
//   an SM (2048 x 64 x 64: 842, 496; 1024 x 1024 x 64: 3479, 2730; 32 x 1000 x 1000: 3413, 2021; 1000 x 200 x 200: 2272,
//   2365).  Every axis then has 60 points or more, that is two stages or more, which the kernels rely on.
// - rows of 160 or more, or all three lengths fixed (144 x 256 x 256: 676, 595; 100 x 250 x 250: 618, 522; 128 x 256 x 256
//   542, 529; 160 x 250 x 250 808, 788).
// - below 64 million points no axis that 27 divides unless 5 divides one: the library's transforms of such lengths are
//   its best (216^3: 789, 697; 128 x 243 x 243: 641, 526; 324^3: 2317, 2257; but 270^3 1361, 1456, 200 x 200 x 216 648,
//   757, 432^3 4790, 5070).
constexpr long long kMinPoints = 5500000, kManyPoints = 64000000;
inline bool supported(int nx, int ny, int nz) {
    const long long points = static_cast<long long>(nx) * ny * nz;
    if (points < kMinPoints || nx % 2 || nx > 2 * kMaxLen || ny > kMaxLen || nz > kMaxLen) return false;
    if (radices(nx / 2).empty() || radices(ny).empty() || radices(nz).empty()) return false;
    if (std::max({nx, ny, nz}) > 5 * std::min({nx, ny, nz})) return false;
    if (nx < 160 && !(fixed_length(nx) && fixed_length(ny) && fixed_length(nz))) return false;
    const bool by27 = nx % 27 == 0 || ny % 27 == 0 || nz % 27 == 0, by5 = nx % 5 == 0 || ny % 5 == 0 || nz % 5 == 0;
    return points >= kManyPoints || !by27 || by5;
}

}  // namespace fftk
}  // namespace cufil
