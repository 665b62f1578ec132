// rules.h -- which form of the pair passes runs, by precision and size.  Host
// code only.
#pragma once

#include <cstddef>

namespace moldy {

// The mixed passes of large systems in lookup mode keep their tables in shared
// memory (k_screen_st, k_forces_st: one block per SM); smaller systems, whose
// atoms would fill few such blocks, and tables above kStNodes nodes read them
// through L1 with blocks of 256.  One block per SM fills late: NPT steps of L1
// forms / screening in shared memory / both (us): 101,306 atoms 59.1 / 59.0 /
// 59.0, 250,000 100 / 96 / 101, 524,288 169 / 160 / 166, 810,448 - / 225 / 230,
// 913,066 - / 242 / 239, 1,024,000 276 / 260 / 254, 2,000,000 499 / 459 / 444.
// So the screening pass takes it from 100,000 atoms on and the force pass from
// 850,000, whatever the variant: a variant chosen or tuned is one of the form
// that is the faster at its size.
constexpr int kStAtoms = 100000;         // screening-density pass
constexpr int kStForceAtoms = 850000;    // force pass
constexpr int kStNodes = 6000;           // 24 bytes per node: 144 KB beside 48 bytes per thread

constexpr bool screen_in_smem(int nm, int nodes, int mid_cap, int pair_cap) {
    // 32-bit row offsets
    return nm >= kStAtoms && nodes <= kStNodes &&
           nm * ((long long)(mid_cap > pair_cap ? mid_cap : pair_cap) + 16) < (1LL << 32);
}

constexpr bool forces_in_smem(int nm, int nodes, int mid_cap, int pair_cap) {
    return nm >= kStForceAtoms && screen_in_smem(nm, nodes, mid_cap, pair_cap);
}

}  // namespace moldy
