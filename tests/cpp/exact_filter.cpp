// Prints the EXACT kernel's trust in its cheap quotient (bpgb::exact_filter: the bound on its
// distance from the reference's, and whether every bin of the plan lies in [0, T)) for a
// geometry: host code, no GPU.
//
//   exact_filter <input.bin>
//
// input.bin (little endian): u32 T, u32 P, u32 N[3], f32 zero[3], f32 inc[9], f32 t0,
// f32 deltaT, then P pairs (32 bytes each).
#include <cstdint>
#include <cstdio>
#include <vector>

#include "bpgb_internal.h"

int main(int argc, char **argv) {
    FILE *f = argc > 1 ? std::fopen(argv[1], "rb") : nullptr;
    if (!f) return 2;
    uint32_t head[5];
    float geo[14];
    if (std::fread(head, 4, 5, f) != 5 || std::fread(geo, 4, 14, f) != 14) return 2;
    std::vector<bpgb_pair> pairs(head[1]);
    if (std::fread(pairs.data(), sizeof(bpgb_pair), pairs.size(), f) != pairs.size()) return 2;
    std::fclose(f);
    bpgb::Volume vol{};
    for (int k = 0; k < 3; k++) vol.n[k] = head[2 + k], vol.zero[k] = geo[k];
    for (int k = 0; k < 9; k++) vol.inc[k] = geo[3 + k];
    const bpgb::BinParams bp{geo[12], geo[13], head[0]};
    const bpgb::ExactFilter e = bpgb::exact_filter(pairs.data(), pairs.size(), vol, bp);
    std::printf("%.9g %d\n", e.error, e.inside ? 1 : 0);
    return 0;
}
