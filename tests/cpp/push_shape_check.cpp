// push_shape on level widths from standard input:
//   available cluster all n_levels  forward widths  backward widths
// prints the level width and the choice: clusters, warps (FP32), warps (FP64).
#include <cstdio>
#include <vector>

#include "fm_setup.hpp"

int main() {
    unsigned available = 0, cluster = 0, all = 0, n = 0;
    if (std::scanf("%u %u %u %u", &available, &cluster, &all, &n) != 4) return 1;
    std::vector<uint32_t> ptr[2];
    for (auto& p : ptr) {
        p.assign(1, 0);
        for (unsigned l = 0, w = 0; l < n; ++l) {
            if (std::scanf("%u", &w) != 1) return 1;
            p.push_back(p.back() + w);
        }
    }
    const double width = fm::level_width(ptr[0].back(), ptr[0], ptr[1]);
    const fm::PushShape s = fm::push_shape(width, available, cluster, all != 0);
    std::printf("%.17g %u %u %u\n", width, s.clusters, s.warps32, s.warps64);
    return 0;
}
