// Dynamic shared memory limits that the launchers set, against a fake runtime
// (fake_cudart.hpp).  The limit belongs to the kernel and the device, not to
// the call: two threads that launch the same kernel in different sizes may
// interleave as limit(large), limit(small), launch(large).  Every call must
// therefore set the same limit, one that covers all sizes the kernel takes,
// and report it when the runtime refuses the limit or the launch.
#include "fake_cudart.hpp"

#include <algorithm>
#include <cstdio>

#include "fm_kernels.hpp"

static int bad = 0;
#define EXPECT(c, ...)                                       \
    do {                                                     \
        if (!(c)) {                                          \
            ++bad;                                           \
            std::printf("%s:%d: ", __FILE__, __LINE__);      \
            std::printf(__VA_ARGS__);                        \
            std::printf("\n");                               \
        }                                                    \
    } while (0)

static std::map<std::string, size_t> most;  // largest launch per kernel

template <typename T>
static void products() {
    for (uint32_t deg = 1; deg <= 32; ++deg)
        for (uint32_t nn : {1u, 16u, 17u, 100000u})
            fm::launch_spmv_nodes<T>(nn, deg, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                     nullptr, nullptr, nullptr, nullptr);
}

int main() {
    fake::on_launch = [](const fake::Launch& l) {
        most[l.kernel] = std::max(most[l.kernel], l.smem);
        return cudaSuccess;
    };
    products<double>();
    products<float>();
    for (uint32_t n : {1u, 40u, 600u, 5000u, 20000u, 27000u})
        for (uint32_t entries : {2u, 4u, 8u})
            for (uint32_t width : {1u, 33u, 600u, 5000u}) {
                fm::SmallTri L, U;
                L.n_levels = U.n_levels = std::max(1u, n / width);
                if (fm::small_tri_smem(n, L.n_levels, U.n_levels) > fm::kSmallMaxSmem) continue;
                fm::launch_trsv_small(L, U, n, entries, std::min(n, width), nullptr, nullptr,
                                      nullptr, nullptr);
            }
    EXPECT(most.size() >= 7, "only %zu kernels were launched", most.size());
    for (const auto& m : most) {
        const auto& lim = fake::smem_limit[m.first];
        EXPECT(lim.size() <= 1, "%s: %zu different limits", m.first.c_str(), lim.size());
        EXPECT(m.second <= 48 * 1024 || (!lim.empty() && m.second <= (size_t)*lim.begin()),
               "%s: a launch of %zu bytes beyond its limit", m.first.c_str(), m.second);
        EXPECT(m.second <= 227 * 1024, "%s: %zu bytes", m.first.c_str(), m.second);
    }
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
