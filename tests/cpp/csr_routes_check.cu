// Which kernels the generic CSR PCG takes for which matrices, against a fake
// runtime (fake_cudart.hpp): the rules look at level widths and row lengths,
// and a matrix on the wrong side of them is slow, not wrong.
#include "fake_cudart.hpp"

#include <cstdio>
#include <functional>
#include <utility>
#include <vector>

#include "fm_api.h"
#include "fm_device.cuh"

static int bad = 0;
#define EXPECT(c, ...)                                  \
    do {                                                \
        if (!(c)) {                                     \
            ++bad;                                      \
            std::printf("%s:%d: ", __FILE__, __LINE__); \
            std::printf(__VA_ARGS__);                   \
            std::printf("\n");                          \
        }                                               \
    } while (0)

static std::set<std::string> launched;

static bool was(const char* name) {
    for (const auto& k : launched)
        if (k.find(name) != std::string::npos) return true;
    return false;
}

using Pairs = std::vector<std::pair<uint32_t, uint32_t>>;  // i > j

// the routes of one solve with the symmetric pattern of `pairs`
static void solve(uint32_t n, const Pairs& pairs) {
    std::vector<std::vector<uint32_t>> rows(n);
    for (const auto& p : pairs) {
        rows[p.first].push_back(p.second);
        rows[p.second].push_back(p.first);
    }
    std::vector<uint32_t> rp{0}, ci;
    std::vector<double> val, b(n, 1.0), x(n, 0.0);
    for (uint32_t i = 0; i < n; ++i) {
        rows[i].push_back(i);
        for (uint32_t j : rows[i]) {
            ci.push_back(j);
            val.push_back(i == j ? 100.0 : -1.0);
        }
        rp.push_back((uint32_t)ci.size());
    }
    fm_ctx* c = nullptr;
    launched.clear();
    EXPECT(fm_create(&c, 0, nullptr) == FM_OK, "fm_create");
    const fm_status st = fm_csr_pcg_ilu0(c, n, rp.data(), ci.data(), val.data(), b.data(), x.data(),
                                         1e-8, 2, nullptr, nullptr);
    EXPECT(st == FM_OK, "n = %u: status %d", n, (int)st);
    fm_destroy(c);
}
static void one_cta(const char* what, bool want, uint32_t n, const Pairs& pairs) {
    solve(n, pairs);
    EXPECT(was("k_trsv_small") == want && was("k_trsv_lower_csr") != want, "%s: %s", what,
           want ? "not in one CTA" : "in one CTA");
}

static void lanes(const char* what, int want, uint32_t n, const Pairs& pairs) {
    solve(n, pairs);
    for (int g : {4, 8, 32})
        EXPECT(was(("k_spmv_csrIdLi" + std::to_string(g) + "E").c_str()) == (g == want),
               "%s: %d lanes a row", what, g);
}

static Pairs band(uint32_t n, uint32_t k, uint32_t step) {
    Pairs p;
    for (uint32_t q = 1; q <= k; ++q)
        for (uint32_t i = q * step; i < n; ++i) p.push_back({i, i - q * step});
    return p;
}
static Pairs grid(uint32_t g, bool red_black) {
    auto id = [&](uint32_t i, uint32_t j) {
        const uint32_t at = i * g + j;
        return !red_black ? at : (i + j) % 2 == 0 ? at / 2 : (g * g + 1) / 2 + at / 2;
    };
    Pairs p;
    auto add = [&](uint32_t a, uint32_t b) { p.push_back({std::max(a, b), std::min(a, b)}); };
    for (uint32_t i = 0; i < g; ++i)
        for (uint32_t j = 0; j < g; ++j) {
            if (i) add(id(i, j), id(i - 1, j));
            if (j) add(id(i, j), id(i, j - 1));
        }
    return p;
}
// k arrowheads of m rows: each one's last row is full
static Pairs arrows(uint32_t m, uint32_t k) {
    Pairs p;
    for (uint32_t q = 0; q < k; ++q)
        for (uint32_t j = 0; j + 1 < m; ++j) p.push_back({q * m + m - 1, q * m + j});
    return p;
}
int main() {
    fake::on_launch = [](const fake::Launch& l) {
        launched.insert(l.kernel);
        const bool init = l.kernel.find("k_pcg_init") != std::string::npos;
        if (init || l.kernel.find("k_pcg_rz") != std::string::npos) {
            auto* r = *static_cast<fm::PcgReport**>(l.args[init ? 9 : 7]);
            r->done = 0;
            r->seq = *static_cast<unsigned*>(l.args[init ? 10 : 8]);
        }
        return cudaSuccess;
    };
    // long chains of narrow levels, and a few levels that a block takes in a
    // few turns: one CTA
    one_cta("one row", true, 1, {});
    one_cta("tridiagonal", true, 5000, band(5000, 1, 1));
    one_cta("five-point 150 x 150", true, 22500, grid(150, false));
    one_cta("three levels of 512, three per side", true, 1536, band(1536, 3, 512));
    one_cta("eight per side, 17 levels", true, 26000, band(26000, 8, 1536));
    one_cta("diagonal, 7000 rows", true, 7000, {});
    one_cta("red-black 64 x 64", true, 4096, grid(64, true));
    one_cta("two per side, four levels of 7000", true, 27000, band(27000, 2, 7000));
    // wide shallow ones: the whole device
    one_cta("diagonal, 27000 rows", false, 27000, {});
    one_cta("red-black 120 x 120", false, 14400, grid(120, true));
    one_cta("red-black 164 x 164", false, 26896, grid(164, true));
    one_cta("two per side, two levels", false, 26000, band(26000, 2, 14336));
    one_cta("eight per side, six levels", false, 26000, band(26000, 8, 5120));
    // beyond its limits: entries, and the vector
    one_cta("nine per side", false, 900, band(900, 9, 5));
    one_cta("28600 rows", false, 28600, band(28600, 2, 7000));

    // lanes per row: by the mean length, more where a long row decides
    lanes("diagonal", 4, 3000, {});
    lanes("five-point 64 x 64", 4, 4096, grid(64, false));
    lanes("nine per row", 8, 4000, band(4000, 4, 9));
    lanes("seventeen per row", 32, 4000, band(4000, 9, 9));
    lanes("arrowhead 500", 32, 500, arrows(500, 1));
    lanes("40 arrowheads 500", 32, 20000, arrows(500, 40));
    lanes("400 arrowheads 500", 8, 200000, arrows(500, 400));
    lanes("8 arrowheads 60", 32, 480, arrows(60, 8));
    lanes("2000 arrowheads 200", 4, 400000, arrows(200, 2000));
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
