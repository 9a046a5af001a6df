// A launch that the runtime refuses inside a call of the C ABI, against a fake
// runtime (fake_cudart.hpp).  Whichever launch it is, the call must return an
// error, leave no error behind for the next call to report, and leave a
// context on which the same call then succeeds.  The fake "kernels" compute
// nothing; the two that report a PCG step to the host do report, so that a
// call which does not look at its launches runs through.
#include "fake_cudart.hpp"

#include <cstdio>
#include <cstring>
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

static std::vector<std::string> launches;  // of the running call, in order
static int refuse = -1;                    // index of the launch to refuse
static const char* refuse_all = nullptr;   // and every launch of this kernel
static unsigned report_status = 0, init_done = 0;
static int rz_seen = 0, rz_stop = 3;       // the step that ends the solve

static int dots = 0;                       // reductions of the running call

static bool is(const std::string& k, const char* name) { return k.find(name) != std::string::npos; }

static cudaError_t hook(const fake::Launch& l) {
    const int at = (int)launches.size();
    launches.push_back(l.kernel);
    if (at == refuse || (refuse_all && is(l.kernel, refuse_all))) return cudaErrorInvalidValue;
    fm::PcgReport* r = nullptr;
    unsigned seq = 0;
    if (is(l.kernel, "k_pcg_init")) {
        r = *static_cast<fm::PcgReport**>(l.args[9]);
        seq = *static_cast<unsigned*>(l.args[10]);
        r->done = init_done;
        rz_seen = 0;
    } else if (is(l.kernel, "k_pcg_rz")) {
        r = *static_cast<fm::PcgReport**>(l.args[7]);
        seq = *static_cast<unsigned*>(l.args[8]);
        r->done = ++rz_seen >= rz_stop;
    }
    // the norms that a Newton step reads: two iterations, then converged
    if (is(l.kernel, "k_dot")) **static_cast<double**>(l.args[5]) = ++dots <= 4 ? 1.0 / dots : 0.0;
    if (r) {
        r->rr = r->relres = 0.25;
        r->status = report_status;
        r->stop = 0;
        r->seq = seq;
    }
    return cudaSuccess;
}

// every launch of `f` refused in turn, each in a context of its own; some may
// be replaced by another kernel
template <typename Call>
static void each_launch(const char* name, Call f, const char* replaced = "(none)") {
    std::vector<std::string> all;
    for (int k = -1; k < (int)all.size(); ++k) {
        fm_ctx* c = nullptr;
        EXPECT(fm_create(&c, 0, nullptr) == FM_OK, "fm_create");
        launches.clear();
        dots = 0;
        refuse = k;
        fm_status st = f(c);
        refuse = -1;
        if (k < 0) {
            all = launches;
            EXPECT(st == FM_OK, "%s: status %d", name, (int)st);
            EXPECT(!all.empty(), "%s launches nothing", name);
        } else if (is(all[k], replaced)) {
            EXPECT(st == FM_OK, "%s: no replacement for %s", name, all[k].c_str());
        } else if (is(all[k], "k_fill_sentinel") && st == FM_OK) {
            // the fill of a push solve: the pipelined solves took its place
            bool piped = false;
            for (const auto& l : launches) piped |= is(l, "k_trsv_upper_pipe");
            EXPECT(piped, "%s: launch %d (%s) refused and forgotten", name, k, all[k].c_str());
        } else {
            EXPECT(st == FM_ERR_CUDA, "%s: launch %d (%s) refused: status %d", name, k,
                   all[k].c_str(), (int)st);
        }
        EXPECT(fake::last_error == cudaSuccess, "%s: launch %d: an error was left behind", name, k);
        fake::last_error = cudaSuccess;
        launches.clear();
        dots = 0;
        st = f(c);
        EXPECT(st == FM_OK, "%s: launch %d: the next call returns %d", name, k, (int)st);
        fm_destroy(c);
    }
}

int main() {
    fake::on_launch = hook;
    // generic CSR: tridiagonal, both paths of its triangular solves
    const uint32_t n = 6;
    std::vector<uint32_t> rp{0}, ci;
    std::vector<double> val, b(n, 1.0), x(n, 0.0);
    for (uint32_t i = 0; i < n; ++i) {
        for (uint32_t j = i ? i - 1 : 0; j <= i + 1 && j < n; ++j) {
            ci.push_back(j);
            val.push_back(i == j ? 4.0 : -1.0);
        }
        rp.push_back((uint32_t)ci.size());
    }
    int it = -1;
    double rel = -1.0;
    auto csr = [&](fm_ctx* c) {
        return fm_csr_pcg_ilu0(c, n, rp.data(), ci.data(), val.data(), b.data(), x.data(), 1e-8, 9,
                               &it, &rel);
    };
    each_launch("csr_pcg", csr, "k_trsv_small");
    EXPECT(it == rz_stop && rel == 0.25, "csr_pcg: %d iterations, %g", it, rel);
    refuse_all = "k_trsv_small";
    each_launch("csr_pcg, warp per row", csr, "k_trsv_small");
    refuse_all = nullptr;

    // without iterations (a cap of zero or below) the entry still counts: its
    // early exit is zero iterations, and its flags are an error
    for (int cap : {0, -1}) {
        fm_ctx* c = nullptr;
        EXPECT(fm_create(&c, 0, nullptr) == FM_OK, "fm_create");
        for (unsigned done : {0u, 1u}) {
            init_done = done;
            it = 77;
            const fm_status st = fm_csr_pcg_ilu0(c, n, rp.data(), ci.data(), val.data(), b.data(),
                                                 x.data(), 1e-8, cap, &it, &rel);
            EXPECT(st == FM_OK && it == (done ? 0 : cap), "cap %d, early exit %u: status %d, %d",
                   cap, done, (int)st, it);
        }
        init_done = 0;
        report_status = FM_FLAG_NONFINITE;
        const fm_status st = fm_csr_pcg_ilu0(c, n, rp.data(), ci.data(), val.data(), b.data(),
                                             x.data(), 1e-8, cap, &it, &rel);
        EXPECT(st == FM_ERR_NONFINITE, "cap %d: a non-finite entry returns %d", cap, (int)st);
        report_status = 0;
        fm_destroy(c);
    }

    // on a mesh: one tet, whose structures the fake leaves empty
    const double xyz[12] = {0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1};
    const uint32_t conn[4] = {0, 1, 2, 3};
    const uint8_t mask[12] = {1, 1, 1};
    std::vector<double> u(12), f(12), y(12), g(1), h(1);
    auto mesh = [&](fm_ctx* c) {
        fm_status st = fm_set_mesh(c, 4, xyz, 1, conn, nullptr);
        if (st == FM_OK) st = fm_set_material(c, 1.0, 0.3, nullptr);
        return st != FM_OK ? st : fm_set_bc(c, mask, nullptr);
    };
    auto factored = [&](fm_ctx* c, fm_precision prec) {
        fm_status st = mesh(c);
        if (st == FM_OK) st = fm_assemble(c, u.data(), nullptr, f.data(), prec, 1);
        return st != FM_OK ? st : fm_ilu0(c, prec);
    };
    each_launch("residual", [&](fm_ctx* c) {
        const fm_status st = mesh(c);
        return st != FM_OK ? st : fm_residual(c, u.data(), f.data());
    });
    each_launch("exact_apply", [&](fm_ctx* c) {
        const fm_status st = mesh(c);
        return st != FM_OK ? st : fm_exact_apply(c, u.data(), f.data(), y.data(), 1);
    });
    each_launch("spmv", [&](fm_ctx* c) {
        fm_status st = factored(c, FM_FP64);
        return st != FM_OK ? st : fm_spmv(c, f.data(), y.data());
    });
    each_launch("ilu0_apply", [&](fm_ctx* c) {
        fm_status st = factored(c, FM_FP64);
        return st != FM_OK ? st : fm_ilu0_apply(c, f.data(), y.data());
    }, "k_trsv_push");
    each_launch("ilu0_apply_noalloc", [&](fm_ctx* c) {
        fm_status st = factored(c, FM_FP64);
        return st != FM_OK ? st : fm_ilu0_apply_noalloc(c, f.data(), y.data());
    }, "k_trsv_push");
    for (const char* path : {"push", "pipe"}) {
        setenv("FM_TRSV_PATH", path, 1);
        for (fm_precision prec : {FM_FP64, FM_MIXED})
            each_launch("pcg", [&](fm_ctx* c) {
                fm_status st = factored(c, prec);
                return st != FM_OK ? st
                                   : fm_pcg(c, f.data(), y.data(), 1e-8, 9, &it, &rel, prec);
            }, "k_trsv_push");
    }
    unsetenv("FM_TRSV_PATH");
    for (int prec : {(int)FM_FP64, (int)FM_MIXED})
        for (int search : {0, 2})
            each_launch("newton", [&](fm_ctx* c) {
                fm_status st = mesh(c);
                fm_newton_config cfg;
                fm_newton_config_default(&cfg);
                cfg.precision = prec;
                cfg.line_search = search;
                cfg.initial_guess = 1;
                fm_newton_result res;
                return st != FM_OK ? st : fm_newton_step_cfg(c, u.data(), 0.5, &cfg, &res);
            }, "k_trsv_push");

    // a mesh that could not be set leaves none: later calls launch nothing
    {
        fm_ctx* c = nullptr;
        EXPECT(fm_create(&c, 0, nullptr) == FM_OK && mesh(c) == FM_OK, "no first mesh");
        launches.clear();
        EXPECT(mesh(c) == FM_OK, "no second mesh");
        for (int k = 0, all = (int)launches.size(); k < all; ++k) {
            launches.clear();
            refuse = k;
            EXPECT(mesh(c) == FM_ERR_CUDA, "launch %d of fm_set_mesh refused", k);
            refuse = -1;
            launches.clear();
            uint32_t nodes = 7;
            EXPECT(fm_sizes(c, &nodes, nullptr, nullptr, nullptr) == FM_OK && nodes == 0,
                   "launch %d: %u nodes", k, nodes);
            EXPECT(fm_residual(c, u.data(), f.data()) == FM_ERR_ARG &&
                       fm_assemble(c, u.data(), nullptr, f.data(), FM_FP64, 0) == FM_ERR_ARG &&
                       fm_spmv(c, f.data(), y.data()) == FM_ERR_ARG && launches.empty(),
                   "launch %d: half a mesh is used", k);
            EXPECT(mesh(c) == FM_OK && fm_residual(c, u.data(), f.data()) == FM_OK,
                   "launch %d: no mesh afterwards", k);
        }
        fm_destroy(c);
    }

    if (!bad) std::printf("ok\n");
    return bad != 0;
}
