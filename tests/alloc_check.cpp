// CPU check: the planners and run_tasks answer a failed allocation with
// QK_ERR_OOM, wherever it happens, and end none of the process's threads
// otherwise.  The k-th allocation after a start mark fails, for k over all
// that a call makes (in steps).
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

static std::atomic<long> g_left{-1};   // allocations until the one that fails; negative: none does
void *operator new(std::size_t n) {
    if (g_left >= 0 && g_left.fetch_sub(1) == 0) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

#include "dense_sim.h"

using namespace dense_sim;

template <typename F> int sweep(const char *what, long step, F &&call) {
    int oom = 0, ok = 0;
    for (long k = 0;; k += step) {
        g_left = k;
        const int rc = call();
        const bool past = g_left >= 0;   // the call made fewer than k allocations
        g_left = -1;
        if (rc == QK_ERR_OOM) ++oom;
        else if (rc == QK_OK) ++ok;
        else return std::printf("%s: code %d at allocation %ld\n", what, rc, k), 1;
        if (past) break;
    }
    // (a thread that cannot be had is made up for: OK as well)
    if (!oom || !ok) return std::printf("%s: %d oom, %d ok\n", what, oom, ok), 1;
    return 0;
}

int main() {
    int bad = 0;
    bad += sweep("tasks", 1, [] { return qk::run_tasks(6, [](size_t) { return std::vector<int>(100).size() ? QK_OK : QK_ERR_ARG; }); });
    Gen G{std::mt19937_64(3), 7, false};
    std::vector<qk_gate> one, two;   // factored, general
    std::vector<int32_t> pidx;
    for (int i = 0; i < 130; ++i) {
        qk_gate g;
        std::memset(&g, 0, sizeof g);
        g.kind = i % 3 == 2 ? QK_GATE_CP : i % 3 ? QK_GATE_RY : QK_GATE_RX;
        g.nq = i % 3 == 2 ? 2 : 1;
        g.q[0] = i % 6;
        g.q[1] = i % 6 + 1;
        g.param = G.u();
        one.push_back(g);
        pidx.push_back(g.nq == 1 ? i : -1);
        two.push_back(i < 60 ? G.gate() : g);
    }
    for (int threads : {0, 1}) {
        qk::PlanOptions o = qk::factored_plan_options(QK_C128, 7), a = qk::factored_adjoint_options(QK_C128, 7);
        o.tile_bits = o.f_tile_bits = a.f_tile_bits = 5;
        o.reg_bits = o.f_reg_bits = a.f_reg_bits = 2;
        o.threads = threads;
        bad += sweep("factored", 7, [&] { qk::HostPlan hp; return qk::plan_forward(one.data(), one.size(), 7, o, hp); });
        bad += sweep("general", 29, [&] { qk::HostPlan hp; return qk::plan_forward(two.data(), two.size(), 7, o, hp); });
        bad += sweep("adjoint", 29, [&] { qk::HostPlan hp; return qk::plan_adjoint(one.data(), one.size(), pidx.data(), 7, a, hp); });
    }
    std::printf("%s\n", bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
