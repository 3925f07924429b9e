// CPU check: the factored planner takes no more than twice the general one's
// time on circuits of one or a few tiles, whose planning is longer than their
// run (best of 15 each; it took 2 to 5 times as long when every candidate was
// compiled and every choice of slots walked all of a pass).
#include <chrono>

#include "dense_sim.h"

using namespace dense_sim;

int main() {
    int bad = 0;
    for (int dtype : {QK_C128, QK_C64})
        for (int n : {8, 10, 12, 14}) {
            Gen G{std::mt19937_64(7), n, false};
            std::vector<qk_gate> gates;
            qk_gate g;
            for (int layer = 0; layer < 20; ++layer) {
                for (int q = 0; q < n; ++q) {
                    const double th = G.u(), ph = G.u(), la = G.u();
                    const cd m[4] = {std::cos(th), -std::polar(1.0, la) * std::sin(th), std::polar(1.0, ph) * std::sin(th),
                                     std::polar(1.0, ph + la) * std::cos(th)};
                    std::memset(&g, 0, sizeof g);
                    g.kind = QK_GATE_U1;
                    g.nq = 1;
                    g.q[0] = q;
                    std::memcpy(g.coeff, m, sizeof m);
                    gates.push_back(g);
                }
                for (int q = layer % 2; q + 1 < n; q += 2) {
                    std::memset(&g, 0, sizeof g);
                    g.kind = QK_GATE_CP;
                    g.nq = 2;
                    g.q[0] = q;
                    g.q[1] = q + 1;
                    g.param = M_PI;
                    gates.push_back(g);
                }
            }
            qk::PlanOptions o = qk::factored_plan_options(dtype, n);
            auto best = [&](auto &&plan) {
                double us = 1e9;
                for (int i = 0; i < 15; ++i) {
                    qk::HostPlan hp;
                    const auto t = std::chrono::steady_clock::now();
                    if (plan(hp)) std::exit(2);
                    us = std::min(us, std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t).count());
                }
                return us;
            };
            const double f = best([&](qk::HostPlan &hp) { return qk::plan_forward(gates.data(), gates.size(), n, o, hp); });
            const double d = best([&](qk::HostPlan &hp) { return qk::build_plan(gates.data(), gates.size(), n, o, hp); });
            std::printf("n %d: factored %.0f us, general %.0f us\n", n, f, d);
            bad += f > 2 * d;
        }
    std::printf("%s\n", bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
