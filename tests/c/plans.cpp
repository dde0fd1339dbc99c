// The planner of the register passes on the host, linked against the library:
//   plans norm N LAYERS    log of the factor by which the split program's
//                          1-qubit matrices change the squared norm, minus
//                          that of the gates it was made from (layers of Rx,
//                          Ry, Rz on N qubits and a CNOT brickwork)
//   plans time N BITS WHAT GATES
//                          seconds to plan GATES gates on the first N of BITS
//                          qubits (and, with "last", one on the next qubit at
//                          the end): WHAT = exact, fused, last, sweep
//   plans sizes            the largest description of a pass in bytes: 300
//                          different 2-qubit channels on 8 bits, phases between
//                          register bits and bits outside the tile on 24
//   plans supported        whether a pass takes a rotation, a matrix without
//                          targets, a swap of a qubit with itself, a control
//                          given twice
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "reg_tiles.h"
#include "sweep.h"

using namespace yao;

static void gate(std::vector<LGate>& prog, uint32_t n, int32_t type, uint32_t target, double angle, int control = -1) {
    GateElem g;
    g.type = type;
    g.targets = {target};
    g.params[0] = angle;
    if (control >= 0) {
        g.ctrls = {(uint32_t)control};
        g.cfgs = {1};
    }
    lower_gate(g, n, 0, false, prog);
}

static std::vector<LGate> layered(uint32_t n, int layers) {
    std::mt19937_64 r(1);
    std::uniform_real_distribution<double> angle(0.0, 6.283185307179586);
    std::vector<LGate> prog;
    for (int l = 0; l < layers; l++) {
        for (uint32_t q = 0; q < n; q++)
            for (int32_t type : {YAO_GATE_RX, YAO_GATE_RY, YAO_GATE_RZ}) gate(prog, n, type, q, angle(r));
        for (uint32_t a = l % 2; a + 1 < n; a += 2) gate(prog, n, YAO_GATE_X, a + 1, 0.0, (int)a);
    }
    return prog;
}

// sum over the uncontrolled matrices of the log of their rows' mean squared length
static long double log_norm(const std::vector<LGate>& prog) {
    long double sum = 0.0L;
    for (const LGate& g : prog) {
        if (g.nc || g.m.empty()) continue;
        long double t = 0.0L;
        for (const Cx& c : g.m) t += (long double)c.re * c.re + (long double)c.im * c.im;
        sum += std::log(t / (1 << g.k));
    }
    return sum;
}

static double seconds(uint32_t n, uint32_t nbits, const char* what, size_t gates) {
    std::mt19937_64 r(1);
    std::uniform_real_distribution<double> angle(0.0, 6.283185307179586);
    std::vector<LGate> prog;
    Circuit c;
    for (size_t i = 0; i < gates; i++) {
        const uint32_t t = (uint32_t)(r() % n), k = (t + 1 + (uint32_t)(r() % (n - 1))) % n;
        GateElem g;
        g.type = i % 4 == 3 ? YAO_GATE_X : YAO_GATE_RY;
        g.targets = {t};
        g.params[0] = angle(r);
        if (i % 4 == 3) {
            g.ctrls = {k};
            g.cfgs = {1};
        }
        Element e;
        e.g = g;
        c.elems.push_back(e);
        lower_gate(g, nbits, 0, false, prog);
    }
    if (!strcmp(what, "last")) gate(prog, nbits, YAO_GATE_RY, n, 0.5);
    double best = 1e9;
    for (int i = 0; i < 3; i++) {
        const auto t0 = std::chrono::steady_clock::now();
        if (!strcmp(what, "sweep")) {
            sweep_plan_free(sweep_plan_new(&c, nbits));
        } else {
            RegPlan plan;
            reg_plan(prog, nbits, YAO_C128, 11, strcmp(what, "fused") != 0, plan);
        }
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
    }
    return best;
}

int main(int argc, char** argv) {
    if (argc == 6 && !strcmp(argv[1], "time")) {
        printf("%.6f\n", seconds((uint32_t)atoi(argv[2]), (uint32_t)atoi(argv[3]), argv[4], (size_t)atoll(argv[5])));
        return 0;
    }
    if (argc == 4 && !strcmp(argv[1], "norm")) {
        const uint32_t n = (uint32_t)atoi(argv[2]);
        const std::vector<LGate> prog = layered(n, atoi(argv[3]));
        std::vector<LGate> split;
        split_single_qubit(prog, n, split);
        printf("%zu %.6Le\n", split.size(), log_norm(split) - log_norm(prog));
        return 0;
    }
    if (argc == 2 && !strcmp(argv[1], "sizes")) {
        std::mt19937_64 r(1);
        std::uniform_real_distribution<double> x(0.0, 1.0);
        std::vector<LGate> channels, phases;
        for (int i = 0; i < 300; i++) {
            LGate g;
            g.cls = GC_CHAN2;
            g.k = 4;
            for (int q = 0; q < 2; q++) {
                g.tb[2 * q] = i < 150 ? q : q + 1;
                g.tb[2 * q + 1] = 4 + g.tb[2 * q];
            }
            for (int op = 0; op < 16; op++) {
                const uint32_t type = (uint32_t)(op & 3);
                Cx head{0.0, 0.0};
                memcpy(&head.re, &type, 4);
                g.m.push_back(head);
                for (int j = 0; j < 4; j++) g.m.push_back(Cx{x(r), x(r)});
            }
            channels.push_back(g);
        }
        for (uint32_t q = 0; q < 24; q++) gate(phases, 24, YAO_GATE_RY, q, x(r));
        for (int i = 0; i < 300; i++) {
            LGate g;
            g.cls = GC_DIAG;
            g.k = 1;
            g.tb[0] = (int)(r() % 7);
            g.nc = 1;
            g.cb[0] = 11 + i % 13;
            g.cv[0] = 1;
            const double t = x(r);
            g.m = {Cx{1.0, 0.0}, Cx{std::cos(t), std::sin(t)}};
            phases.push_back(g);
        }
        RegPlan plan;
        for (auto* prog : {&channels, &phases}) {
            reg_plan(*prog, prog == &channels ? 8 : 24, YAO_C128, 11, prog == &channels, plan);
            size_t most = 0;
            for (const RegPass& p : plan.passes) most = std::max(most, p.blob_bytes);
            printf("%zu ", most);
        }
        puts("");
        return 0;
    }
    if (argc == 2 && !strcmp(argv[1], "supported")) {
        GateElem one, swap, twice;
        one.type = YAO_GATE_CUSTOM;
        one.custom_dim = 1;
        one.custom = {Cx{0.0, 1.0}};
        swap.type = YAO_GATE_SWAP;
        swap.targets = {2, 2};
        twice.type = YAO_GATE_X;
        twice.targets = {0};
        twice.ctrls = {1, 1};
        twice.cfgs = {1, 1};
        std::vector<LGate> prog;
        gate(prog, 6, YAO_GATE_RY, 3, 0.4);
        printf("%d", reg_supported(prog, 6));
        for (const GateElem* g : {&one, &swap, &twice}) {
            std::vector<LGate> with(prog);
            lower_gate(*g, 6, 0, false, with);
            printf(" %d", reg_supported(with, 6));
        }
        puts("");
        return 0;
    }
    return 1;
}
