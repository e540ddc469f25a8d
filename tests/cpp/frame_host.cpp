// frame_host.cpp — pauli_frame (quantr_gb300/csrc/plan.cpp) over the whole range of angles: the undo of
// runs with one Rx near 0, pi and the smallest numbers is the frame's product up to a phase.
// Prints the largest difference of an entry.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>

#include "../../quantr_gb300/csrc/plan.h"

namespace qgpu {
int fail(int code, const std::string& msg) {
    std::fprintf(stderr, "error: %s\n", msg.c_str());
    return code;
}
}  // namespace qgpu
using namespace qgpu;

int main() {
    const double angles[] = {1.0, 3.14159265358979, 1e-8, 1e-149, 1e-151, 1e-300, 1e-307, 1e-310, 1e-315,
                             1e-320, 1e-322, 1e-323, 5e-324, 0.0};
    const int before[] = {QGPU_GATE_RZ, QGPU_GATE_X90, QGPU_GATE_H, QGPU_GATE_Y};
    double worst = 0.0;
    for (double a : angles)
        for (int kind : before)
            for (int v = 0; v < 200; ++v) {
                qgpu_op ops[3];
                std::memset(ops, 0, sizeof(ops));
                ops[0].kind = kind;
                ops[0].param = 0.1 + 0.03 * v;
                ops[1].kind = QGPU_GATE_RX;
                ops[1].param = v % 2 ? -a : a;
                ops[2].kind = QGPU_GATE_RZ;
                ops[2].param = 0.7 + 0.01 * v;
                PauliRun run;
                if (pauli_run(ops, {2, 1, 0}, 1, &run) != QGPU_OK) return 1;
                const PauliFrame f = pauli_frame(&run);
                const cd u[4] = {f.c, -f.s * f.rho1, f.rho2 * f.s, f.rho2 * f.c * f.rho1};
                const int lead = std::abs(u[0]) > std::abs(u[2]) ? 0 : 2;
                const cd phase = run.undo[lead] / u[lead];
                double d = std::fabs(std::abs(phase) - 1.0);
                for (int k = 0; k < 4; ++k) d = std::max(d, std::abs(phase * u[k] - run.undo[k]));
                if (!(d <= worst)) worst = std::isnan(d) ? HUGE_VAL : d;
            }
    std::printf("%.3g\n", worst);
    return 0;
}
