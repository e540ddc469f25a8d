// plan_emulator.cpp over plans with wide passes: every step of a wide pass becomes a pass of its
// own (in round order), which the emulator then applies to the whole register.
#include "../../quantr_gb300/csrc/plan.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace qgpu {
int fail(int code, const std::string& msg);  // plan_emulator.cpp

int build_plan_wide(const qgpu_op* ops, size_t n_ops, int n, const double* mats, size_t n_mats,
                    const uint8_t* none, size_t n_none, PlanOptions opt, Plan* plan) {
    auto env = [](const char* name) { return std::atoi(std::getenv(name)); };
    opt.wide_bits = env("WIDE_BITS");
    opt.wide_regs = env("WIDE_REGS");
    opt.wide_low = env("WIDE_LOW");
    opt.wide_pairs = env("WIDE_PAIRS");
    int st = build_plan(ops, n_ops, n, mats, n_mats, none, n_none, opt, plan);
    if (st != QGPU_OK) return st;
    std::vector<Pass> out;
    size_t nwide = 0, nrounds = 0, nsteps = 0;
    for (const Pass& p : plan->passes) {
        if (p.wide < 0) {
            out.push_back(p);
            continue;
        }
        ++nwide;
        const WidePass& w = plan->wides[p.wide];
        size_t count = 0;
        bool bad = __builtin_popcountll(w.mask) > opt.wide_bits;
        auto step = [&](const WideStep& s, uint64_t bits) {
            ++count;
            Pass q;
            q.arith = true;
            int b[2] = {s.bit[0], s.bit[1]};
            for (int k = 0; k < 2; ++k) bad = bad || (b[k] >= 0 && !((bits >> b[k]) & 1ull));
            if (s.pair >= 0) {
                q.pair = s.pair;
                q.nbits = 2;
                q.bits[0] = std::min(b[0], b[1]);
                q.bits[1] = std::max(b[0], b[1]);
                out.push_back(q);
                return;
            }
            DevStep d = s.s;
            if (b[0] < 0) b[0] = 0;
            q.nbits = b[1] >= 0 ? 2 : 1;
            q.bits[0] = b[1] >= 0 ? std::min(b[0], b[1]) : b[0];
            if (b[1] >= 0) q.bits[1] = std::max(b[0], b[1]);
            d.lb = (uint8_t)(q.bits[0] == b[0] ? 0 : 1);
            d.lb2 = (uint8_t)(1 - d.lb);
            q.steps.push_back(d);
            out.push_back(q);
        };
        uint64_t outside = 0;
        auto moves = [&](const std::vector<WideMove>& ms) {
            for (const WideMove& m : ms) {
                WideStep s;
                std::memset(&s.s, 0, sizeof(s.s));
                s.s.type = m.swap ? ST_SWAP : ST_PERM;
                s.s.anti = 1;
                s.bit[0] = m.a;
                if (m.swap) s.bit[1] = m.b;
                else if (m.b >= 0) s.s.cm = 1ull << m.b;
                outside |= s.s.cm & ~w.mask;
                step(s, w.mask);
            }
        };
        for (const WideRound& r : w.rounds) {
            uint64_t bits = 0;
            for (int m = 0; m < r.nbits; ++m) bits |= 1ull << r.bits[m];
            bad = bad || r.nbits > opt.wide_regs || (bits & ~w.mask);
            moves(r.moves);
            for (int m = 0; m < r.nbits; ++m) {
                for (const WideStep* s : {r.has_pre[m] ? &r.pre[m] : nullptr, r.has_rot[m] ? &r.rot[m] : nullptr,
                                          r.has_post[m] ? &r.post[m] : nullptr}) {
                    if (!s) continue;
                    bad = bad || s->bit[0] != r.bits[m];
                    step(*s, bits);
                }
            }
            for (int k = 0; k < 2; ++k)
                if (r.has_pair[k]) {
                    bad = bad || std::min(r.pairs[k].bit[0], r.pairs[k].bit[1]) != r.bits[2 * k] ||
                          std::max(r.pairs[k].bit[0], r.pairs[k].bit[1]) != r.bits[2 * k + 1];
                    step(r.pairs[k], bits);
                }
            for (const WideStep& s : r.steps) step(s, bits);
        }
        moves(w.moves);
        if (bad || __builtin_popcountll(outside) > WIDE_MAX_OUTSIDE)
            return fail(QGPU_ERR_INVALID, "wide pass: a step outside its round, or a limit");
        if (count > (size_t)WIDE_MAX_STEPS || w.rounds.size() > (size_t)WIDE_MAX_ROUNDS)
            return fail(QGPU_ERR_INVALID, "wide pass over its limits");
        nrounds += w.rounds.size();
        nsteps += count;
    }
    std::printf("wide %zu rounds %zu steps %zu ", nwide, nrounds, nsteps);
    plan->passes.swap(out);
    return QGPU_OK;
}
}  // namespace qgpu

#define build_plan build_plan_wide
#include "plan_emulator.cpp"
