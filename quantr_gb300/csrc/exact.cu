// exact.cu — tile passes of QGPU_MODE_EXACT: runs of standard gates in the reference's arithmetic
// and order (simulation.rs:64-181), many per launch.
//
// Every standard gate is a controlled 2x2 (or a swap) whose images have at most two non-zero
// entries per output. k_group (program.cu) forms every product of the gate's 2^k x 2^k table; here
// the products with entries 0 and 1 are left out. On finite amplitudes that changes no value: such
// a product is a zero or the amplitude itself, and a zero added to the sum leaves it as it is (only
// the sign of a zero result may differ). What remains is the reference's: f64 products and sums
// without contraction, the input of the lower index first. Gates keep their order (rounding does
// not commute); a pass takes the next ones as long as the bits they change fit its tile of 2^K
// amplitudes in shared memory. Controls and diagonal gates need no bit in the tile.
// Bound: the FP64 pipe (2 lanes per cycle and SM), so small registers take small tiles that fill
// the SMs. One launch per gate against tile passes: 14 qubits, 20 brickwork layers + QFT (1082 gates)
// 7.42 / 0.83 ms; 18 qubits, 6 layers + QFT 9.92 / 1.78 ms; 24 qubits, 1 layer + QFT 374 / 44 ms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.cuh"
#include "plan.h"

namespace qgpu {

constexpr int EX_BITS = 10;        // widest tile
constexpr int EX_MAX_OPS = 192;    // gates per pass (their table lies in shared memory)

enum : int32_t { EX_DIAG, EX_SWAP, EX_FLIP, EX_ANTI, EX_REAL, EX_CROSS };

struct ExOp {
    int32_t type;
    int32_t bit, bit2;      // tile bit (EX_DIAG: -1 - index bit when outside the tile); swap's second
    uint32_t lcm;           // controls inside the tile,
    uint64_t ocm;           // and outside
    int32_t one0, one1;     // EX_DIAG: factor 1 for bit value 0 / 1
    double m[8];            // EX_DIAG: d0, d1; EX_ANTI: out0 = m01 b, out1 = m10 a; EX_REAL: m00 m01 m10
                            // m11 (real); EX_CROSS: m00, m11 real, m01, m10 imaginary
};
static_assert(sizeof(ExOp) % 16 == 0, "copied in 16-byte pieces");

struct ExParams {
    uint64_t ntiles;
    const ExOp* ops;
    int nops;
    int nbits;
    int nfields;                      // runs of index bits outside the tile
    uint8_t bits[EX_BITS];
    uint8_t src[EX_BITS + 1], dst[EX_BITS + 1];
    uint64_t field[EX_BITS + 1];
};

// num-complex Mul, no FMA contraction
__device__ __forceinline__ double2 ex_mul(double mx, double my, double2 x) {
    return make_double2(__dsub_rn(__dmul_rn(mx, x.x), __dmul_rn(my, x.y)),
                        __dadd_rn(__dmul_rn(mx, x.y), __dmul_rn(my, x.x)));
}

// One thread per amplitude of the tile, the amplitude in a register: a gate that mixes pairs takes
// one exchange through shared memory (two buffers, one barrier) and every thread forms its own
// output, so all four FP64 units of the SM work (a thread per pair: 1.16 ms for the 14-qubit
// circuit).
__global__ void __launch_bounds__(1024) k_exact(double2* __restrict__ st, const __grid_constant__ ExParams p) {
    extern __shared__ __align__(16) double2 ex_buf[];  // [2][tile]
    const int t = threadIdx.x, TH = blockDim.x, T = 1 << p.nbits;
    ExOp* ops = reinterpret_cast<ExOp*>(ex_buf + 2 * T);
    {
        const uint4* src = reinterpret_cast<const uint4*>(p.ops);
        uint4* dst = reinterpret_cast<uint4*>(ops);
        for (int i = t; i < p.nops * (int)(sizeof(ExOp) / 16); i += TH) dst[i] = __ldg(src + i);
    }
    uint64_t offset = 0;
    for (int m = 0; m < p.nbits; ++m)
        if ((t >> m) & 1) offset |= 1ull << p.bits[m];
    const bool live = t < T;  // (a warp at least is launched)
    int which = 0;
    __syncthreads();
    for (uint64_t g = blockIdx.x; g < p.ntiles; g += gridDim.x) {
        uint64_t base = 0;
        for (int f = 0; f < p.nfields; ++f) base |= (g >> p.src[f]) << p.dst[f] & p.field[f];
        double2 v = live ? st[base | offset] : make_double2(0.0, 0.0);
        for (int k = 0; k < p.nops; ++k) {
            const ExOp& o = ops[k];
            if ((base & o.ocm) != o.ocm) continue;  // (the same for the whole tile)
            const int type = o.type, bit = o.bit;
            const bool on = ((uint32_t)t & o.lcm) == o.lcm;
            if (type == EX_DIAG) {
                const int b = bit < 0 ? (int)((base >> (-1 - bit)) & 1ull) : (t >> bit) & 1;
                if (on && !(b ? o.one1 : o.one0)) v = ex_mul(o.m[2 * b], o.m[2 * b + 1], v);
                continue;
            }
            double2* buf = ex_buf + which * T;
            which ^= 1;
            if (live) buf[t] = v;
            __syncthreads();
            if (!live || !on) continue;
            const int b = (t >> bit) & 1;
            if (type == EX_SWAP) {
                if (b != ((t >> o.bit2) & 1)) v = buf[t ^ (1 << bit) ^ (1 << o.bit2)];
                continue;
            }
            const double2 w = buf[t ^ (1 << bit)];
            if (type == EX_FLIP) {
                v = w;
            } else if (type == EX_ANTI) {
                v = ex_mul(o.m[2 * b], o.m[2 * b + 1], w);
            } else {
                // the inputs in index order: x at bit value 0, y at 1
                const double2 x = b ? w : v, y = b ? v : w;
                const double m0 = o.m[2 * b], m1 = o.m[2 * b + 1];
                if (type == EX_REAL) {
                    v = make_double2(__dadd_rn(__dmul_rn(m0, x.x), __dmul_rn(m1, y.x)),
                                     __dadd_rn(__dmul_rn(m0, x.y), __dmul_rn(m1, y.y)));
                } else if (b == 0) {  // EX_CROSS: an imaginary entry i s times (x, y) is (-s y, s x)
                    v = make_double2(__dadd_rn(__dmul_rn(m0, x.x), -__dmul_rn(m1, y.y)),
                                     __dadd_rn(__dmul_rn(m0, x.y), __dmul_rn(m1, y.x)));
                } else {
                    v = make_double2(__dadd_rn(-__dmul_rn(m0, x.y), __dmul_rn(m1, y.x)),
                                     __dadd_rn(__dmul_rn(m0, x.x), __dmul_rn(m1, y.y)));
                }
            }
        }
        if (live) st[base | offset] = v;
    }
}

// One gate with full-index bits.
struct ExGate {
    ExOp op;
    int bit = 0, bit2 = -1;
    uint64_t cm = 0, need = 0;
};

// False for forms no standard gate takes and for entries that are not finite: of an angle's NaN or
// infinity some amplitudes become NaN, and the products with 0 of this gate and the next ones spread
// them.
static bool exact_gate(const qgpu_op& op, const LocalGate& lg, int n, ExGate* g) {
    std::memset(&g->op, 0, sizeof(g->op));
    const int k = lg.k;
    const size_t d = (size_t)1 << k, call = (d - 1) & ~(size_t)1;
    for (cd z : lg.M)
        if (!std::isfinite(z.real()) || !std::isfinite(z.imag())) return false;
    g->bit = n - 1 - lg.wires[k - 1];
    if (op.kind == QGPU_GATE_SWAP) {
        g->op.type = EX_SWAP;
        g->bit2 = n - 1 - lg.wires[0];
        g->need = (1ull << g->bit) | (1ull << g->bit2);
        return true;
    }
    for (int m = 0; m < k - 1; ++m) g->cm |= 1ull << (n - 1 - lg.wires[m]);
    for (size_t j = 0; j < d; ++j)  // identity wherever a control is 0
        for (size_t l = 0; l < d; ++l) {
            if ((j & call) == call && (l & call) == call) continue;
            if (lg.M[j * d + l] != cd(j == l ? 1.0 : 0.0, 0.0)) return false;
        }
    cd u[2][2];
    for (int out = 0; out < 2; ++out)
        for (int in = 0; in < 2; ++in) u[out][in] = lg.M[(call | in) * d + (call | out)];
    auto zero = [](cd z) { return z == cd(0.0, 0.0); };
    auto put = [&](int at, cd z) {
        g->op.m[at] = z.real();
        g->op.m[at + 1] = z.imag();
    };
    if (zero(u[0][1]) && zero(u[1][0])) {
        g->op.type = EX_DIAG;
        put(0, u[0][0]);
        put(2, u[1][1]);
        g->op.one0 = u[0][0] == cd(1.0, 0.0);
        g->op.one1 = u[1][1] == cd(1.0, 0.0);
        return true;
    }
    g->need = 1ull << g->bit;
    if (zero(u[0][0]) && zero(u[1][1])) {
        put(0, u[0][1]);
        put(2, u[1][0]);
        g->op.type = u[0][1] == cd(1.0, 0.0) && u[1][0] == cd(1.0, 0.0) ? EX_FLIP : EX_ANTI;
        return true;
    }
    bool real = true, cross = true;
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) {
            real = real && u[r][c].imag() == 0.0;
            cross = cross && (r == c ? u[r][c].imag() : u[r][c].real()) == 0.0;
        }
    if (!real && !cross) return false;
    g->op.type = real ? EX_REAL : EX_CROSS;
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c)
            g->op.m[2 * r + c] = real || r == c ? u[r][c].real() : u[r][c].imag();
    return true;
}

int exact_passes(qgpu_handle* h, const qgpu_op* ops, const std::vector<LocalGate>& gates,
                 const std::vector<size_t>& at, size_t* taken) {
    const int n = h->n_qubits;
    // tiles that fill the SMs: 2^7 of them where the register allows tiles of 2^6 and more (14
    // qubits: tiles of 2^7 0.83 ms, 2^8 0.94 ms in 54 launches, 2^9 1.28 ms)
    const int width = std::min(n, std::min(EX_BITS, std::max(6, n - 7)));
    const int low = n >= 22 ? 2 : 0;  // (registers beyond L2: 64-byte runs)
    struct PassRange {
        uint64_t mask;
        size_t first, count;
    };
    std::vector<ExGate> list;
    std::vector<PassRange> passes;
    uint64_t mask = 0;
    size_t first = 0;
    const uint64_t low_mask = (1ull << low) - 1ull;
    *taken = 0;
    for (size_t i = 0; i < gates.size(); ++i) {
        ExGate g;
        if (ops[at[i]].kind == QGPU_GATE_CUSTOM || !exact_gate(ops[at[i]], gates[i], n, &g)) break;
        const bool fits = __builtin_popcountll(mask | low_mask | g.need) <= width &&
                          list.size() - first < (size_t)EX_MAX_OPS;
        if (!fits) {
            passes.push_back({mask, first, list.size() - first});
            mask = 0;
            first = list.size();
        }
        mask |= g.need;
        list.push_back(g);
        *taken = i + 1;
    }
    if (list.size() > first) passes.push_back({mask, first, list.size() - first});
    if (passes.empty()) return QGPU_OK;
    std::vector<ExOp> dev(list.size());
    std::vector<ExParams> prm(passes.size());
    for (size_t q = 0; q < passes.size(); ++q) {
        PassRange& ps = passes[q];
        ps.mask |= low_mask;
        for (int b = 0; b < n && __builtin_popcountll(ps.mask) < width; ++b) ps.mask |= 1ull << b;
        ExParams& p = prm[q];
        std::memset(&p, 0, sizeof(p));
        int local[64];
        for (int b = 0, out = 0; b < n; ++b) {
            if ((ps.mask >> b) & 1ull) {
                local[b] = p.nbits;
                p.bits[p.nbits++] = (uint8_t)b;
                continue;
            }
            local[b] = -1;
            if (p.nfields == 0 || ((ps.mask >> (b - 1)) & 1ull)) {
                p.src[p.nfields] = (uint8_t)out;
                p.dst[p.nfields++] = (uint8_t)b;
            }
            p.field[p.nfields - 1] |= 1ull << b;
            ++out;
        }
        p.ntiles = h->dim >> p.nbits;
        p.nops = (int)ps.count;
        for (size_t i = ps.first; i < ps.first + ps.count; ++i) {
            ExOp& o = dev[i];
            o = list[i].op;
            o.bit = local[list[i].bit] >= 0 ? local[list[i].bit] : -1 - list[i].bit;
            if (list[i].bit2 >= 0) o.bit2 = local[list[i].bit2];
            for (int b = 0; b < n; ++b) {
                if (!((list[i].cm >> b) & 1ull)) continue;
                if (local[b] >= 0) o.lcm |= 1u << local[b];
                else o.ocm |= 1ull << b;
            }
        }
    }
    int st = h->gates.ensure(dev.size() * sizeof(ExOp));
    if (st != QGPU_OK) return st;
    QGPU_CUDA(copy_async(h, h->gates.ptr, dev.data(), dev.size() * sizeof(ExOp), cudaMemcpyHostToDevice));
    for (size_t q = 0; q < passes.size(); ++q) {
        ExParams& p = prm[q];
        p.ops = (const ExOp*)h->gates.ptr + passes[q].first;
        const int threads = std::max(32, 1 << p.nbits);
        const size_t smem = ((size_t)2 << p.nbits) * sizeof(double2) + (size_t)p.nops * sizeof(ExOp);
        if (smem > 48 * 1024) {
            const cudaError_t e = smem_opt_in((const void*)k_exact, smem);
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_exact)");
        }
        const uint64_t grid = std::max<uint64_t>(1, std::min<uint64_t>(p.ntiles, (uint64_t)h->sm_count * 8));
        k_exact<<<(unsigned)grid, threads, smem, h->stream>>>((double2*)h->state, p);
        QGPU_CHECK_LAUNCH("k_exact");
        h->launches++;
        h->h2d_bytes += sizeof(p);
    }
    QGPU_CUDA(cudaStreamSynchronize(h->stream));
    return QGPU_OK;
}

}  // namespace qgpu
