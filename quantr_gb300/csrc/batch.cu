// batch.cu — many independent circuits: energies and adjoint gradients (no counterpart in quantr).
//
// Circuits whose two work vectors fit in one SM's shared memory (complex128 up to 12 qubits,
// complex64 up to 13) run in persistent launches, queued first: a CTA takes circuit after circuit
// from an atomic work counter (no CTA ever waits on another) and runs the forward pass, lambda =
// H psi, the energy and the adjoint reverse sweep entirely in shared memory. Registers of more
// than 10 qubits take CTAs of 1024 threads, smaller ones four CTAs of 256 threads per SM beside
// them. Meanwhile the larger circuits run through the register passes and qgpu_adjoint_grad on a
// few host threads, in the batch's precision. 96 complex128 circuits of 10 to 20 qubits, 4 layers:
// 45.8 -> 21.9 ms.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "internal.cuh"
#include "plan.h"
#include "workers.h"

namespace qgpu {

PlanOptions plan_options_for(const qgpu_handle* h);

constexpr int BATCH_MAX_Q = 40;
constexpr int BATCH_SMALL_BITS = 13;   // widest register of the shared-memory path (complex64)
constexpr int BATCH_NARROW_BITS = 10;  // registers up to this size take CTAs of 256 threads

// A circuit as records in order: runs of single-wire gates (each wire's gates as one frame, see
// PauliFrame), runs of CNot and Swap as one index map, and any other multi-wire gate.
enum : int32_t { B_RUN, B_MAP, B_GATE };
struct BRec {
    int32_t kind, first, count;   // B_RUN: wires; B_GATE: one gate
    int32_t d1, d2;               // B_RUN: whether any wire has a first / second diagonal
    uint16_t fwd[BATCH_SMALL_BITS + 1], rev[BATCH_SMALL_BITS + 1];  // B_MAP: new[y] = old[h(y)], h's
                                                                    // columns and, last, its offset
    int32_t pad;
};
struct BWire {
    int32_t lb;
    int32_t row[4];  // sums of X, Y (after the first diagonal), Z and -I (-1: not needed)
    int32_t pad;
    double c, s;     // the undo: diag(1, rho2) [[c, -s], [s, c]] diag(1, rho1)
    double2 rho1, rho2;
};

// One other gate in controlled-2x2 form (or a swap of two bits).
struct BOp {
    uint8_t swap, t, b2, pad;
    uint32_t cm;               // control bits that must be 1
    double u[8];               // U row-major (complex)
    double v[8];               // U^dagger row-major
};

struct BCirc {
    int n, nrec;
    int64_t rec0, wire0, op0;
    int64_t obs0;   // a[n] then b[n] in the observable array
    int64_t row0;   // first row sum
};

// Arithmetic of the two precisions. Sums are f64 (complex128), or error-free products and sums of
// f32 (complex64), a few per thread, added up in f64.
struct B128 {
    using T = double2;
    struct Sum {
        double v;
        __device__ __forceinline__ void clear() { v = 0.0; }
        // += Re(conj(a) b); Im(conj(a) b)
        __device__ __forceinline__ void re(T a, T b, double sign) {
            v = fma(sign * a.x, b.x, fma(sign * a.y, b.y, v));
        }
        __device__ __forceinline__ void im(T a, T b, double sign) {
            v = fma(sign * a.x, b.y, fma(-sign * a.y, b.x, v));
        }
        __device__ __forceinline__ double value() const { return v; }
    };
    struct Rot {
        double c, s;
        __device__ __forceinline__ explicit Rot(double c_, double s_) : c(c_), s(s_) {}
    };
    static __device__ __forceinline__ void rotate(T& a, T& b, const Rot& r) {
        const T x = make_double2(fma(r.c, a.x, -(r.s * b.x)), fma(r.c, a.y, -(r.s * b.y)));
        b = make_double2(fma(r.s, a.x, r.c * b.x), fma(r.s, a.y, r.c * b.y));
        a = x;
    }
    static __device__ __forceinline__ T make(double2 z) { return z; }
    static __device__ __forceinline__ T mul(T a, T b) {
        return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
    }
};
struct B64 {
    using T = float2;
    struct Sum {
        u64 s, e;
        __device__ __forceinline__ void clear() { s = e = 0; }
        __device__ __forceinline__ void add(u64 a, u64 b) {
            const u64 p = pmul(a, b), r = pfma(a, b, p ^ 0x8000000080000000ull);
            const u64 t = padd(s, p), bb = psub(t, s);
            e = padd(e, padd(padd(psub(s, psub(t, bb)), psub(p, bb)), r));
            s = t;
        }
        __device__ __forceinline__ void re(T a, T b, float sign) { add(p2(sign * a.x, sign * a.y), p2(b.x, b.y)); }
        __device__ __forceinline__ void im(T a, T b, float sign) { add(p2(sign * a.x, -sign * a.y), p2(b.y, b.x)); }
        __device__ __forceinline__ double value() const {
            float a, b, c, d;
            up2(s, a, b);
            up2(e, c, d);
            return ((double)a + (double)b) + ((double)c + (double)d);
        }
    };
    struct Rot {  // (hi, lo): only the amplitudes are rounded to f32
        float c, cl, s, sl;
        __device__ __forceinline__ explicit Rot(double c_, double s_)
            : c((float)c_), cl((float)(c_ - (double)(float)c_)), s((float)s_), sl((float)(s_ - (double)(float)s_)) {}
    };
    static __device__ __forceinline__ void rotate(T& a, T& b, const Rot& r) {
        auto dot = [](float x, float xl, float p, float y, float yl, float q) {
            return fmaf(x, p, fmaf(y, q, fmaf(xl, p, yl * q)));
        };
        const T o = make_float2(dot(r.c, r.cl, a.x, -r.s, -r.sl, b.x), dot(r.c, r.cl, a.y, -r.s, -r.sl, b.y));
        b = make_float2(dot(r.s, r.sl, a.x, r.c, r.cl, b.x), dot(r.s, r.sl, a.y, r.c, r.cl, b.y));
        a = o;
    }
    static __device__ __forceinline__ T make(double2 z) { return make_float2((float)z.x, (float)z.y); }
    static __device__ __forceinline__ T mul(T a, T b) {
        return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
    }
};

template <class T>
__device__ __forceinline__ void apply2(T* v, const BOp& o, const double* m, int dim) {
    using R = decltype(T::x);
    const R m0 = (R)m[0], m1 = (R)m[1], m2 = (R)m[2], m3 = (R)m[3], m4 = (R)m[4], m5 = (R)m[5],
            m6 = (R)m[6], m7 = (R)m[7];
    for (int p = threadIdx.x; p < dim / 2; p += blockDim.x) {
        const int i0 = (int)insert_zero((uint64_t)p, o.t), i1 = i0 | (1 << o.t);
        if (o.swap) {
            // exchange (bit t, bit b2) = (1, 0) with (0, 1): visit each exchanged pair once
            if (((i0 >> o.b2) & 1) == 1) {
                const int j = i0 ^ (1 << o.b2) ^ (1 << o.t);
                const T x = v[i0];
                v[i0] = v[j];
                v[j] = x;
            }
            continue;
        }
        if (((uint32_t)i0 & o.cm) != o.cm) continue;
        const T a = v[i0], b = v[i1];
        T r0, r1;
        r0.x = m0 * a.x - m1 * a.y + m2 * b.x - m3 * b.y;
        r0.y = m0 * a.y + m1 * a.x + m2 * b.y + m3 * b.x;
        r1.x = m4 * a.x - m5 * a.y + m6 * b.x - m7 * b.y;
        r1.y = m4 * a.y + m5 * a.x + m6 * b.y + m7 * b.x;
        v[i0] = r0;
        v[i1] = r1;
    }
}

// k_batch_small: forward pass, H psi, energy and reverse sweep of circuits in shared memory. Bound: the FP64 pipe (complex128), so gates are merged first: a run of single-wire gates
// costs 4 f64 operations per amplitude and wire (a real rotation) plus 8 for all diagonals together,
// and in the sweep 10 per amplitude and wire (both vectors, and the Y sum) plus 20 (diagonals, and
// one product from which all Z sums come), where gate by gate a Ry Rz pair with its CNot took 20 and
// 48; a CNot ring is one index map. A sum's terms, one per thread, go through shared memory to one
// warp each, so that the other warps go on (shuffles in every warp took a fifth of the FP64 time).
// 30 complex128 circuits of 10 to 12 qubits, 4 layers: 4.9 -> 1.2 ms; 300 complex64 circuits of 10
// to 13 qubits: 1.2 ms of a 9.5 ms call (13.2 before), the rest of which is lowering on the host.
template <class A, int TH, int PER, int CTAS>
__global__ void __launch_bounds__(TH, CTAS)
k_batch_small(const BCirc* __restrict__ circs, int ncirc, const BRec* __restrict__ recs,
              const BWire* __restrict__ wires, const BOp* __restrict__ ops,
              const double* __restrict__ obs, double* __restrict__ energy, double* __restrict__ sums,
              unsigned* __restrict__ counter, int bits) {
    using T = typename A::T;
    using Sum = typename A::Sum;
    constexpr int LOG_TH = TH == 1024 ? 10 : 8, WARPS = TH / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ T tab_lo[64], tab_hi[128];                       // diagonal factors of bits 0..5, 6..12
    __shared__ double red[4][TH];  // one term per thread of up to four sums
    __shared__ int cur;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    T* phi = reinterpret_cast<T*>(smem);
    T* lam = phi + ((size_t)1 << bits);
    // One warp adds up a row of `red`, signed by bit `lb` of the thread (none: -1); in lane 0.
    auto row_sum = [&](const double* row, int lb) {
        double v = 0.0;
#pragma unroll 8
        for (int k = lane; k < TH; k += 32) v += lb >= 0 && ((k >> lb) & 1) ? -row[k] : row[k];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
        return v;
    };
    for (;;) {
        if (t == 0) cur = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int ci = cur;
        __syncthreads();
        if (ci >= ncirc) return;
        const BCirc C = circs[ci];
        const int dim = 1 << C.n;
        const BRec* rec = recs + C.rec0;
        const BWire* wire = wires + C.wire0;
        // factors of one diagonal of a run (its inverse with conj)
        auto tables = [&](const BRec& r, bool second, bool conj) {
            for (int e = t; e < 64 + 128; e += TH) {
                const int hi = e >= 64, x = hi ? e - 64 : e;
                double2 f = make_double2(1.0, 0.0);
                for (int w = 0; w < r.count; ++w) {
                    const BWire& bw = wire[r.first + w];
                    const int b = bw.lb - (hi ? 6 : 0);
                    if (b < 0 || b >= (hi ? 7 : 6) || !((x >> b) & 1)) continue;
                    const double2 z = second ? bw.rho2 : bw.rho1;
                    f = B128::mul(f, make_double2(z.x, conj ? -z.y : z.y));
                }
                (hi ? tab_hi : tab_lo)[x] = A::make(f);
            }
            __syncthreads();
        };
        auto diagonal = [&](T* v, int x) { v[x] = A::mul(v[x], A::mul(tab_lo[x & 63], tab_hi[x >> 6])); };
        auto gather = [&](T* v, const uint16_t* h) {  // new[y] = old[h(y)]
            T x[PER];
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int y = t + j * TH;
                if (y >= dim) break;
                int src = h[BATCH_SMALL_BITS];
                for (int b = 0; b < C.n; ++b) src ^= (y >> b) & 1 ? h[b] : 0;
                x[j] = v[src];
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (t + j * TH < dim) v[t + j * TH] = x[j];
            __syncthreads();
        };
        for (int x = t; x < dim; x += TH) {
            phi[x].x = x == 0 ? 1 : 0;
            phi[x].y = 0;
        }
        __syncthreads();
        for (int k = 0; k < C.nrec; ++k) {
            const BRec& r = rec[k];
            if (r.kind == B_MAP) {
                gather(phi, r.fwd);
            } else if (r.kind == B_GATE) {
                apply2(phi, ops[C.op0 + r.first], ops[C.op0 + r.first].u, dim);
                __syncthreads();
            } else {
                if (r.d2) {
                    tables(r, true, true);
                    for (int x = t; x < dim; x += TH) diagonal(phi, x);
                    __syncthreads();
                }
                for (int w = 0; w < r.count; ++w) {
                    const BWire& bw = wire[r.first + w];
                    const int lb = bw.lb;
                    const typename A::Rot rot(bw.c, -bw.s);
                    for (int p = t; p < dim / 2; p += TH) {
                        const int i0 = ((p >> lb) << (lb + 1)) | (p & ((1 << lb) - 1)), i1 = i0 | (1 << lb);
                        T a = phi[i0], b = phi[i1];
                        A::rotate(a, b, rot);
                        phi[i0] = a;
                        phi[i1] = b;
                    }
                    __syncthreads();
                }
                if (r.d1) {
                    tables(r, false, true);
                    for (int x = t; x < dim; x += TH) diagonal(phi, x);
                    __syncthreads();
                }
            }
        }
        // lambda = H phi, energy = Re <phi|lambda>
        const double* a = obs + C.obs0;
        const double* b = a + C.n;
        double e = 0.0;
        for (int x = t; x < dim; x += TH) {
            double d = 0.0;
            for (int i = 0; i < C.n; ++i) {
                const int j = (i + 1) % C.n;
                const int par = ((x >> (C.n - 1 - i)) ^ (x >> (C.n - 1 - j))) & 1;
                d += par ? -a[i] : a[i];
            }
            double re = d * (double)phi[x].x, im = d * (double)phi[x].y;
            for (int i = 0; i < C.n; ++i) {
                const T w = phi[x ^ (1 << (C.n - 1 - i))];
                re = fma(b[i], (double)w.x, re);
                im = fma(b[i], (double)w.y, im);
            }
            lam[x].x = re;
            lam[x].y = im;
            e = fma((double)phi[x].x, re, fma((double)phi[x].y, im, e));
        }
        red[0][t] = e;
        __syncthreads();
        if (warp == 0) {
            e = row_sum(red[0], -1);
            if (lane == 0) energy[ci] = e;
        }
        __syncthreads();
        // reverse sweep
        for (int k = C.nrec - 1; k >= 0; --k) {
            const BRec& r = rec[k];
            if (r.kind == B_MAP) {
                gather(phi, r.rev);
                gather(lam, r.rev);
                continue;
            }
            if (r.kind == B_GATE) {
                const BOp& o = ops[C.op0 + r.first];
                apply2(phi, o, o.v, dim);
                apply2(lam, o, o.v, dim);
                __syncthreads();
                continue;
            }
            // q = Im(conj(l) f) of every amplitude: its sum, and signed by the register bits
            Sum all, bit[3];
            all.clear();
#pragma unroll
            for (int m = 0; m < 3; ++m) bit[m].clear();
            if (r.d1) tables(r, false, false);
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int x = t + j * TH;
                if (x >= dim) break;
                const T f = phi[x], l = lam[x];
                all.im(l, f, 1);
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    if ((PER >> m) > 1) bit[m].im(l, f, (j >> m) & 1 ? -1 : 1);
                if (r.d1) {
                    const T d = A::mul(tab_lo[x & 63], tab_hi[x >> 6]);
                    phi[x] = A::mul(f, d);
                    lam[x] = A::mul(l, d);
                }
            }
            red[0][t] = all.value();
#pragma unroll
            for (int m = 0; m < 3; ++m)
                if ((PER >> m) > 1) red[1 + m][t] = bit[m].value();
            __syncthreads();
            for (int w = warp; w < r.count; w += WARPS) {
                const BWire& bw = wire[r.first + w];
                if (bw.row[2] >= 0) {
                    const double z = bw.lb < LOG_TH ? row_sum(red[0], bw.lb) : row_sum(red[1 + bw.lb - LOG_TH], -1);
                    if (lane == 0) sums[C.row0 + bw.row[2]] = z;
                }
                if (bw.row[3] >= 0) {
                    const double z = row_sum(red[0], -1);
                    if (lane == 0) sums[C.row0 + bw.row[3]] = -z;
                }
            }
            __syncthreads();
            for (int w = 0; w < r.count; ++w) {
                const BWire& bw = wire[r.first + w];
                const int lb = bw.lb;
                const typename A::Rot rot(bw.c, bw.s);
                const bool nx = bw.row[0] >= 0, ny = bw.row[1] >= 0;
                Sum sx, sy;
                sx.clear();
                sy.clear();
                for (int p = t; p < dim / 2; p += TH) {
                    const int i0 = ((p >> lb) << (lb + 1)) | (p & ((1 << lb) - 1)), i1 = i0 | (1 << lb);
                    T f0 = phi[i0], f1 = phi[i1], l0 = lam[i0], l1 = lam[i1];
                    if (nx) {  // Im(l0* f1) + Im(l1* f0)
                        sx.im(l0, f1, 1);
                        sx.im(l1, f0, 1);
                    }
                    if (ny) {  // -Re(l0* f1) + Re(l1* f0)
                        sy.re(l0, f1, -1);
                        sy.re(l1, f0, 1);
                    }
                    A::rotate(f0, f1, rot);
                    A::rotate(l0, l1, rot);
                    phi[i0] = f0;
                    phi[i1] = f1;
                    lam[i0] = l0;
                    lam[i1] = l1;
                }
                // two wires' rows in turn: one warp adds a wire's up while the others go on
                double* rx = red[(w & 1) * 2];
                double* ry = red[(w & 1) * 2 + 1];
                if (nx) rx[t] = sx.value();
                if (ny) ry[t] = sy.value();
                __syncthreads();
                if (warp == w % WARPS) {
                    if (nx) {
                        const double v = row_sum(rx, -1);
                        if (lane == 0) sums[C.row0 + bw.row[0]] = v;
                    }
                    if (ny) {
                        const double v = row_sum(ry, -1);
                        if (lane == 0) sums[C.row0 + bw.row[1]] = v;
                    }
                }
            }
            if (r.d2) {
                tables(r, true, false);
                for (int x = t; x < dim; x += TH) {
                    diagonal(phi, x);
                    diagonal(lam, x);
                }
            }
            __syncthreads();
        }
    }
}

// Host tabulation of one op into controlled-2x2 / swap form.
static int to_bop(const qgpu_op& op, int n, BOp* out) {
    LocalGate lg;
    int st = tabulate(op, n, nullptr, 0, nullptr, 0, &lg);
    if (st != QGPU_OK) return st;
    std::memset(out, 0, sizeof(BOp));
    if (op.kind == QGPU_GATE_SWAP) {
        out->swap = 1;
        out->t = (uint8_t)(n - 1 - op.target);
        out->b2 = (uint8_t)(n - 1 - op.controls[0]);
        return QGPU_OK;
    }
    const int k = lg.k;
    const size_t d = (size_t)1 << k, call = (d - 1) & ~(size_t)1;
    out->t = (uint8_t)(n - 1 - op.target);
    for (int m = 0; m < k - 1; ++m) out->cm |= 1u << (n - 1 - lg.wires[m]);
    cd U[2][2];
    for (int lo = 0; lo < 2; ++lo)
        for (int in = 0; in < 2; ++in) U[lo][in] = lg.M[(call | in) * d + (call | lo)];
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) {
            out->u[2 * (2 * r + c)] = U[r][c].real();
            out->u[2 * (2 * r + c) + 1] = U[r][c].imag();
            out->v[2 * (2 * r + c)] = U[c][r].real();   // conjugate transpose
            out->v[2 * (2 * r + c) + 1] = -U[c][r].imag();
        }
    return QGPU_OK;
}

// One circuit of the shared-memory path: its records, and per rotation the rows and coefficients of
// its gradient.
struct BProgram {
    std::vector<BRec> recs;
    std::vector<BWire> wires;
    std::vector<BOp> gates;
    int rows = 0;
    std::vector<std::pair<int, std::pair<int, double>>> terms;  // (op, (row, coefficient))
};

// x^2 + y^2 - 1 of two numbers near the unit circle, without the rounding of the squares.
static double unit_error(double x, double y) {
    const double xx = x * x, yy = y * y, lo = std::fma(x, x, -xx) + std::fma(y, y, -yy);
    return (xx >= yy ? (xx - 1.0) + yy : (yy - 1.0) + xx) + lo;
}

static int lower_circuit(const qgpu_op* ops, int n_ops, int n, BProgram* out) {
    for (int g = 0; g < n_ops; ++g) {
        if (ops[g].kind == QGPU_GATE_CUSTOM)
            return fail(QGPU_ERR_NONUNITARY, "batched gradients need invertible gates; found a Custom gate");
        int k;
        int st = op_arity(ops[g], n, &k);
        if (st != QGPU_OK) return st;
    }
    double drift = 0.0;
    auto arity = [&](int g) {
        int k = 1;
        op_arity(ops[g], n, &k);
        return k;
    };
    for (int g = 0; g < n_ops;) {
        int e = g;
        BRec r;
        std::memset(&r, 0, sizeof(r));
        if (arity(g) == 1) {
            std::vector<std::vector<size_t>> gates(n);
            for (; e < n_ops && arity(e) == 1; ++e) gates[n - 1 - ops[e].target].push_back((size_t)e);
            r.kind = B_RUN;
            r.first = (int)out->wires.size();
            for (int b = 0; b < n; ++b) {
                if (gates[b].empty()) continue;
                std::reverse(gates[b].begin(), gates[b].end());
                PauliRun run;
                int st = pauli_run(ops, gates[b], n, &run);
                if (st != QGPU_OK) return st;
                const PauliFrame f = pauli_frame(&run);
                BWire w;
                std::memset(&w, 0, sizeof(w));
                w.lb = b;
                for (int m = 0; m < 4; ++m) w.row[m] = run.need[m + 1] ? out->rows++ : -1;
                for (const auto& rot : run.rots)
                    for (int m = 1; m <= 4; ++m)
                        if (rot.second[m] != 0.0)
                            out->terms.push_back({(int)rot.first, {w.row[m - 1], rot.second[m]}});
                // The norm's drift by the rounding of the constants, taken out as it arises.
                w.c = f.c - f.c * drift;
                w.s = f.s - f.s * drift;
                drift += 0.5 * unit_error(w.c, w.s) + 0.25 * unit_error(f.rho1.real(), f.rho1.imag()) +
                         0.25 * unit_error(f.rho2.real(), f.rho2.imag());
                w.rho1 = make_double2(f.rho1.real(), f.rho1.imag());
                w.rho2 = make_double2(f.rho2.real(), f.rho2.imag());
                r.d1 = r.d1 || f.rho1 != cd(1.0, 0.0);
                r.d2 = r.d2 || f.rho2 != cd(1.0, 0.0);
                out->wires.push_back(w);
            }
            r.count = (int)out->wires.size() - r.first;
            out->recs.push_back(r);
            g = e;
            continue;
        }
        for (; e < n_ops && arity(e) > 1; ++e) {}
        std::vector<uint64_t> fwd, rev;
        uint64_t fd = 0, rd = 0;
        std::vector<qgpu_op> back;
        for (int q = e; q-- > g;) back.push_back(inverse_op(ops[q]));
        if (e - g >= 2 && affine_columns(ops + g, e - g, n, &fwd, &fd) &&
            affine_columns(back.data(), back.size(), n, &rev, &rd)) {
            r.kind = B_MAP;
            for (int b = 0; b < n; ++b) {
                r.fwd[b] = (uint16_t)fwd[b];
                r.rev[b] = (uint16_t)rev[b];
            }
            r.fwd[BATCH_SMALL_BITS] = (uint16_t)fd;
            r.rev[BATCH_SMALL_BITS] = (uint16_t)rd;
            out->recs.push_back(r);
        } else {
            for (int q = g; q < e; ++q) {
                BOp o;
                int st = to_bop(ops[q], n, &o);
                if (st != QGPU_OK) return st;
                r.kind = B_GATE;
                r.first = (int)out->gates.size();
                r.count = 1;
                out->gates.push_back(o);
                out->recs.push_back(r);
            }
        }
        g = e;
    }
    return QGPU_OK;
}

// The small circuits of a batch: queued on streams of their own by start(), read back by finish().
struct SmallBatch {
    std::vector<size_t> items;        // batch items, largest circuits first
    std::vector<BProgram> progs;
    std::vector<size_t> row0;
    size_t rows = 0, out_at = 0, total = 0;
    uint8_t* dev = nullptr;
    cudaStream_t s = nullptr, s2 = nullptr;
    cudaEvent_t ready = nullptr;
    ~SmallBatch() {
        if (s) cudaStreamSynchronize(s);  // (nothing of it is in flight when the memory goes)
        if (s2) cudaStreamSynchronize(s2);
        if (ready) cudaEventDestroy(ready);
        if (s) cudaStreamDestroy(s);
        if (s2) cudaStreamDestroy(s2);
        if (dev) cudaFree(dev);
    }
    int start(const qgpu_batch_item* all, const qgpu_op* ops, const double* obs, size_t n_obs, int precision,
              int small_max, int sm_count);
    int finish(const qgpu_batch_item* all, double* energies, double* grads);
};

template <class A, int TH, int PER, int CTAS>
static cudaError_t launch_small(const uint8_t* dev, const size_t* at, int first, int count, int bits, int sm_count,
                                unsigned* counter, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    const size_t smem = 2 * sizeof(typename A::T) << bits;
    const BCirc* c = (const BCirc*)(dev + at[0]) + first;
    double* energy = (double*)(dev + at[5]) + first;
    k_batch_small<A, TH, PER, CTAS><<<std::min(count, sm_count * CTAS), TH, smem, s>>>(
        c, count, (const BRec*)(dev + at[1]), (const BWire*)(dev + at[2]), (const BOp*)(dev + at[3]),
        (const double*)(dev + at[4]), energy, (double*)(dev + at[6]), counter, bits);
    return cudaGetLastError();
}

int SmallBatch::start(const qgpu_batch_item* all, const qgpu_op* ops, const double* obs, size_t n_obs,
                      int precision, int small_max, int sm_count) {
    std::stable_sort(items.begin(), items.end(),
                     [&](size_t x, size_t y) { return all[x].n_qubits > all[y].n_qubits; });
    progs.resize(items.size());
    std::vector<BCirc> circs;
    size_t nrec = 0, nwire = 0, nop = 0;
    int wide = 0;  // circuits that take the large CTAs
    for (size_t q = 0; q < items.size(); ++q) {
        const qgpu_batch_item& it = all[items[q]];
        int st = lower_circuit(ops + it.op_offset, it.n_ops, it.n_qubits, &progs[q]);
        if (st != QGPU_OK) return st;
        BCirc c;
        c.n = it.n_qubits;
        c.nrec = (int)progs[q].recs.size();
        c.rec0 = (int64_t)nrec;
        c.wire0 = (int64_t)nwire;
        c.op0 = (int64_t)nop;
        c.obs0 = it.obs_offset;
        c.row0 = (int64_t)rows;
        row0.push_back(rows);
        nrec += progs[q].recs.size();
        nwire += progs[q].wires.size();
        nop += progs[q].gates.size();
        rows += progs[q].rows;
        wide += it.n_qubits > BATCH_NARROW_BITS;
        circs.push_back(c);
    }
    // one device buffer: circuits | records | wires | gates | observables | energies | row sums | counters
    size_t at[8], end = 0;
    auto reserve = [&](int k, size_t bytes) {
        at[k] = end;
        end = (end + bytes + 255) / 256 * 256;
    };
    reserve(0, circs.size() * sizeof(BCirc));
    reserve(1, nrec * sizeof(BRec));
    reserve(2, nwire * sizeof(BWire));
    reserve(3, nop * sizeof(BOp));
    reserve(4, n_obs * sizeof(double));
    const size_t in_bytes = end;
    reserve(5, circs.size() * sizeof(double));
    reserve(6, rows * sizeof(double));
    reserve(7, 2 * sizeof(unsigned));
    out_at = at[5];
    total = end;
    std::vector<uint8_t> host(in_bytes, 0);
    std::memcpy(host.data() + at[0], circs.data(), circs.size() * sizeof(BCirc));
    size_t r = 0, w = 0, o = 0;
    for (const BProgram& p : progs) {
        auto put = [&](size_t to, const void* src, size_t bytes) { if (bytes) std::memcpy(host.data() + to, src, bytes); };
        put(at[1] + r * sizeof(BRec), p.recs.data(), p.recs.size() * sizeof(BRec));
        put(at[2] + w * sizeof(BWire), p.wires.data(), p.wires.size() * sizeof(BWire));
        put(at[3] + o * sizeof(BOp), p.gates.data(), p.gates.size() * sizeof(BOp));
        r += p.recs.size();
        w += p.wires.size();
        o += p.gates.size();
    }
    std::memcpy(host.data() + at[4], obs, n_obs * sizeof(double));
    QGPU_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    QGPU_CUDA(cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking));
    QGPU_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    QGPU_CUDA(cudaMalloc((void**)&dev, total));
    QGPU_CUDA(cudaMemcpyAsync(dev, host.data(), in_bytes, cudaMemcpyHostToDevice, s));
    const int count = (int)circs.size();
    const size_t esz = precision == QGPU_C128 ? 16 : 8;
    if (precision == QGPU_C128) QGPU_CUDA(smem_opt_in((const void*)k_batch_small<B128, 1024, 4, 1>, 2 * esz << small_max));
    else QGPU_CUDA(smem_opt_in((const void*)k_batch_small<B64, 1024, 8, 1>, 2 * esz << small_max));
    // counters reset, then both persistent kernels side by side
    unsigned* counters = (unsigned*)(dev + at[7]);
    QGPU_CUDA(cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned), s));
    QGPU_CUDA(cudaEventRecord(ready, s));
    QGPU_CUDA(cudaStreamWaitEvent(s2, ready, 0));
    if (precision == QGPU_C128) {
        QGPU_CUDA((launch_small<B128, 1024, 4, 1>(dev, at, 0, wide, small_max, sm_count, counters, s)));
        QGPU_CUDA((launch_small<B128, 256, 4, 4>(dev, at, wide, count - wide, BATCH_NARROW_BITS, sm_count,
                                                 counters + 1, s2)));
    } else {
        QGPU_CUDA((launch_small<B64, 1024, 8, 1>(dev, at, 0, wide, small_max, sm_count, counters, s)));
        QGPU_CUDA((launch_small<B64, 256, 4, 4>(dev, at, wide, count - wide, BATCH_NARROW_BITS, sm_count,
                                                counters + 1, s2)));
    }
    return QGPU_OK;
}

int SmallBatch::finish(const qgpu_batch_item* all, double* energies, double* grads) {
    std::vector<uint8_t> out(total - out_at);
    QGPU_CUDA(cudaEventRecord(ready, s2));
    QGPU_CUDA(cudaStreamWaitEvent(s, ready, 0));
    QGPU_CUDA(cudaMemcpyAsync(out.data(), dev + out_at, out.size(), cudaMemcpyDeviceToHost, s));
    QGPU_CUDA(cudaStreamSynchronize(s));
    const double* energy = (const double*)out.data();
    const double* sums = (const double*)(out.data() + (items.size() * sizeof(double) + 255) / 256 * 256);
    for (size_t q = 0; q < items.size(); ++q) {
        const qgpu_batch_item& it = all[items[q]];
        energies[items[q]] = energy[q];
        double* g = grads + it.grad_offset;
        std::fill(g, g + it.n_ops, 0.0);
        for (const auto& t : progs[q].terms) g[t.first] += t.second.second * sums[row0[q] + t.second.first];
    }
    return QGPU_OK;
}

}  // namespace qgpu

using namespace qgpu;

extern "C" int qgpu_batch_run(const qgpu_batch_item* items, size_t n_items, const qgpu_op* ops,
                              size_t n_ops_total, const double* obs, size_t n_obs, int precision,
                              double* energies, double* grads, int* tuned_budget) {
    if (!items || !ops || !obs || !energies || !grads)
        return fail(QGPU_ERR_INVALID, "qgpu_batch_run: NULL argument");
    if (precision != QGPU_C128 && precision != QGPU_C64)
        return fail(QGPU_ERR_INVALID, "qgpu_batch_run: precision must be QGPU_C128 or QGPU_C64");
    const int small_max = precision == QGPU_C128 ? 12 : 13;
    if (tuned_budget)
        for (int q = 0; q <= BATCH_MAX_Q; ++q) tuned_budget[q] = 0;
    // ---- validate and split
    std::vector<size_t> small, large;
    for (size_t i = 0; i < n_items; ++i) {
        const qgpu_batch_item& it = items[i];
        if (it.n_qubits < 1 || it.n_qubits > BATCH_MAX_Q || it.n_ops < 0 || it.op_offset < 0 ||
            (size_t)(it.op_offset + it.n_ops) > n_ops_total || it.obs_offset < 0 ||
            (size_t)(it.obs_offset + 2 * it.n_qubits) > n_obs || it.grad_offset < 0)
            return fail(QGPU_ERR_INVALID, "qgpu_batch_run: item " + std::to_string(i) + " out of range");
        (it.n_qubits <= small_max ? small : large).push_back(i);
    }
    int dev = 0;
    QGPU_CUDA(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    QGPU_CUDA(cudaGetDeviceProperties(&prop, dev));
    // ---- small circuits: persistent launches, beside the large ones
    SmallBatch sb;
    if (!small.empty()) {
        sb.items = small;
        int st = sb.start(items, ops, obs, n_obs, precision, small_max, prop.multiProcessorCount);
        if (st != QGPU_OK) return st;
    }
    if (large.empty()) return small.empty() ? QGPU_OK : sb.finish(items, energies, grads);
    // ---- large circuits: one after another on W host threads, each with a handle (and so a stream)
    // of its own, largest first from a shared counter, so that the launch and synchronisation
    // overhead of medium circuits overlaps with other circuits' kernels. A thread's handle keeps
    // its buffers from circuit to circuit (an allocation or a free between them waits for the
    // whole device). 34 complex128 circuits of 13 to 16 qubits: 14.3 -> 7.7 ms; 32 of 17 to 20
    // qubits: 29 -> 16.7 ms (2 threads 10.6 and 19.5, 8 threads 8.3 and 18.7).
    std::stable_sort(large.begin(), large.end(), [&](size_t x, size_t y) {
        return items[x].n_qubits > items[y].n_qubits;
    });
    const char* env = std::getenv("QGPU_BATCH_WORKERS");
    const int workers = std::max(1, std::min(16, env ? std::atoi(env) : 4));
    std::atomic<size_t> next{0};
    std::atomic<int> first_err{QGPU_OK};
    std::string err_msg;
    std::mutex err_mu;
    auto failed = [&](int st, const std::string& msg) {
        int expect = QGPU_OK;
        if (first_err.compare_exchange_strong(expect, st)) {
            std::lock_guard<std::mutex> lk(err_mu);
            err_msg = msg;
        }
    };
    auto enter = [&]() {  // handles are created on the thread's current device
        const cudaError_t e = cudaSetDevice(dev);
        if (e != cudaSuccess) failed(cuda_fail(e, "cudaSetDevice"), qgpu_last_error());
        return e == cudaSuccess;
    };
    auto work = [&]() {
        qgpu_handle* h = nullptr;
        for (;;) {
            if (first_err.load() != QGPU_OK) break;
            const size_t q = next.fetch_add(1);
            if (q >= large.size()) break;
            const size_t i = large[q];
            const qgpu_batch_item& it = items[i];
            int st = QGPU_OK;
            if (!h) st = qgpu_create(it.n_qubits, precision, &h);  // (its largest circuit)
            if (st == QGPU_OK) {
                h->n_qubits = it.n_qubits;
                h->dim = 1ull << it.n_qubits;
                st = qgpu_set_zero(h);
                if (tuned_budget) {
                    std::lock_guard<std::mutex> lk(err_mu);
                    tuned_budget[it.n_qubits] = plan_options_for(h).budget + 65536;  // (grouped sweep)
                }
            }
            if (st == QGPU_OK)
                st = qgpu_adjoint_grad(h, ops + it.op_offset, (size_t)it.n_ops, nullptr, 0, nullptr, 0,
                                       obs + it.obs_offset, obs + it.obs_offset + it.n_qubits,
                                       &energies[i], grads + it.grad_offset);
            if (st != QGPU_OK) {
                failed(st, qgpu_last_error());
                break;
            }
        }
        if (h) qgpu_destroy(h);
    };
    run_workers(workers, enter, work);
    if (first_err.load() != QGPU_OK) return fail(first_err.load(), err_msg);
    return small.empty() ? QGPU_OK : sb.finish(items, energies, grads);
}
