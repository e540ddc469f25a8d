// wide.cuh — wide passes (WidePass, plan.h): many gates per read and write of the register.
// Included by program.cu after the arithmetic policies.
//
// A CTA stages a tile of the register in shared memory: the 2^K amplitudes that share every bit
// outside the pass's K tile bits. The pass's steps run in rounds: in each, a thread holds the 2^R
// amplitudes that differ in the round's R bits in registers, applies the round's steps and writes
// them back. Steps that only read a bit (controls, phases) do not need it in the tile. X, CNot and
// Swap on tile bits move nothing: the slot of an amplitude is a linear function of its index over
// GF(2), kept as one vector per bit, and they change the vectors.
// Rotations and pair blocks are straight-line code per register bit: with one dispatch per gate
// the selects and register moves around it took more issue slots than the arithmetic (57 % of the
// ALU pipe against 41 % of the FMA pipe).
// Against register-tile passes (k_tile, k_pair2) a wide pass does the work of three to ten of
// them per trip through HBM (complex64) and per launch (small registers). Bound: arithmetic and
// issue, the FMA pipe at 42 to 56 % of its cycles (24 qubits, complex128) and 29 to 48 %
// (complex64, 29 to 36 % where every round is a pair block); DRAM at 13 to 28 %.
// Measured, tile against wide passes, time on the GPU: 17 qubits of complex128, 40 random columns
// 352 / 107 us (47 / 6 launches); 16-qubit ansatz, 4 layers 320 / 110 us; complex64 at 24 qubits 3.56 /
// 1.5 ms; complex64 at 30 qubits, 4 brickwork layers 53.2 / 43.0 ms.
#pragma once

namespace qgpu {

constexpr int WIDE_RBITS_MAX = 4;

// A pass's program: rounds, steps and constants, uploaded with the plan and copied to shared
// memory by each CTA (read from the parameter bank, whose indexed loads take the address unit,
// they bounded the kernel: 77 % of that pipe, 1382 against 321 us per 26-qubit complex64 pass).
struct WideStepD {
    uint8_t type, m, m2;   // StepType; register bits
    uint8_t rcm;           // controls: register bits,
    uint16_t xcm;          // other tile bits (tile index mask)
    uint16_t at;           // first constant
    uint64_t ocm;          // and bits outside the tile
    uint8_t u0, u1, unit, pad0;
    uint32_t pad;
    uint64_t pad2;
};
static_assert(sizeof(WideStepD) == 32, "steps are copied in 16-byte pieces");
enum : uint8_t { WIDE_PRE = 1, WIDE_REAL = 2, WIDE_DENSE = 4, WIDE_POST = 8 };
struct WideRoundD {
    // where the round's amplitudes lie in the shared tile: an XOR of a vector per set bit of the
    // thread (tc) and register (rc) index and of the index bits obits outside the tile (ov)
    uint16_t rc[WIDE_RBITS_MAX], tc[8], c0;
    uint16_t first, count;              // other steps
    uint16_t rot_at[WIDE_RBITS_MAX], pair_at[2];
    uint16_t ov[WIDE_MAX_OUTSIDE];
    uint8_t rot[WIDE_RBITS_MAX];        // WIDE_* parts of each register bit's rotation
    uint8_t pairs;                      // bit k: a pair block on register bits 2k, 2k + 1
    uint8_t rl[WIDE_RBITS_MAX], tl[8];  // tile bit of each register and thread bit
    uint8_t pad[13];
};
static_assert(sizeof(WideRoundD) == 96, "rounds are copied in 16-byte pieces");
struct WideParams {
    uint64_t ngroups;
    const float4* tab_ff;
    const uint4* prog;     // rounds | steps | constants
    int prog_bytes, steps_at, consts_at;
    int nbits, tile;       // tile bits; log2 of the shared tile (at least R: the rest stays zero)
    int nfields;           // runs of index bits outside the tile: g's bits from src go to dst on
    int nruns;             // runs of tile bits: tile index bits from rsrc go to rdst on
    int nrounds;           // and one more record: where the tile lies after them
    int nout;
    uint8_t obits[WIDE_MAX_OUTSIDE];
    uint8_t bits[MAX_WIDE_BITS];
    uint8_t src[MAX_WIDE_BITS + 1], dst[MAX_WIDE_BITS + 1];
    uint8_t rsrc[MAX_WIDE_BITS], rdst[MAX_WIDE_BITS];
    uint16_t run[MAX_WIDE_BITS];
    uint64_t field[MAX_WIDE_BITS + 1];
};

// ---- arithmetic on the packed values of a round ---------------------------------------------
struct WideFF {
    using V = ffp;
    static constexpr int R = 3, TBITS = 7, RBITS = 3, CTAS = 4;
    static constexpr int FACTOR = 8, REAL = 16;  // constants of a phase, of a real 2x2
    static __device__ __forceinline__ V zero() { return V{0, 0}; }
    static __device__ __forceinline__ void real(V& a, V& b, const u64* c) {
        PDot2 d;
        V o0, o1;
        d.first3(c + 0, a.h, a.l);
        d.add3(c + 4, b.h, b.l);
        d.result(o0.h, o0.l);
        d.first3(c + 8, a.h, a.l);
        d.add3(c + 12, b.h, b.l);
        d.result(o1.h, o1.l);
        a = o0;
        b = o1;
    }
    static __device__ __forceinline__ void dense(V& a, V& b, const u64* c) { ff_dense(a, b, c); }
    static __device__ __forceinline__ void mul(V& a, const u64* c) {
        PDot2 d;
        d.first3(c, a.h, a.l);
        d.add3(c + 4, pswap(a.h), pswap(a.l));
        d.result(a.h, a.l);
    }
    static __device__ __forceinline__ void unit(V& a, int code) { unit_mul(a, code); }
    static __device__ __forceinline__ void table(V& a, const float4* tab, uint32_t e) {
        const float4 v = __ldg(tab + e);
        const u64 c[8] = {p2(v.x, v.x), p2(v.y, v.y), p2(-v.x, -v.x), p2(-v.y, -v.y),
                          p2(-v.z, v.z), p2(-v.w, v.w), p2(v.z, -v.z), p2(v.w, -v.w)};
        PolFF::mul_pk(a, c);
    }
    template <int M>
    static __device__ __forceinline__ void pair(V* v, const u64* c) {  // register bits 0, 1
        ff_pair(v, c);
        ff_pair(v + 4, c);
    }
};

struct WideF32 {
    using V = u64;
    static constexpr int R = 4, TBITS = 7, RBITS = 4, CTAS = 4;
    static constexpr int FACTOR = 4, REAL = 8;
    static __device__ __forceinline__ V zero() { return 0; }
    // constants as (hi, lo) pairs of floats, so that only the amplitudes are rounded to f32
    static __device__ __forceinline__ void real(V& a, V& b, const u64* c) {
        const V o0 = pfma(c[0], a, pfma(c[2], b, pfma(c[1], a, pmul(c[3], b))));
        const V o1 = pfma(c[4], a, pfma(c[6], b, pfma(c[5], a, pmul(c[7], b))));
        a = o0;
        b = o1;
    }
    // a + i b for the packed sums a, b of the products with real and imaginary parts
    static __device__ __forceinline__ V turn(V a, V b) {
        float ax, ay, bx, by;
        up2(a, ax, ay);
        up2(b, bx, by);
        return p2(ax - by, ay + bx);
    }
    // c: per entry re (hi, lo), im (hi, lo)
    static __device__ __forceinline__ V row(V a, V b, const u64* c) {
        return turn(pfma(c[0], a, pfma(c[4], b, pfma(c[1], a, pmul(c[5], b)))),
                    pfma(c[2], a, pfma(c[6], b, pfma(c[3], a, pmul(c[7], b)))));
    }
    static __device__ __forceinline__ void dense(V& a, V& b, const u64* c) {
        const V o0 = row(a, b, c), o1 = row(a, b, c + 8);
        a = o0;
        b = o1;
    }
    static __device__ __forceinline__ void mul(V& a, const u64* c) {
        a = turn(pfma(c[0], a, pmul(c[1], a)), pfma(c[2], a, pmul(c[3], a)));
    }
    static __device__ __forceinline__ void unit(V& a, int code) {
        float2 v;
        up2(a, v.x, v.y);
        unit_mul(v, code);
        a = p2(v.x, v.y);
    }
    static __device__ __forceinline__ void table(V& a, const float4* tab, uint32_t e) {
        const float4 v = __ldg(tab + e);
        const u64 c[4] = {p2(v.x, v.x), p2(v.y, v.y), p2(v.z, v.z), p2(v.w, v.w)};
        mul(a, c);
    }
    // register bits M, M + 1: row by row over all quads, so that a row's constants load once
    template <int M>
    static __device__ __forceinline__ void pair(V* v, const u64* c) {
        V o[1 << R];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            u64 k[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2 e = reinterpret_cast<const ulonglong2*>(c)[4 * r + q];
                k[2 * q] = e.x;
                k[2 * q + 1] = e.y;
            }
#pragma unroll
            for (int g = 0; g < (1 << R) / 4; ++g) {
                const int i = M == 0 ? 4 * g : g;
                V a = pmul(k[0], v[i]), b = pmul(k[1], v[i]);
#pragma unroll
                for (int q = 1; q < 4; ++q) {
                    a = pfma(k[2 * q], v[i | (q << M)], a);
                    b = pfma(k[2 * q + 1], v[i | (q << M)], b);
                }
                o[i | (r << M)] = turn(a, b);
            }
        }
#pragma unroll
        for (int q = 0; q < (1 << R); ++q) v[q] = o[q];
    }
};

// Shared-memory slot of tile index l (linear in its bits): a round's gather leaves out R bits of
// l; higher bits folded into the lowest ones keep the lanes that share a wavefront (8 of 16 bytes,
// 16 of 8 bytes) on distinct banks for nearly every round.
template <class A>
__host__ __device__ __forceinline__ int wide_slot(int l) {
    if constexpr (sizeof(typename A::V) == 16)
        return l ^ ((l >> 3) & 1 ? 3 : 0) ^ ((l >> 4) & 1 ? 5 : 0) ^ ((l >> 5) & 1 ? 6 : 0);
    else
        return l ^ ((l >> 4) & 1 ? 3 : 0) ^ ((l >> 5) & 1 ? 5 : 0) ^ ((l >> 6) & 1 ? 9 : 0) ^
               ((l >> 7) & 1 ? 14 : 0);
}

// The rotation of register bit M: phase, 2x2, phase, each where present.
template <class A, int M>
__device__ __forceinline__ void wide_rotate(typename A::V* v, int parts, const u64* c) {
    constexpr int Q = 1 << A::R;
    if (parts & WIDE_PRE) {
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if ((i >> M) & 1) A::mul(v[i], c);
        c += A::FACTOR;
    }
    if (parts & WIDE_REAL) {
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if (!((i >> M) & 1)) A::real(v[i], v[i | (1 << M)], c);
        c += A::REAL;
    }
    if (parts & WIDE_DENSE) {
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if (!((i >> M) & 1)) A::dense(v[i], v[i | (1 << M)], c);
        c += 2 * A::REAL;
    }
    if (parts & WIDE_POST) {
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if ((i >> M) & 1) A::mul(v[i], c);
    }
}

// Other steps: controlled 2x2s, phases, tables, swaps.
template <class A, int M>
__device__ __forceinline__ void wide_2x2(typename A::V* v, const WideStepD& s, const u64* c) {
    constexpr int Q = 1 << A::R;
    const int type = s.type, rcm = s.rcm, u0 = s.u0, u1 = s.u1;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        if ((i >> M) & 1 || (i & rcm) != rcm) continue;
        const int k = i | (1 << M);
        if (type == ST_REAL) {
            A::real(v[i], v[k], c);
        } else if (type == ST_DENSE) {
            A::dense(v[i], v[k], c);
        } else if (type == ST_PERM) {  // antidiagonal
            const typename A::V t = v[i];
            v[i] = v[k];
            v[k] = t;
            A::unit(v[i], u0);
            A::unit(v[k], u1);
        }
    }
}

template <class A>
__device__ __noinline__ void wide_other(typename A::V* v, const WideStepD& s, const u64* c,
                                        const WideParams& p, uint64_t base, int l0, const int* lr) {
    constexpr int R = A::R, Q = 1 << R;
    const int type = s.type, m = s.m, rcm = s.rcm;
    if (type <= ST_PERM) {
        if (m == 0) wide_2x2<A, 0>(v, s, c);
        else if (m == 1) wide_2x2<A, 1>(v, s, c);
        else if (m == 2) wide_2x2<A, 2>(v, s, c);
        if constexpr (R > 3) if (m == 3) wide_2x2<A, 3>(v, s, c);
        return;
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        if ((i & rcm) != rcm) continue;
        if (type == ST_DIAG) {
            const int bit = (i >> m) & 1;
            if (s.unit) A::unit(v[i], bit ? s.u1 : s.u0);
            else A::mul(v[i], c + bit * A::FACTOR);
        } else if (type == ST_PHASE) {
            if (s.unit) A::unit(v[i], s.u0);
            else A::mul(v[i], c);
        } else {  // ST_TABLE: m fields, c[f] = offset | shift << 32 | width << 40
            int l = l0;
#pragma unroll
            for (int e = 0; e < R; ++e) l |= (i >> e) & 1 ? lr[e] : 0;
            uint64_t idx = base;
            for (int f = 0; f < p.nruns; ++f)
                idx |= (uint64_t)((l >> p.rsrc[f]) & p.run[f]) << p.rdst[f];
            for (int f = 0; f < m; ++f) {
                const u64 d = c[f];
                const uint32_t y = (uint32_t)(idx >> ((d >> 32) & 255)) &
                                   ((1u << (uint32_t)(d >> 40)) - 1u);
                A::table(v[i], p.tab_ff, (uint32_t)d + y);
            }
        }
    }
}

template <class A, class P>
__global__ void __launch_bounds__(1 << A::TBITS, A::CTAS)
k_wide(typename P::S* __restrict__ st, const __grid_constant__ WideParams p) {
    using V = typename A::V;
    constexpr int R = A::R, Q = 1 << R, TH = 1 << A::TBITS, PER = 1 << A::RBITS;
    static_assert(A::R == A::RBITS, "a round takes the whole tile");
    extern __shared__ __align__(16) unsigned char wide_smem[];
    V* tile = reinterpret_cast<V*>(wide_smem);
    uint4* prog = reinterpret_cast<uint4*>(tile + (PER << A::TBITS));
    const WideRoundD* rounds = reinterpret_cast<const WideRoundD*>(prog);
    const WideStepD* steps = reinterpret_cast<const WideStepD*>((unsigned char*)prog + p.steps_at);
    const u64* consts = reinterpret_cast<const u64*>((unsigned char*)prog + p.consts_at);
    const int t = threadIdx.x;
    for (int i = t; i < p.prog_bytes / 16; i += TH) prog[i] = __ldg(p.prog + i);
    const int T = 1 << p.nbits;
    uint64_t off_t = 0;
    for (int m = 0; m < p.nbits && m < A::TBITS; ++m)
        if ((t >> m) & 1) off_t |= 1ull << p.bits[m];
    uint64_t off_j[A::RBITS];
#pragma unroll
    for (int m = 0; m < A::RBITS; ++m)
        off_j[m] = A::TBITS + m < p.nbits ? 1ull << p.bits[A::TBITS + m] : 0;
    auto offset = [&](int j) {
        uint64_t o = 0;
#pragma unroll
        for (int m = 0; m < A::RBITS; ++m)
            if ((j >> m) & 1) o |= off_j[m];
        return o;
    };
    if (t >= T && t < (1 << p.tile)) tile[wide_slot<A>(t)] = A::zero();
    const bool active = t < ((1 << p.tile) >> R);
    __syncthreads();  // the program is in place
    for (uint64_t g = blockIdx.x; g < p.ngroups; g += gridDim.x) {
        uint64_t base = 0;
        for (int f = 0; f < p.nfields; ++f) base |= (g >> p.src[f]) << p.dst[f] & p.field[f];
        // this thread's first slot of a round
        auto first_slot = [&](const WideRoundD& rd) {
            int a = rd.c0;
#pragma unroll
            for (int k = 0; k < A::TBITS; ++k)
                if ((t >> k) & 1) a ^= rd.tc[k];
            for (int e = 0; e < p.nout; ++e)
                if ((base >> p.obits[e]) & 1ull) a ^= rd.ov[e];
            return a;
        };
        if (t < T) {
            typename P::S raw[PER];
            const typename P::S* src = st + base + off_t;
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (t + j * TH < T) raw[j] = src[offset(j)];
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (t + j * TH < T) tile[wide_slot<A>(t + j * TH)] = P::load(raw[j]);
        }
        __syncthreads();
        for (int r = 0; r < p.nrounds; ++r) {
            const WideRoundD& rd = rounds[r];
            if (active) {
                int at[Q];
                at[0] = first_slot(rd);
#pragma unroll
                for (int i = 1; i < Q; ++i)
                    at[i] = at[i & (i - 1)] ^ rd.rc[i & 1 ? 0 : i & 2 ? 1 : i & 4 ? 2 : 3];
                V v[Q];
#pragma unroll
                for (int i = 0; i < Q; ++i) v[i] = tile[at[i]];
                if (rd.rot[0]) wide_rotate<A, 0>(v, rd.rot[0], consts + rd.rot_at[0]);
                if (rd.rot[1]) wide_rotate<A, 1>(v, rd.rot[1], consts + rd.rot_at[1]);
                if (rd.rot[2]) wide_rotate<A, 2>(v, rd.rot[2], consts + rd.rot_at[2]);
                if constexpr (R > 3)
                    if (rd.rot[3]) wide_rotate<A, 3>(v, rd.rot[3], consts + rd.rot_at[3]);
                if (rd.pairs & 1) A::template pair<0>(v, consts + rd.pair_at[0]);
                if constexpr (R > 3)
                    if (rd.pairs & 2) A::template pair<2>(v, consts + rd.pair_at[1]);
                if (rd.count) {
                    int l0 = 0, lr[R];  // tile index of the thread, and of each register bit
#pragma unroll
                    for (int k = 0; k < A::TBITS; ++k)
                        if ((t >> k) & 1) l0 |= 1 << rd.tl[k];
#pragma unroll
                    for (int m = 0; m < R; ++m) lr[m] = 1 << rd.rl[m];
                    V w[Q];  // (wide_other is a call: its array lives in local memory)
#pragma unroll
                    for (int i = 0; i < Q; ++i) w[i] = v[i];
                    for (int k = rd.first; k < rd.first + rd.count; ++k) {
                        const WideStepD& s = steps[k];
                        if ((base & s.ocm) != s.ocm) continue;  // (the same for the whole tile)
                        if ((l0 & s.xcm) != s.xcm) continue;
                        wide_other<A>(w, s, consts + s.at, p, base, l0, lr);
                    }
#pragma unroll
                    for (int i = 0; i < Q; ++i) v[i] = w[i];
                }
#pragma unroll
                for (int i = 0; i < Q; ++i) tile[at[i]] = v[i];
            }
            __syncthreads();
        }
        if (t < T) {
            const WideRoundD& rd = rounds[p.nrounds];
            const int a = first_slot(rd);
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                if (t + j * TH >= T) break;
                int at = a;
#pragma unroll
                for (int m = 0; m < A::RBITS; ++m)
                    if ((j >> m) & 1) at ^= rd.rc[m];
                st[(base | off_t) + offset(j)] = P::store(tile[at]);
            }
        }
        __syncthreads();  // (moves may leave a thread's next slots to other readers)
    }
}

// complex64 values as packed registers
struct PolPackedF32 {
    using S = float2;
    using R = u64;
    static __device__ __forceinline__ R load(S a) { return p2(a.x, a.y); }
    static __device__ __forceinline__ S store(R v) {
        S a;
        up2(v, a.x, a.y);
        return a;
    }
};

// ---- host side ----------------------------------------------------------------------------------
static u64 wide_pack(float x, float y) {
    uint32_t a, b;
    std::memcpy(&a, &x, 4);
    std::memcpy(&b, &y, 4);
    return (u64)a | ((u64)b << 32);
}

// A step's constants. Rounding an unconditional 2x2 or 4x4 changes the register's norm a little
// (f64 rounding already does: 1e-14 over 200 rotations): *drift is the relative change so far, and
// the next such step takes it out before it is rounded, so that it does not grow with the gates.
// A step of library gates is unitary but for its rounding; what a Custom gate's entries are off a
// unitary matrix belongs to the gate, so there only the entries' split into floats counts (240 gates
// scaling by 1 - 6.7e-14 each otherwise came out as if they did not).
template <class A>
static std::vector<u64> wide_constants(const Plan& plan, const WideStep& ws, double* drift) {
    constexpr bool ff = sizeof(typename A::V) == 16;
    const DevStep& s = ws.s;
    std::vector<cd> e;
    switch (s.type) {
        case ST_REAL:
        case ST_DENSE: for (int k = 0; k < 4; ++k) e.emplace_back(s.d[2 * k], s.d[2 * k + 1]); break;
        case ST_PHASE: if (!s.unit) e.emplace_back(s.d[0], s.d[1]); break;
        case ST_DIAG:
            for (int k = 0; k < 2 && !s.unit; ++k) e.emplace_back(s.d[2 * k], s.d[2 * k + 1]);
            break;
        case ST_DENSE4:
            for (int r = 0; r < 4; ++r)
                for (int q = 0; q < 4; ++q) e.push_back(plan.pairs[ws.pair].m[r][q]);
            break;
        default: break;
    }
    std::vector<u64> c;
    if (s.type == ST_TABLE) {
        for (int f = 0; f < s.nfields; ++f)
            c.push_back((u64)s.tab_off[f] | ((u64)s.tab_shift[f] << 32) | ((u64)s.tab_width[f] << 40));
    }
    const bool pair32 = !ff && s.type == ST_DENSE4;  // (complex64 pair blocks: hi alone)
    const bool whole = s.cm == 0 && (s.type == ST_REAL || s.type == ST_DENSE || s.type == ST_DENSE4);
    const bool third_kept = ff && s.type != ST_DENSE && s.type != ST_DENSE4;
    const bool given = s.given || (s.type == ST_DENSE4 && plan.pairs[ws.pair].given);
    const bool phase = s.type == ST_PHASE && !s.unit && __builtin_popcountll(s.cm) == 1;
    // sums of x^2 over the entries, of its rounding, and of x'^2 - x^2 for the entries x' uploaded
    double size = 0.0, exact = 0.0, change = 0.0;
    auto part = [&](double x, float* h, float* l, float* third) {
        const double y = whole ? x - x * *drift : x;
        *h = (float)y;
        *l = pair32 ? 0.0f : (float)(y - (double)*h);
        *third = (float)((y - (double)*h) - (double)*l);
        if (!whole && !phase) return;
        const double kept = ((double)*h + (double)*l) + (third_kept ? (double)*third : 0.0);
        change += (kept - x) * (kept + x);
        const double sq = x * x, sum = size + sq, b = sum - size;
        exact += std::fma(x, x, -sq) + ((size - (sum - b)) + (sq - b));
        size = sum;
    };
    auto term = [&](float h, float l, float third, bool mixed) {  // hi, -third, -hi, -lo
        const float s0 = mixed ? -1.0f : 1.0f;  // (the real lane of an imaginary part)
        c.push_back(wide_pack(s0 * h, h));
        c.push_back(wide_pack(-s0 * third, -third));
        c.push_back(wide_pack(-s0 * h, -h));
        c.push_back(wide_pack(-s0 * l, -l));
    };
    for (cd z : e) {
        float rh, rl, r3, ih, il, i3;
        part(z.real(), &rh, &rl, &r3);
        part(z.imag(), &ih, &il, &i3);
        if (ff) {
            term(rh, rl, r3, false);
            if (s.type != ST_REAL) term(ih, il, i3, true);
        } else {
            c.push_back(wide_pack(rh, rh));
            if (!pair32) c.push_back(wide_pack(rl, rl));
            if (s.type != ST_REAL) c.push_back(wide_pack(ih, ih));
            if (s.type != ST_REAL && !pair32) c.push_back(wide_pack(il, il));
        }
    }
    // sum |e|^2 of a unitary d x d matrix is d (sizes that are not finite count for nothing)
    const double d = given ? size : s.type == ST_DENSE4 ? 4.0 : s.type == ST_PHASE ? 1.0 : 2.0;
    const double off = given ? 0.0 : (size - d) + exact;
    const bool known = given ? size > 0.0 && size < HUGE_VAL : std::fabs(size - d) < 1e-12;
    if (whole && known) *drift += 0.5 * (off + change) / d;
    if (phase && known) *drift += 0.25 * (off + change) / d;  // (half the amplitudes)
    if (c.size() & 1) c.push_back(0);  // 16-byte aligned
    return c;
}

// The parameters and the program (appended to `prog`, 16-byte aligned) of one pass.
template <class A>
static void wide_fill(const Plan& plan, const WidePass& w, int n, uint64_t dim, WideParams* p,
                      std::vector<uint8_t>* prog, double* drift) {
    std::memset(p, 0, sizeof(*p));
    int local[64];
    for (int b = 0, at = 0; b < n; ++b) {
        if ((w.mask >> b) & 1ull) {
            if (p->nruns == 0 || b == 0 || !((w.mask >> (b - 1)) & 1ull)) {
                p->rsrc[p->nruns] = (uint8_t)p->nbits;
                p->rdst[p->nruns++] = (uint8_t)b;
            }
            p->run[p->nruns - 1] = (uint16_t)((p->run[p->nruns - 1] << 1) | 1);
            local[b] = p->nbits;
            p->bits[p->nbits++] = (uint8_t)b;
            continue;
        }
        local[b] = -1;
        if (p->nfields == 0 || ((w.mask >> (b - 1)) & 1ull)) {
            p->src[p->nfields] = (uint8_t)at;
            p->dst[p->nfields++] = (uint8_t)b;
        }
        p->field[p->nfields - 1] |= 1ull << b;
        ++at;
    }
    p->tile = std::max(p->nbits, A::R);
    p->ngroups = dim >> p->nbits;
    std::vector<WideRoundD> rounds;
    std::vector<WideStepD> steps;
    std::vector<u64> consts;
    // where the tile lies: slot vectors of its bits, of the outside bits that moves read, offset
    int col[MAX_WIDE_BITS + WIDE_RBITS_MAX], ocol[64] = {0}, c0 = 0;
    for (int b = 0; b < p->tile; ++b) col[b] = wide_slot<A>(1 << b);
    uint64_t seen = 0;
    auto note = [&](const WideMove& m) {
        if (!m.swap && m.b >= 0 && local[m.b] < 0) seen |= 1ull << m.b;
    };
    for (const WideRound& r : w.rounds)
        for (const WideMove& m : r.moves) note(m);
    for (const WideMove& m : w.moves) note(m);
    for (int b = 0; b < n; ++b)
        if ((seen >> b) & 1ull) p->obits[p->nout++] = (uint8_t)b;
    auto move = [&](const WideMove& m) {
        const int a = local[m.a];
        if (m.swap) std::swap(col[a], col[local[m.b]]);
        else if (m.b < 0) c0 ^= col[a];
        else if (local[m.b] < 0) ocol[m.b] ^= col[a];
        else col[local[m.b]] ^= col[a];
    };
    auto place = [&](const std::vector<int>& rbits, const std::vector<int>& tbits) {
        WideRoundD rd;
        std::memset(&rd, 0, sizeof(rd));
        for (size_t m = 0; m < rbits.size(); ++m) {
            rd.rc[m] = (uint16_t)col[rbits[m]];
            rd.rl[m] = (uint8_t)rbits[m];
        }
        for (size_t k = 0; k < tbits.size(); ++k) {
            rd.tc[k] = (uint16_t)col[tbits[k]];
            rd.tl[k] = (uint8_t)tbits[k];
        }
        rd.c0 = (uint16_t)c0;
        for (int e = 0; e < p->nout; ++e) rd.ov[e] = (uint16_t)ocol[p->obits[e]];
        return rd;
    };
    auto add = [&](const WideStep& ws) {
        const size_t at = consts.size();
        const std::vector<u64> c = wide_constants<A>(plan, ws, drift);
        consts.insert(consts.end(), c.begin(), c.end());
        return (uint16_t)at;
    };
    for (const WideRound& r : w.rounds) {
        for (const WideMove& m : r.moves) move(m);
        // the round's bits, filled up with the highest tile bits it leaves free
        std::vector<int> rbits, tbits;
        for (int m = 0; m < r.nbits; ++m) rbits.push_back(local[r.bits[m]]);
        for (int b = p->tile - 1; b >= 0 && (int)rbits.size() < A::R; --b)
            if (std::find(rbits.begin(), rbits.end(), b) == rbits.end()) rbits.push_back(b);
        // thread bits: first those whose slots differ in the lowest bits (the lanes of one
        // wavefront on distinct banks), then the rest
        const int lane = sizeof(typename A::V) == 16 ? 3 : 4;
        std::vector<int> rest;
        int basis[4] = {0, 0, 0, 0};
        for (int b = 0; b < p->tile; ++b) {
            if (std::find(rbits.begin(), rbits.end(), b) != rbits.end()) continue;
            int v = col[b] & ((1 << lane) - 1);
            for (int k = lane - 1; k >= 0; --k)
                if ((v >> k) & 1) {
                    if (!basis[k]) {
                        basis[k] = v;
                        break;
                    }
                    v ^= basis[k];
                }
            (v && (int)tbits.size() < lane ? tbits : rest).push_back(b);
        }
        tbits.insert(tbits.end(), rest.begin(), rest.end());
        WideRoundD rd = place(rbits, tbits);
        rd.first = (uint16_t)steps.size();
        for (int m = 0; m < r.nbits; ++m) {
            rd.rot_at[m] = (uint16_t)consts.size();
            if (r.has_pre[m]) {
                add(r.pre[m]);
                rd.rot[m] |= WIDE_PRE;
            }
            if (r.has_rot[m]) {
                add(r.rot[m]);
                rd.rot[m] |= r.rot[m].s.type == ST_REAL ? WIDE_REAL : WIDE_DENSE;
            }
            if (r.has_post[m]) {
                add(r.post[m]);
                rd.rot[m] |= WIDE_POST;
            }
        }
        for (int k = 0; k < 2; ++k)
            if (r.has_pair[k]) {
                rd.pair_at[k] = add(r.pairs[k]);
                rd.pairs |= (uint8_t)(1 << k);
            }
        auto reg = [&](int full_bit) {
            return (int)(std::find(rbits.begin(), rbits.end(), local[full_bit]) - rbits.begin());
        };
        for (const WideStep& ws : r.steps) {
            WideStepD s;
            std::memset(&s, 0, sizeof(s));
            s.type = ws.s.type;
            s.u0 = ws.s.u0;
            s.u1 = ws.s.u1;
            s.unit = ws.s.unit;
            if (ws.bit[0] >= 0) s.m = (uint8_t)reg(ws.bit[0]);
            if (s.type == ST_TABLE) s.m = ws.s.nfields;
            for (int b = 0; b < n; ++b) {
                if (!((ws.s.cm >> b) & 1ull)) continue;
                if (local[b] < 0) s.ocm |= 1ull << b;
                else if (reg(b) < A::R) s.rcm |= (uint8_t)(1 << reg(b));
                else s.xcm |= (uint16_t)(1 << local[b]);
            }
            s.at = add(ws);
            steps.push_back(s);
        }
        rd.count = (uint16_t)(steps.size() - rd.first);
        rounds.push_back(rd);
    }
    for (const WideMove& m : w.moves) move(m);
    std::vector<int> own_t, own_j;  // the store: thread bits, then register bits, in tile order
    for (int b = 0; b < p->nbits; ++b) (b < A::TBITS ? own_t : own_j).push_back(b);
    rounds.push_back(place(own_j, own_t));
    p->nrounds = (int)rounds.size() - 1;
    p->steps_at = (int)(rounds.size() * sizeof(WideRoundD));
    p->consts_at = p->steps_at + (int)(steps.size() * sizeof(WideStepD));
    p->prog_bytes = p->consts_at + (int)(consts.size() * sizeof(u64));
    const size_t at = prog->size();
    prog->resize(at + p->prog_bytes);
    std::memcpy(prog->data() + at, rounds.data(), rounds.size() * sizeof(WideRoundD));
    std::memcpy(prog->data() + at + p->steps_at, steps.data(), steps.size() * sizeof(WideStepD));
    std::memcpy(prog->data() + at + p->consts_at, consts.data(), consts.size() * sizeof(u64));
}

template <class A, class P>
static int launch_wide_pol(qgpu_handle* h, const WideParams& p) {
    const size_t smem = sizeof(typename A::V) * ((size_t)1 << (A::TBITS + A::RBITS)) + p.prog_bytes;
    QGPU_CUDA(smem_opt_in((const void*)k_wide<A, P>, smem));
    const uint64_t grid = std::max<uint64_t>(
        1, std::min<uint64_t>(p.ngroups, (uint64_t)h->sm_count * A::CTAS));
    k_wide<A, P><<<(unsigned)grid, 1 << A::TBITS, smem, h->stream>>>((typename P::S*)cur_state(h), p);
    QGPU_CHECK_LAUNCH("k_wide");
    h->launches++;
    h->h2d_bytes += sizeof(p);
    return QGPU_OK;
}

}  // namespace qgpu
