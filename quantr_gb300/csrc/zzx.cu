// zzx.cu — tiled H psi and energy of the ZZ + X observable (no counterpart in quantr).
//
// (H psi)[x] = d(x) psi[x] + sum_b c_b psi[x ^ 2^b] needs the n neighbours of every amplitude. The
// plain kernel (k_apply_zzx, adjoint.cu) gathers them from global memory with f64 arithmetic:
// n reads through L2 and ~3n operations on the FP64 pipe (1/64 of the FP32 rate) per amplitude.
// Here a pass takes the neighbours along the bits of a tile of 2^11 amplitudes held in shared
// memory: the first pass along the 11 lowest bits (and the diagonal), each further pass along 8
// higher bits (tile: 3 low bits, so that 128-byte runs load together, and the 8 bits), so an n-qubit
// vector is read 1 + ceil((n - 11) / 8) times. complex128 runs in float pairs (packed Dot2), the
// energy sum included; complex64 in f32 with the energy as error-free transformed products.
// What bounds it: the float-pair multiply-adds (12 packed operations per amplitude and bit, ~2.1
// cycles per amplitude and SM in an 11-bit pass, against 0.7 cycles for its HBM read; the energy
// alone takes half of them, k_zzx_energy); complex64: the shared-memory reads (8 of 11 neighbours,
// 64 B per amplitude) and HBM.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include <math_constants.h>

#include "internal.cuh"
#include "zzx.cuh"

namespace qgpu {

constexpr int ZZX_THREADS = 256;
constexpr int ZZX_BITS = 11;    // tile bits: 8 in the thread index, 3 in a thread's registers
constexpr int ZZX_LOW = 3;      // low bits of the tiles of the later passes
constexpr int ZZX_REGS = 8;     // amplitudes per thread
constexpr int ZZX_FIELD = ZZX_BITS - ZZX_LOW;
constexpr u64 ZZX_SIGNS = 0x8000000080000000ull;  // both lanes negated

// Coefficients as the packed operands of a Dot2 term (hi, lo, -hi, -lo), both lanes alike.
struct ZzxCoef {
    u64 c[4];
};
struct ZzxParams {
    uint64_t ntiles;
    int shift;                  // first bit of the tile's high field (later passes)
    unsigned terms;             // tile bits whose X term this pass adds
    int n;
    ZzxCoef x[ZZX_BITS];        // X coefficient of tile bit m
    // the diagonal (first pass): ZZ coefficient of bits (q, q+1) and of the wrap (0, n-1)
    float2 zz[MAX_HAM_QUBITS];
    float2 wrap;
    u64 twice[ZZX_BITS][3];     // twice the X coefficient of tile bit m in three floats
};

struct ZvFF {
    using S = double2;
    using V = ffp;
    static __device__ __forceinline__ V split(S a) { return to_ffp(a); }
    // place of a tile index in shared memory: each arrangement of k_zzx_energy reads 8 different
    // 16-byte banks per phase
    static __device__ __forceinline__ unsigned place(unsigned x) { return x ^ ((x >> 3) & 7u); }
    // the split keeps neither magnitudes past the float range nor infinities and NaN
    static __device__ __forceinline__ bool too_large(S a) {
        constexpr int most = (1023 + 40) << 20;
        return (__double2hiint(a.x) & 0x7FFFFFFF) >= most || (__double2hiint(a.y) & 0x7FFFFFFF) >= most;
    }
    static __device__ __forceinline__ V get(const S* p) { return ffr_load(*p); }
    static __device__ __forceinline__ void put(S* p, const V& v) { *p = ffr_store(v); }
    struct Sum {  // sum of coefficient x amplitude
        PDot2 d;
        __device__ __forceinline__ void first(const u64* c, const V& v) { d.first(c, v.h, v.l); }
        __device__ __forceinline__ void add(const u64* c, const V& v) { d.add(c, v.h, v.l); }
        __device__ __forceinline__ V result() const {
            V r;
            d.result(r.h, r.l);
            return r;
        }
    };
    static __device__ __forceinline__ void term(PDot2& acc, const V& a, const V& b) {
        const u64 c[4] = {a.h, a.l, a.h ^ ZZX_SIGNS, a.l ^ ZZX_SIGNS};
        acc.add(c, b.h, b.l);
    }
    static __device__ __forceinline__ V plus(const V& a, const V& b) {
        const u64 t = padd(a.h, b.h);  // TwoSum of the heads, then the tails
        const u64 bb = psub(t, a.h);
        u64 e = padd(psub(a.h, psub(t, bb)), psub(b.h, bb));
        e = padd(e, padd(a.l, b.l));
        V r;
        r.h = padd(t, e);
        r.l = psub(e, psub(r.h, t));
        return r;
    }
};

struct ZvF32 {
    using S = float2;
    using V = u64;
    static __device__ __forceinline__ V split(S a) { return p2(a.x, a.y); }
    static __device__ __forceinline__ bool too_large(S) { return false; }  // the norm's sum shows it
    static __device__ __forceinline__ V get(const S* p) { return split(*p); }
    static __device__ __forceinline__ void put(S* p, V v) {
        float2 r;
        up2(v, r.x, r.y);
        *p = r;
    }
    struct Sum {
        V s;
        __device__ __forceinline__ void first(const u64* c, V v) { s = pmul(c[0], v); }
        __device__ __forceinline__ void add(const u64* c, V v) { s = pfma(c[0], v, s); }
        __device__ __forceinline__ V result() const { return s; }
    };
    // the product's rounding error and the sum's both go to the error sum, as in PDot2::add
    static __device__ __forceinline__ void term(PDot2& acc, V a, V b) {
        const u64 p = pmul(a, b);
        const u64 rn = pfma(a ^ ZZX_SIGNS, b, p);
        const u64 t = padd(acc.s, p);
        const u64 bb = psub(t, acc.s);
        const u64 q = padd(psub(acc.s, psub(t, bb)), psub(p, bb));
        acc.s = t;
        acc.en = padd(psub(acc.en, q), rn);
    }
    static __device__ __forceinline__ V plus(V a, V b) { return padd(a, b); }
};

// (h, l) + (b.x, b.y) as float pairs
__device__ __forceinline__ float2 ff_plus(float2 a, float2 b) {
    const float s = __fadd_rn(a.x, b.x);
    const float bb = __fsub_rn(s, a.x);
    float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb));
    e = __fadd_rn(e, __fadd_rn(a.y, b.y));
    const float h = __fadd_rn(s, e);
    return make_float2(h, __fsub_rn(e, __fsub_rn(h, s)));
}
__device__ __forceinline__ float2 ff_sign(float2 a, unsigned negative) {
    return negative & 1u ? make_float2(-a.x, -a.y) : a;
}

// A thread's sum over its tiles, in three floats per lane (about 72 bits). A PDot2 carries the few
// terms of one tile: its error sum is a float, and over equal terms its own rounding errors are equal
// too (kept over all tiles, a register whose amplitudes depend on two wires came out 2.4e-11 off at 27
// qubits of complex128 and 7.6e-11 of complex64; now 7e-15 and 4e-15, the f64 kernel 5e-15 and 1.7e-14).
// Energy calls: complex128 24 qubits 385 -> 444 us, 30 qubits 26.2 -> 30.9 ms; complex64 30 qubits 12.6 ->
// 13.1 ms.
struct ZzxTotal {
    u64 a, b, c;
    __device__ __forceinline__ void clear() { a = b = c = 0; }
    static __device__ __forceinline__ u64 two_sum(u64& s, u64 x) {  // s += x, the rounding error
        const u64 t = padd(s, x), bb = psub(t, s);
        const u64 e = padd(psub(s, psub(t, bb)), psub(x, bb));
        s = t;
        return e;
    }
    __device__ __forceinline__ void add(u64 h, u64 l) {
        const u64 e = two_sum(a, h), e2 = two_sum(b, l), e3 = two_sum(b, e);
        c = padd(c, padd(e2, e3));
    }
    __device__ __forceinline__ void add(const PDot2& d) { add(d.s, d.en ^ ZZX_SIGNS); }
    // += w * d
    __device__ __forceinline__ void add(const PDot2& d, const u64* w) {
        const u64 p = pmul(w[0], d.s);
        u64 r = pfma(w[0], d.s, p ^ ZZX_SIGNS);
        r = pfma(w[1], d.s, r);
        r = pfma(w[2], d.s, r);
        add(p, pfma(w[0] ^ ZZX_SIGNS, d.en, r));
    }
    __device__ __forceinline__ double value() const {
        float x[2], y[2], z[2];
        up2(a, x[0], x[1]);
        up2(b, y[0], y[1]);
        up2(c, z[0], z[1]);
        return ((double)x[0] + (double)x[1]) + (((double)y[0] + (double)y[1]) + ((double)z[0] + (double)z[1]));
    }
};

// Amplitude of tile index t + 256 j of tile g: base + j * step.
template <bool FIRST>
__device__ __forceinline__ void zzx_place(const ZzxParams& p, uint64_t g, unsigned t, uint64_t& base,
                                          uint64_t& step) {
    if (FIRST) {
        base = (g << ZZX_BITS) + t;
        step = ZZX_THREADS;
    } else {
        const uint64_t mid = g & ((1ull << (p.shift - ZZX_LOW)) - 1ull);
        const uint64_t top = g >> (p.shift - ZZX_LOW);
        base = (top << (p.shift + ZZX_FIELD)) | (mid << ZZX_LOW) | (t & ((1u << ZZX_LOW) - 1u)) |
               ((uint64_t)(t >> ZZX_LOW) << p.shift);
        step = 1ull << (p.shift + 8 - ZZX_LOW);
    }
}

// The diagonal in three parts: pairs of bits 0..5 and of bits 5..10 (tables by thread, once), and
// what lies above the tile g, one lane of a warp per pair of bits, with its four combinations with
// the pairs (10, 11) and (0, n-1) that reach into the tile.
struct ZzxDiag {
    float2 low[64], high[64], base[4];
    __device__ __forceinline__ void tables(const ZzxParams& p, unsigned t) {
        if (t < 128) {
            const unsigned x = t & 63u;
            const int q0 = t < 64 ? 0 : 5;
            float2 d = make_float2(0.f, 0.f);
            for (int q = 0; q < 5; ++q) d = ff_plus(d, ff_sign(p.zz[q0 + q], (x >> q) ^ (x >> (q + 1))));
            (t < 64 ? low : high)[x] = d;
        }
    }
    __device__ __forceinline__ void above(const ZzxParams& p, uint64_t g, unsigned t) {
        if (t >= 32) return;
        const int q = ZZX_BITS + (int)t;
        float2 d = make_float2(0.f, 0.f);
        if (q + 1 < p.n) d = ff_sign(p.zz[q], (unsigned)((g >> t) ^ (g >> (t + 1))));
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, d.x, w),
                                         __shfl_xor_sync(0xffffffffu, d.y, w));
            d = ff_plus(d, o);
        }
        if (t < 4) {
            d = ff_plus(d, ff_sign(p.zz[ZZX_BITS - 1], (t & 1u) ^ (unsigned)(g & 1ull)));
            d = ff_plus(d, ff_sign(p.wrap, (t >> 1) ^ (unsigned)(g >> (p.n - 1 - ZZX_BITS))));
            base[t] = d;
        }
    }
    // the diagonal entry of tile index t + 256 j as a Dot2 coefficient
    __device__ __forceinline__ ZzxCoef entry(unsigned t, int j) const {
        float2 d = ff_plus(low[t & 63u], high[((t >> 5) & 7u) | (j << 3)]);
        d = ff_plus(d, base[(j >> 2) | ((t & 1u) << 1)]);
        return {{p2(d.x, d.x), p2(d.y, d.y), p2(-d.x, -d.x), p2(-d.y, -d.y)}};
    }
};

// Per-CTA sums of a pass: warp shuffles, then one value per warp.
template <bool FIRST>
__device__ __forceinline__ void zzx_sums(double e, double q, double* __restrict__ partial) {
    const unsigned t = threadIdx.x;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        e += __shfl_down_sync(0xffffffffu, e, w);
        if (FIRST) q += __shfl_down_sync(0xffffffffu, q, w);
    }
    __shared__ double sums[2][ZZX_THREADS / 32];
    if ((t & 31u) == 0) {
        sums[0][t >> 5] = e;
        sums[1][t >> 5] = q;
    }
    __syncthreads();
    if (t < (FIRST ? 2u : 1u)) {
        double s = 0.0;
        for (int w = 0; w < ZZX_THREADS / 32; ++w) s += sums[t][w];
        partial[t * gridDim.x + blockIdx.x] = s;
    }
}

// H psi and the energy. FIRST: the diagonal and the 11 lowest bits; otherwise the bits of p.terms
// (above the 3 lowest). psi's copy goes to phi and H psi to lam, both in the sweep's layout
// (P::put); later passes read phi and add to lam. Without VEC only the energy is formed (complex64;
// the next tile's amplitudes are loaded while this one is worked on: 14.7 -> 12.6 ms at 30 qubits,
// with a pass that takes all its bits not testing each). partial[blockIdx] gets the
// pass's share of Re <psi|H psi>, and with FIRST partial[gridDim + blockIdx] that of <psi|psi>.
template <class P, bool FIRST, bool VEC>
__global__ void __launch_bounds__(ZZX_THREADS, sizeof(typename P::S) == 8 ? (VEC ? 4 : 2) : FIRST ? 2 : 3)
k_zzx(const typename P::S* __restrict__ psi, typename P::S* __restrict__ phi,
      typename P::S* __restrict__ lam, const __grid_constant__ ZzxParams p,
      double* __restrict__ partial) {
    using V = typename P::V;
    __shared__ __align__(16) V tile[1 << ZZX_BITS];
    __shared__ ZzxDiag diag;
    const unsigned t = threadIdx.x;
    if (FIRST) diag.tables(p, t);
    bool large = false;
    ZzxTotal energy, norm;
    energy.clear();
    norm.clear();
    typename P::S raw[ZZX_REGS];
    auto load = [&](uint64_t g) {
        uint64_t base, step;
        zzx_place<FIRST>(p, g, t, base, step);
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) raw[j] = psi[base + j * step];
    };
    if (!VEC && blockIdx.x < p.ntiles) load(blockIdx.x);
    for (uint64_t g = blockIdx.x; g < p.ntiles; g += gridDim.x) {
        uint64_t base, step;
        zzx_place<FIRST>(p, g, t, base, step);
        V v[ZZX_REGS];
        if constexpr (!FIRST && VEC) {
#pragma unroll
            for (int j = 0; j < ZZX_REGS; ++j) v[j] = P::get(phi + base + j * step);
        } else {
            if (VEC) load(g);
#pragma unroll
            for (int j = 0; j < ZZX_REGS; ++j) {
                v[j] = P::split(raw[j]);
                if constexpr (FIRST) large = large || P::too_large(raw[j]);
            }
        }
        __syncthreads();  // the previous tile's readers are done
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) tile[t + ZZX_THREADS * j] = v[j];
        if (!VEC && g + gridDim.x < p.ntiles) load(g + gridDim.x);
        if (FIRST) diag.above(p, g, t);
        __syncthreads();
        // (a pass that takes all bits of its tile, as all but the last do, tests none of them)
        auto work = [&](auto every) {
            PDot2 acc, nrm;
            acc.s = acc.en = nrm.s = nrm.en = 0;
#pragma unroll
            for (int j = 0; j < ZZX_REGS; ++j) {
                typename P::Sum s;
                if constexpr (FIRST) {
                    s.first(diag.entry(t, j).c, v[j]);
                } else {
                    const u64 zero[4] = {0, 0, 0, 0};
                    s.first(zero, v[j]);
                }
#pragma unroll
                for (int m = FIRST ? 0 : ZZX_LOW; m < 8; ++m)
                    if (decltype(every)::value || ((p.terms >> m) & 1u))
                        s.add(p.x[m].c, tile[(t ^ (1u << m)) + ZZX_THREADS * j]);
#pragma unroll
                for (int m = 8; m < ZZX_BITS; ++m)
                    if (decltype(every)::value || ((p.terms >> m) & 1u)) s.add(p.x[m].c, v[j ^ (1 << (m - 8))]);
                const V o = s.result();
                P::term(acc, v[j], o);
                if constexpr (FIRST) P::term(nrm, v[j], v[j]);
                if constexpr (VEC) {
                    if constexpr (FIRST) {
                        P::put(phi + base + j * step, v[j]);
                        P::put(lam + base + j * step, o);
                    } else {
                        P::put(lam + base + j * step, P::plus(P::get(lam + base + j * step), o));
                    }
                }
            }
            energy.add(acc);
            if constexpr (FIRST) norm.add(nrm);
        };
        if constexpr (FIRST) {
            work(std::true_type{});
        } else {
            if (p.terms == (1u << ZZX_BITS) - (1u << ZZX_LOW)) work(std::true_type{});
            else work(std::false_type{});
        }
    }
    zzx_sums<FIRST>(energy.value(), FIRST ? (large ? CUDART_INF : norm.value()) : 0.0, partial);
}

// The energy alone, complex128: the X term of bit m is 2 c_m sum Re conj(psi[x]) psi[x ^ 2^m] over the pairs,
// one product per pair where H psi takes two per amplitude (half the operations), summed per bit
// over the tile and then weighted. Three bits at a time lie in a thread's registers: the tile
// is written to shared memory once and read in three more arrangements (two in a later pass), 24
// reads of an amplitude per thread instead of one per bit. Energy call, k_zzx /
// k_zzx_energy: 17 qubits 38.5 / 36.0 us, 20 73 / 64, 24 564 / 444, 30 qubits 41.0 / 30.9 ms (8.9 of them the reads at HBM speed; L2
// prefetches of the next tile cost 4). Not for complex64, whose H psi takes one operation per
// amplitude and bit (30 qubits 18.1 against 12.6 ms before the sums in three floats).
template <bool FIRST>
__global__ void __launch_bounds__(ZZX_THREADS, 2)
k_zzx_energy(const double2* __restrict__ psi, const __grid_constant__ ZzxParams p,
             double* __restrict__ partial) {
    using P = ZvFF;
    using V = typename P::V;
    __shared__ __align__(16) V tile[1 << ZZX_BITS];
    __shared__ ZzxDiag diag;
    const unsigned t = threadIdx.x;
    if (FIRST) diag.tables(p, t);
    bool large = false;
    ZzxTotal energy, norm;
    energy.clear();
    norm.clear();
    const unsigned at0 = P::place(t), at1 = P::place((t & 31u) | ((t >> 5) << 8)),
                   at2 = P::place((t & 3u) | ((t >> 2) << 5)), at3 = P::place(t << 3);
    for (uint64_t g = blockIdx.x; g < p.ntiles; g += gridDim.x) {
        uint64_t base, step;
        zzx_place<FIRST>(p, g, t, base, step);
        V v[ZZX_REGS];
        typename P::S raw[ZZX_REGS];
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) raw[j] = psi[base + j * step];
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) {
            v[j] = P::split(raw[j]);
            if constexpr (FIRST) large = large || P::too_large(raw[j]);
        }
        __syncthreads();  // the previous tile's readers are done
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) tile[at0 ^ P::place(ZZX_THREADS * j)] = v[j];
        if (FIRST) diag.above(p, g, t);
        __syncthreads();
        if constexpr (FIRST) {
            PDot2 acc, nrm;
            acc.s = acc.en = nrm.s = nrm.en = 0;
#pragma unroll
            for (int j = 0; j < ZZX_REGS; ++j) {
                typename P::Sum s;
                s.first(diag.entry(t, j).c, v[j]);
                P::term(acc, v[j], s.result());
                P::term(nrm, v[j], v[j]);
            }
            energy.add(acc);
            norm.add(nrm);
        }
        // the pairs of tile bits m0 .. m0 + COUNT - 1, in register bits 0 ..
        auto pairs = [&](auto m0, auto count) {
#pragma unroll
            for (int k = 0; k < decltype(count)::value; ++k) {
                constexpr int M0 = decltype(m0)::value;
                if (!((p.terms >> (M0 + k)) & 1u)) continue;
                PDot2 bit;
                bit.s = bit.en = 0;
#pragma unroll
                for (int j = 0; j < ZZX_REGS; ++j)
                    if (!(j & (1 << k))) P::term(bit, v[j], v[j | (1 << k)]);
                energy.add(bit, p.twice[M0 + k]);
            }
        };
        constexpr std::integral_constant<int, 3> three{};
        pairs(std::integral_constant<int, 8>{}, three);
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) v[j] = tile[at1 ^ P::place(j << 5)];
        pairs(std::integral_constant<int, 5>{}, three);
#pragma unroll
        for (int j = 0; j < ZZX_REGS; ++j) v[j] = tile[at2 ^ P::place(j << 2)];
        pairs(std::integral_constant<int, 2>{}, three);
        if constexpr (FIRST) {
#pragma unroll
            for (int j = 0; j < ZZX_REGS; ++j) v[j] = tile[at3 ^ P::place(j)];
            pairs(std::integral_constant<int, 0>{}, std::integral_constant<int, 2>{});
        }
    }
    zzx_sums<FIRST>(energy.value(), FIRST ? (large ? CUDART_INF : norm.value()) : 0.0, partial);
}

// out[r] = sum of row r (nb values each): one warp per row, fixed order
__global__ void k_zzx_rows(const double* __restrict__ partial, int nb, double* __restrict__ out) {
    const int row = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
    for (int b = lane; b < nb; b += 32) s += partial[(size_t)row * nb + b];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
    if (lane == 0) out[row] = s;
}

static float2 coef_pair(double c) {
    const float h = (float)c;
    return make_float2(h, (float)(c - (double)h));
}
static u64 both(float f) {
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return (u64)b | ((u64)b << 32);
}

template <class P, bool VEC>
static int run_zzx(qgpu_handle* h, const typename P::S* psi, typename P::S* phi,
                   typename P::S* lam, const Ham& H, double* energy, bool* ok) {
    const int n = H.n;
    static_assert(1 + (MAX_HAM_QUBITS - ZZX_BITS + ZZX_FIELD - 1) / ZZX_FIELD + 1 <= 8, "row sums");
    const int npass = 1 + (n - ZZX_BITS + ZZX_FIELD - 1) / ZZX_FIELD;
    int occ = 0;
    constexpr bool pairs = !VEC && sizeof(typename P::S) == 16;  // k_zzx_energy
    cudaError_t e;
    if constexpr (pairs) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_zzx_energy<true>, ZZX_THREADS, 0);
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_zzx<P, true, VEC>, ZZX_THREADS, 0);
    if (e != cudaSuccess || occ < 1) occ = 1;
    const uint64_t ntiles = h->dim >> ZZX_BITS;
    const int nb = (int)std::min<uint64_t>(ntiles, (uint64_t)h->sm_count * occ);
    int st = h->work.ensure(((size_t)(npass + 1) * nb + npass + 1) * sizeof(double));
    if (st != QGPU_OK) return st;
    double* partial = (double*)h->work.ptr;
    double* sums = partial + (size_t)(npass + 1) * nb;
    ZzxParams p;
    std::memset(&p, 0, sizeof(p));
    p.ntiles = ntiles;
    p.n = n;
    for (int q = 0; q + 1 < n; ++q) p.zz[q] = coef_pair(H.a[n - 2 - q]);  // wires n-2-q, n-1-q
    p.wrap = coef_pair(H.a[n - 1]);
    int done = 0;  // bits whose X term has been added
    for (int pass = 0; pass < npass; ++pass) {
        int first = 0, low = 0;  // tile bit m >= low is index bit first + m - low
        if (pass > 0) {
            first = std::min(done, n - ZZX_FIELD);  // the last field may reach back over done bits
            low = ZZX_LOW;
            p.shift = first;
        }
        p.terms = 0;
        std::memset(p.twice, 0, sizeof(p.twice));
        for (int m = low; m < ZZX_BITS; ++m) {
            const int bit = first + m - low;
            if (bit < done || bit >= n) continue;
            p.terms |= 1u << m;
            const double w = 2.0 * H.b[n - 1 - bit];
            const float wh = (float)w, wl = (float)(w - (double)wh);
            p.twice[m][0] = both(wh);
            p.twice[m][1] = both(wl);
            p.twice[m][2] = both((float)((w - (double)wh) - (double)wl));
            const float2 c = coef_pair(H.b[n - 1 - bit]);
            p.x[m].c[0] = both(c.x);
            p.x[m].c[1] = both(c.y);
            p.x[m].c[2] = both(-c.x);
            p.x[m].c[3] = both(-c.y);
        }
        done = first + ZZX_BITS - low;
        double* row = partial + (pass == 0 ? 0 : (size_t)(pass + 1) * nb);
        if constexpr (pairs) {
            if (pass == 0) k_zzx_energy<true><<<nb, ZZX_THREADS, 0, h->stream>>>(psi, p, row);
            else k_zzx_energy<false><<<nb, ZZX_THREADS, 0, h->stream>>>(psi, p, row);
        } else {
            if (pass == 0) k_zzx<P, true, VEC><<<nb, ZZX_THREADS, 0, h->stream>>>(psi, phi, lam, p, row);
            else k_zzx<P, false, VEC><<<nb, ZZX_THREADS, 0, h->stream>>>(psi, phi, lam, p, row);
        }
        QGPU_CHECK_LAUNCH("k_zzx");
        h->launches++;
        h->h2d_bytes += sizeof(p);
    }
    k_zzx_rows<<<1, 32 * (npass + 1), 0, h->stream>>>(partial, nb, sums);
    QGPU_CHECK_LAUNCH("k_zzx_rows");
    h->launches++;
    double host[8];
    QGPU_CUDA(copy_async(h, host, sums, (npass + 1) * sizeof(double), cudaMemcpyDeviceToHost));
    QGPU_CUDA(cudaStreamSynchronize(h->stream));
    *energy = host[0];
    for (int r = 2; r <= npass; ++r) *energy += host[r];
    // amplitudes near one scale: their products keep their rounding errors in float range
    *ok = host[1] > 0x1p-40 && host[1] < 0x1p40;
    return QGPU_OK;
}

bool zzx_tiled_supported(const qgpu_handle* h, const Ham& H) {
    if (h->n_qubits < ZZX_MIN_QUBITS || (h->precision == QGPU_C128 && h->mode != QGPU_MODE_FAST))
        return false;
    double most = 0.0;
    for (int i = 0; i < H.n; ++i) {
        if (!std::isfinite(H.a[i]) || !std::isfinite(H.b[i])) return false;
        most = std::max(most, std::max(std::fabs(H.a[i]), std::fabs(H.b[i])));
    }
    return most > 0x1p-40 && most < 0x1p40;
}

int zzx_tiled(qgpu_handle* h, const void* psi, void* phi, void* lam, const Ham& H, double* energy,
              bool* ok) {
    if (h->precision == QGPU_C64)
        return lam ? run_zzx<ZvF32, true>(h, (const float2*)psi, (float2*)phi, (float2*)lam, H, energy, ok)
                   : run_zzx<ZvF32, false>(h, (const float2*)psi, nullptr, nullptr, H, energy, ok);
    return lam ? run_zzx<ZvFF, true>(h, (const double2*)psi, (double2*)phi, (double2*)lam, H, energy, ok)
               : run_zzx<ZvFF, false>(h, (const double2*)psi, nullptr, nullptr, H, energy, ok);
}

}  // namespace qgpu
