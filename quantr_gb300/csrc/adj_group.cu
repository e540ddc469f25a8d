// adj_group.cu — grouped passes of the adjoint sweep: the runs of single-wire gates of up to 11
// wires per pass over phi and lambda (no counterpart in quantr).
//
// A CTA stages a tile of both vectors in shared memory: the 2^K amplitudes that share every bit
// outside the pass's K tile bits (the wires' bits and the lowest other bits, so that runs of
// consecutive amplitudes load together). A wire's undo is exp(i a) D2 R D1 with D = diag(1, rho) and
// R real (pauli_frame, plan.cpp), the phase exp(i a) common to both vectors and left out. Per tile:
//   load   q = Im(conj(l) f) of every amplitude (the wires' Z sums and the -I sum are signed sums
//          of it: the sign of tile bits held in the thread index is applied once, at the end),
//          then D1 of all wires at once as one factor per amplitude;
//   rounds of P::R wires: their amplitudes in registers, per wire the Y sum (and X sum) over its
//          pairs, then R on both vectors;
//   store  D2 of all wires, where any is needed.
// Against a dense 2x2 and three Pauli sums per wire this takes 50 packed float-pair operations per
// amplitude and wire instead of 134 (complex128), and shared memory is crossed once per two
// (complex64: three) wires. Tiles of 2^10 amplitudes and CTAs of 128 threads (complex128): four CTAs
// per SM load, compute and store at different times, and a 20-qubit pass still fills the SMs
// evenly (256 threads and 2^11: 117 us against 58 us per pass). The per-CTA sums are taken a warp per
// row in triples of floats; in f64 they took up to 40 us per pass on the FP64 pipe.
// Bound (complex128, 23 qubits): the FMA pipe, 64 % busy. Measured, 4-layer ansatz, per pass of 8
// wires: 24 qubits 717 us (a pass per wire: 188 us each, and 980 us for a dense 2x2 with three
// sums); complex64 at 24 qubits 224 us (295 us before), where loads and index arithmetic bound it.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "adj_group.cuh"
#include "internal.cuh"

namespace qgpu {

constexpr int AG_BITS = ADJ_GROUP_TILE_BITS;  // widest tile
constexpr int AG_RBITS = 3;                   // tile bits in a thread's register index
constexpr int AG_PER = 1 << AG_RBITS;         // amplitudes per thread and vector

constexpr int AG_SLOTS = 12;                         // rounds x wires per round

struct AgWire {
    int lb;              // tile bit
    int row[3];          // partial rows of its X, Y, Z sums (-1: not needed)
    float4 rho1, rho2;   // (re_h, re_l, im_h, im_l) of its D1 and D2
    u64 c[16];           // R as Dot2 terms: out0 = c0 a + c1 b, out1 = c2 a + c3 b (hi, -third, -hi, -lo)
};
struct AgParams {
    uint64_t ngroups;
    int nbits;
    int bits[AG_BITS];   // ascending
    // the runs of index bits outside the tile: g's bits from `src` go to `dst` on
    int nfields;
    int src[AG_BITS + 1], dst[AG_BITS + 1];
    uint64_t field[AG_BITS + 1];  // the run's bits
    int tile;            // log2 of the shared tile: nbits, at least P::R (the rest stays zero)
    int nwires;
    int nrounds;
    int row_i;           // partial row of the sum of -Im(conj(l) f) (-1: not needed)
    int d1, d2, xsum, zsum;
    int nb;              // row length of partial (>= the grid)
    int ins[AG_SLOTS];   // per round, its bits in ascending order
    float4 dt1[256];     // D1's factor for the tile bits in the thread index
    AgWire w[AG_SLOTS];  // round r: wires r * R ..., filled up with other tile bits
};

// (h, l) += (bh, bl) in float-pair arithmetic (TwoSum of the heads, then the tails)
__device__ __forceinline__ void ag_acc(float2& a, float bh, float bl) {
    const float s = __fadd_rn(a.x, bh);
    const float bb = __fadd_rn(s, -a.x);
    float e = __fadd_rn(__fadd_rn(a.x, -__fadd_rn(s, -bb)), __fadd_rn(bh, -bb));
    e = __fadd_rn(e, __fadd_rn(a.y, bl));
    const float h = __fadd_rn(s, e);
    a.y = __fadd_rn(e, -__fadd_rn(h, -s));
    a.x = h;
}
// Sum of three floats (about 72 bits): the sums over threads, where large parts of either sign meet
// (in float pairs their rounding showed in gradients: 1e-14 of ||lambda||).
struct AgF3 {
    float a, b, c;
};
__device__ __forceinline__ float ag_two_sum(float& a, float x) {  // a += x, the rounding error
    const float s = __fadd_rn(a, x);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(x, bb));
    a = s;
    return e;
}
__device__ __forceinline__ void ag_acc3(AgF3& v, float h, float l) {
    const float e = ag_two_sum(v.a, h);
    const float e2 = ag_two_sum(v.b, l);
    const float e3 = ag_two_sum(v.b, e);
    v.c = __fadd_rn(v.c, __fadd_rn(e2, e3));
}
__device__ __forceinline__ u64 pneg(u64 a) { return a ^ 0x8000000080000000ull; }

// Product of complex constants in float pairs, (re_h, re_l, im_h, im_l).
__device__ __forceinline__ float4 ag_cmul(float4 a, float4 v) {
    const u64 c[8] = {p2(v.x, v.x), p2(v.y, v.y), p2(-v.x, -v.x), p2(-v.y, -v.y),
                      p2(-v.z, v.z), p2(-v.w, v.w), p2(v.z, -v.z), p2(v.w, -v.w)};
    const u64 h = p2(a.x, a.z), l = p2(a.y, a.w);
    PDot2 d;
    d.first(c, h, l);
    d.add(c + 4, pswap(h), pswap(l));
    u64 rh, rl;
    d.result(rh, rl);
    float4 r;
    up2(rh, r.x, r.z);
    up2(rl, r.y, r.w);
    return r;
}

struct AgFF {
    using S = double2;
    using V = ffp;
    using C = float4;  // complex constant (re_h, re_l, im_h, im_l)
    static __device__ __forceinline__ C combine(C a, C b) { return ag_cmul(a, b); }
    static constexpr int R = 2, TBITS = 7, CTAS = 4;  // TBITS: tile bits in the thread index
    static __device__ __forceinline__ V get(S a) { return ffr_load(a); }
    static __device__ __forceinline__ S put(const V& v) { return ffr_store(v); }
    static __device__ __forceinline__ V swap(const V& v) { return V{pswap(v.h), pswap(v.l)}; }
    static __device__ __forceinline__ V neg(const V& v) { return V{pneg(v.h), pneg(v.l)}; }
    static __device__ __forceinline__ void mul(V& a, C v) {
        const u64 c[8] = {p2(v.x, v.x), p2(v.y, v.y), p2(-v.x, -v.x), p2(-v.y, -v.y),
                          p2(-v.z, v.z), p2(-v.w, v.w), p2(v.z, -v.z), p2(v.w, -v.w)};
        PDot2 d;
        d.first(c, a.h, a.l);
        d.add(c + 4, pswap(a.h), pswap(a.l));
        d.result(a.h, a.l);
    }
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
    struct Sum {  // lane sums of products
        PDot2 d;
        __device__ __forceinline__ void clear() { d.s = d.en = 0; }
        // += a * b, na = -a
        __device__ __forceinline__ void add(const V& a, const V& na, const V& b) {
            const u64 c[4] = {a.h, a.l, na.h, na.l};
            d.add(c, b.h, b.l);
        }
        // lane 0 + sign * lane 1
        __device__ __forceinline__ float2 lanes(float sign) const {
            u64 h, l;
            d.result(h, l);
            float h0, h1, l0, l1;
            up2(h, h0, h1);
            up2(l, l0, l1);
            float2 r = make_float2(h0, l0);
            ag_acc(r, sign * h1, sign * l1);
            return r;
        }
        // v += lane 0 - lane 1, or minus that
        __device__ __forceinline__ void lanes3(AgF3& v, bool minus) const {
            u64 h, l;
            d.result(h, l);
            if (minus) {
                h = pneg(h);
                l = pneg(l);
            }
            float h0, h1, l0, l1;
            up2(h, h0, h1);
            up2(l, l0, l1);
            ag_acc3(v, h0, l0);
            ag_acc3(v, -h1, -l1);
        }
    };
};

// Z and -I sums of a thread's products, lane 0 - lane 1: one Dot2 per register index, folded every
// FLUSH tiles into sums of three floats. Kept over all tiles the Dot2's float error sum rounds more and
// more, and where amplitudes take few values alike in every thread (27 qubits: a gradient off by
// 4e-13 of sum|b|, now 3e-15). The 20-qubit gradient 3.25 -> 3.30 ms; three floats per product and register
// index instead 3.64 ms, for the registers.
struct AgZFF {
    static constexpr int FLUSH = 16;
    AgFF::Sum z[AG_PER];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < AG_PER; ++j) z[j].clear();
    }
    __device__ __forceinline__ void begin_tile() {}
    __device__ __forceinline__ void add(int j, const ffp& l, const ffp& f) {
        z[j].add(l, AgFF::neg(l), AgFF::swap(f));
    }
    __device__ __forceinline__ void end_tile() {}
    // v += the sum (m < 0), or the sum signed by bit m of the register index
    __device__ __forceinline__ void value(int m, AgF3& v) const {
#pragma unroll
        for (int j = 0; j < AG_PER; ++j) z[j].lanes3(v, m >= 0 && ((j >> m) & 1));
    }
};

struct AgF32 {
    using S = float2;
    using V = u64;
    using C = float4;
    static constexpr int R = 3, TBITS = 8, CTAS = 3;
    static __device__ __forceinline__ V get(S a) { return p2(a.x, a.y); }
    static __device__ __forceinline__ S put(V v) {
        S r;
        up2(v, r.x, r.y);
        return r;
    }
    static __device__ __forceinline__ V swap(V v) { return pswap(v); }
    static __device__ __forceinline__ V neg(V v) { return pneg(v); }
    // a b rounded to f32 (a factor per tile index: its rounding differs from one to the next)
    static __device__ __forceinline__ C combine(C a, C b) {
        const u64 bs = p2(-b.z, b.x), bl = p2(-b.w, b.y), bh = p2(b.x, b.z), bm = p2(b.y, b.w);
        u64 r = pmul(p2(a.y, a.y), bh);
        r = pfma(p2(a.w, a.w), bs, r);
        r = pfma(p2(a.x, a.x), bm, r);
        r = pfma(p2(a.z, a.z), bl, r);
        r = pfma(p2(a.x, a.x), bh, r);
        r = pfma(p2(a.z, a.z), bs, r);
        C c = make_float4(0.f, 0.f, 0.f, 0.f);
        up2(r, c.x, c.z);
        return c;
    }
    static __device__ __forceinline__ void mul(V& a, C c) {
        const u64 r = pmul(p2(c.x, c.x), a), i = pmul(p2(c.z, c.z), a);
        float rx, ry, ix, iy;
        up2(r, rx, ry);
        up2(i, ix, iy);
        a = p2(rx - iy, ry + ix);
    }
    static __device__ __forceinline__ void real(V& a, V& b, const u64* c) {
        // c + 3: minus the low parts, which keep all but the amplitudes from being rounded to f32
        const V o0 = pfma(c[0], a, pfma(c[4], b, pneg(pfma(c[3], a, pmul(c[7], b)))));
        const V o1 = pfma(c[8], a, pfma(c[12], b, pneg(pfma(c[11], a, pmul(c[15], b)))));
        a = o0;
        b = o1;
    }
    struct Sum {
        u64 s, en;
        __device__ __forceinline__ void clear() { s = en = 0; }
        // the few products of one tile: f32
        __device__ __forceinline__ void add(V a, V, V b) { s = pfma(a, b, s); }
        // sums over all tiles: the rounding error of every addition is kept
        __device__ __forceinline__ void add_tile(u64 p) {
            const u64 t = padd(s, p);
            const u64 bb = psub(t, s);
            const u64 q = padd(psub(s, psub(t, bb)), psub(p, bb));
            s = t;
            en = psub(en, q);
        }
        __device__ __forceinline__ float2 lanes(float sign) const {
            float h0, h1, l0, l1;
            up2(s, h0, h1);
            up2(pneg(en), l0, l1);
            float2 r = make_float2(h0, l0);
            ag_acc(r, sign * h1, sign * l1);
            return r;
        }
        __device__ __forceinline__ void lanes3(AgF3& v, bool) const {
            float h0, h1, l0, l1;
            up2(s, h0, h1);
            up2(pneg(en), l0, l1);
            ag_acc3(v, h0, l0);
            ag_acc3(v, -h1, -l1);
        }
    };
};

// The same with f32 sums of one tile's products, the sum and the three signed sums.
struct AgZF32 {
    static constexpr int FLUSH = 0;  // (never: the error sums' rounding lies far below the f32 products')
    AgF32::Sum z[4];
    u64 q[4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k].clear();
    }
    __device__ __forceinline__ void begin_tile() { q[0] = q[1] = q[2] = q[3] = 0; }
    __device__ __forceinline__ void add(int j, u64 l, u64 f) {
        const u64 p = pmul(l, pswap(f));
        q[3] = padd(q[3], p);
#pragma unroll
        for (int m = 0; m < 3; ++m) q[m] = (j >> m) & 1 ? psub(q[m], p) : padd(q[m], p);
    }
    __device__ __forceinline__ void end_tile() {
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k].add_tile(q[k]);
    }
    __device__ __forceinline__ void value(int m, AgF3& v) const { z[m < 0 ? 3 : m].lanes3(v, false); }
};
template <class P>
struct AgZ {
    using type = AgZFF;
};
template <>
struct AgZ<AgF32> {
    using type = AgZF32;
};

// Shared-memory slot of tile index l: the gathers of a round leave out up to three bits of l; bits
// 3..5 folded into the low three keep eight consecutive lanes of nearly every round on distinct
// 16-byte bank groups.
__device__ __forceinline__ int ag_slot(int l) {
    return l ^ ((l >> 3) & 1 ? 3 : 0) ^ ((l >> 4) & 1 ? 5 : 0) ^ ((l >> 5) & 1 ? 6 : 0);
}

template <class P>
constexpr size_t ag_smem(bool xsum) {
    return 2 * sizeof(typename P::V) * ((size_t)AG_PER << P::TBITS) +
           (size_t)(xsum ? 2 : 1) * (P::TBITS + AG_RBITS) * sizeof(float2) * ((size_t)1 << P::TBITS);
}

// First amplitude of tile g.
__device__ __forceinline__ uint64_t ag_base(const AgParams& p, uint64_t g) {
    uint64_t base = 0;
    for (int f = 0; f < p.nfields; ++f) base |= (g >> p.src[f]) << p.dst[f] & p.field[f];
    return base;
}

// XS: some wire needs its X sum (a rotation that D1 does not turn into Y and Z).
template <class P, bool XS>
__global__ void __launch_bounds__(1 << P::TBITS, P::CTAS)
k_adj_group(typename P::S* __restrict__ phi, typename P::S* __restrict__ lam,
            const __grid_constant__ AgParams p, double* __restrict__ partial) {
    using V = typename P::V;
    using C = typename P::C;
    constexpr int R = P::R, Q = 1 << R, AG_TBITS = P::TBITS, AG_THREADS = 1 << P::TBITS;
    constexpr int TILE = AG_PER << P::TBITS, WIRES = P::TBITS + AG_RBITS;
    extern __shared__ __align__(16) unsigned char smem[];
    V* sf = reinterpret_cast<V*>(smem);
    V* sl = sf + TILE;
    float2* red = reinterpret_cast<float2*>(sl + TILE);  // [Y, X][wire][thread]
    __shared__ C dj1[AG_PER], dj2[AG_PER];
    const int t = threadIdx.x;
    const int T = 1 << p.nbits;
    // offsets and diagonal factors of this thread's tile bits and of the register bits
    uint64_t off_t = 0;
    C dt1 = p.dt1[t];
    // (kept in registers: a constant indexed by the thread is read lane by lane)
    asm volatile("" : "+f"(dt1.x), "+f"(dt1.y), "+f"(dt1.z), "+f"(dt1.w));
    C dt2 = make_float4(1.f, 0.f, 0.f, 0.f);
    for (int m = 0; m < p.nbits && m < AG_TBITS; ++m)
        if ((t >> m) & 1) off_t |= 1ull << p.bits[m];
    uint64_t off_j[AG_RBITS] = {0, 0, 0};
#pragma unroll
    for (int m = 0; m < AG_RBITS; ++m)
        if (AG_TBITS + m < p.nbits) off_j[m] = 1ull << p.bits[AG_TBITS + m];
    for (int w = 0; w < p.nwires; ++w)
        if (p.w[w].lb < AG_TBITS && ((t >> p.w[w].lb) & 1)) {
            dt2 = ag_cmul(dt2, p.w[w].rho2);
        }
    if (t < AG_PER) {
        C a = make_float4(1.f, 0.f, 0.f, 0.f), b = a;
        for (int w = 0; w < p.nwires; ++w)
            if (p.w[w].lb >= AG_TBITS && ((t >> (p.w[w].lb - AG_TBITS)) & 1)) {
                a = ag_cmul(a, p.w[w].rho1);
                b = ag_cmul(b, p.w[w].rho2);
            }
        dj1[t] = a;
        dj2[t] = b;
    }
    for (int i = t; i < (XS ? 2 : 1) * WIRES * AG_THREADS; i += AG_THREADS)
        red[i] = make_float2(0.f, 0.f);
    typename AgZ<P>::type z;
    z.clear();
    // sums up to the last flush (all, register bits 0..2; indexed in a loop: they lie in local memory)
    constexpr int FLUSH = AgZ<P>::type::FLUSH;
    AgF3 ztot[AG_RBITS + 1];
    if constexpr (FLUSH > 0) {
#pragma unroll 1
        for (int k = 0; k <= AG_RBITS; ++k) ztot[k] = {0.f, 0.f, 0.f};
    }
    auto flush = [&]() {
#pragma unroll 1
        for (int k = 0; k <= AG_RBITS; ++k) {
            AgF3 v = ztot[k];
            z.value(k - 1, v);
            ztot[k] = v;
        }
        z.clear();
    };
    int tiles = 0;
    if (t >= T && t < (1 << p.tile)) sf[ag_slot(t)] = sl[ag_slot(t)] = V{};
    __syncthreads();
    for (uint64_t g = blockIdx.x; g < p.ngroups; g += gridDim.x) {
        const uint64_t base = ag_base(p, g) | off_t;
        if (t < T) {
            z.begin_tile();
#pragma unroll
            for (int j = 0; j < AG_PER; ++j) {
                if (t + j * AG_THREADS >= T) break;
                const uint64_t o = base | ((j & 1) ? off_j[0] : 0) | ((j & 2) ? off_j[1] : 0) |
                                   ((j & 4) ? off_j[2] : 0);
                V f = P::get(phi[o]), l = P::get(lam[o]);
                if (p.zsum) z.add(j, l, f);
                if (p.d1) {
                    const C dc = P::combine(dt1, dj1[j]);
                    P::mul(f, dc);
                    P::mul(l, dc);
                }
                sf[ag_slot(t + j * AG_THREADS)] = f;
                sl[ag_slot(t + j * AG_THREADS)] = l;
            }
            z.end_tile();
        }
        if constexpr (FLUSH > 0) {
            if (p.zsum && ++tiles == FLUSH) {
                flush();
                tiles = 0;
            }
        }
        __syncthreads();
        if (t < T && g + gridDim.x < p.ngroups) {  // the next tile heads for L2
            const uint64_t next = ag_base(p, g + gridDim.x) | off_t;
#pragma unroll
            for (int j = 0; j < AG_PER; ++j) {
                if (t + j * AG_THREADS >= T) break;
                const uint64_t o = next | ((j & 1) ? off_j[0] : 0) | ((j & 2) ? off_j[1] : 0) |
                                   ((j & 4) ? off_j[2] : 0);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(phi + o));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(lam + o));
            }
        }
        for (int r = 0; r < p.nrounds; ++r) {
            // the round's wires and, for a short last round, other bits of the tile
            int step[R], ins[R];
#pragma unroll
            for (int m = 0; m < R; ++m) {
                step[m] = ag_slot(1 << p.w[r * R + m].lb);
                ins[m] = p.ins[r * R + m];
            }
            typename P::Sum sy[R], sx[R];
#pragma unroll
            for (int m = 0; m < R; ++m) {
                sy[m].clear();
                if (XS) sx[m].clear();
            }
            for (int q = t; q < ((1 << p.tile) >> R); q += AG_THREADS) {
                int b = q;
#pragma unroll
                for (int m = 0; m < R; ++m) b = ((b >> ins[m]) << (ins[m] + 1)) | (b & ((1 << ins[m]) - 1));
                V f[Q], l[Q];
                int at[Q];
                at[0] = ag_slot(b);
#pragma unroll
                for (int i = 1; i < Q; ++i) {  // (ag_slot is linear in the index's bits)
                    const int m = i & 1 ? 0 : i & 2 ? 1 : 2;
                    at[i] = at[i & (i - 1)] ^ step[m];
                }
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    f[i] = sf[at[i]];
                    l[i] = sl[at[i]];
                }
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    if (r * R + m >= p.nwires) break;
                    const AgWire& w = p.w[r * R + m];
#pragma unroll
                    for (int i = 0; i < Q; ++i) {
                        if ((i >> m) & 1) continue;
                        const int k = i | (1 << m);
                        if (w.row[1] >= 0) {  // Y: -Re(l0* f1) + Re(l1* f0), both lanes added
                            sy[m].add(P::neg(l[i]), l[i], f[k]);
                            sy[m].add(l[k], P::neg(l[k]), f[i]);
                        }
                        if (XS && w.row[0] >= 0) {  // X: Im(l0* f1) + Im(l1* f0), lane 0 - lane 1
                            sx[m].add(l[i], P::neg(l[i]), P::swap(f[k]));
                            sx[m].add(l[k], P::neg(l[k]), P::swap(f[i]));
                        }
                        P::real(f[i], f[k], w.c);
                        P::real(l[i], l[k], w.c);
                    }
                }
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    sf[at[i]] = f[i];
                    sl[at[i]] = l[i];
                }
            }
#pragma unroll
            for (int m = 0; m < R; ++m) {
                const int w = r * R + m;
                if (w >= p.nwires) break;
                if (p.w[w].row[1] >= 0) {
                    const float2 v = sy[m].lanes(1.f);
                    ag_acc(red[w * AG_THREADS + t], v.x, v.y);
                }
                if (XS && p.w[w].row[0] >= 0) {
                    const float2 v = sx[m].lanes(-1.f);
                    ag_acc(red[(WIRES + w) * AG_THREADS + t], v.x, v.y);
                }
            }
            __syncthreads();
        }
        if (t < T) {
#pragma unroll
            for (int j = 0; j < AG_PER; ++j) {
                if (t + j * AG_THREADS >= T) break;
                const uint64_t o = base | ((j & 1) ? off_j[0] : 0) | ((j & 2) ? off_j[1] : 0) |
                                   ((j & 4) ? off_j[2] : 0);
                V f = sf[ag_slot(t + j * AG_THREADS)], l = sl[ag_slot(t + j * AG_THREADS)];
                if (p.d2) {
                    const C dc = P::combine(dt2, dj2[j]);
                    P::mul(f, dc);
                    P::mul(l, dc);
                }
                phi[o] = P::put(f);
                lam[o] = P::put(l);
            }
        }
        // (each thread refills exactly the slots it has just read)
    }
    // per-CTA sums, one warp per row, each a sum of three floats: the threads' Z and -I sums go
    // where the tile was
    __syncthreads();
    AgF3* zs = reinterpret_cast<AgF3*>(smem);  // [all, register bits 0..2][thread]
    if (p.zsum) {
        if constexpr (FLUSH > 0) {
            flush();
#pragma unroll 1
            for (int k = 0; k <= AG_RBITS; ++k) zs[k * AG_THREADS + t] = ztot[k];
        } else {
#pragma unroll
            for (int k = 0; k <= AG_RBITS; ++k) {
                AgF3 v = {0.f, 0.f, 0.f};
                z.value(k - 1, v);
                zs[k * AG_THREADS + t] = v;
            }
        }
    }
    __syncthreads();
    const int lane = t & 31;
    // rows: per wire X, Y, Z, then the -I sum
    for (int k = t >> 5; k < 3 * p.nwires + 1; k += AG_THREADS / 32) {
        const int w = k / 3, kind = k - 3 * w;
        const int row = w == p.nwires ? p.row_i : p.w[w].row[kind];
        if (row < 0) continue;
        AgF3 a = {0.f, 0.f, 0.f};
        if (w < p.nwires && kind < 2) {
            const float2* src = red + ((kind == 0 && XS ? WIRES : 0) + w) * AG_THREADS;
            for (int i = lane; i < AG_THREADS; i += 32) ag_acc3(a, src[i].x, src[i].y);
        } else {
            // Z of a thread bit: the bit gives the sign; of a register bit: summed with its sign
            const int lb = w < p.nwires ? p.w[w].lb : 0;
            const AgF3* src = zs + (lb < AG_TBITS ? 0 : lb - AG_TBITS + 1) * AG_THREADS;
            for (int i = lane; i < AG_THREADS; i += 32) {
                const bool n = w == p.nwires || (lb < AG_TBITS && ((i >> lb) & 1));
                const AgF3 v = src[i];
                ag_acc3(a, n ? -v.a : v.a, n ? -v.b : v.b);
                a.c += n ? -v.c : v.c;
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const float oa = __shfl_down_sync(0xffffffffu, a.a, d);
            const float ob = __shfl_down_sync(0xffffffffu, a.b, d);
            const float oc = __shfl_down_sync(0xffffffffu, a.c, d);
            ag_acc3(a, oa, ob);
            a.c += oc;
        }
        if (lane == 0) {  // column blockIdx.x; columns past the grid get 0
            double* dst = partial + (size_t)row * p.nb;
            dst[blockIdx.x] = (double)a.a + ((double)a.b + (double)a.c);
            for (int c = blockIdx.x + gridDim.x; c < p.nb; c += gridDim.x) dst[c] = 0.0;
        }
    }
}

static float4 ff_of(cd c) {
    float4 r;
    r.x = (float)c.real();
    r.y = (float)(c.real() - (double)r.x);
    r.z = (float)c.imag();
    r.w = (float)(c.imag() - (double)r.z);
    return r;
}
static void real_term(u64* c, double v) {
    const float h = (float)v, l = (float)(v - (double)h), third = (float)((v - (double)h) - (double)l);
    const float e[4] = {h, -third, -h, -l};
    for (int k = 0; k < 4; ++k) {
        uint32_t b;
        std::memcpy(&b, &e[k], 4);
        c[k] = (u64)b | ((u64)b << 32);
    }
}

// x^2 + y^2 - 1 for a value near 0, exact but for its own rounding
static double square_off(double x, double y) {
    const double p = x * x, q = y * y, t = p + q, b = t - p;
    const double e = (p - (t - b)) + (q - b);
    return (t - 1.0) + (e + (std::fma(x, x, -p) + std::fma(y, y, -q)));
}

template <class P, bool XS>
static int launch(qgpu_handle* h, void* phi, void* lam, const AgParams& p, double* partial,
                  uint64_t grid_cap) {
    const size_t smem = ag_smem<P>(XS);
    QGPU_CUDA(smem_opt_in((const void*)k_adj_group<P, XS>, smem));
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_adj_group<P, XS>, 1 << P::TBITS, smem) !=
            cudaSuccess || occ < 1)
        occ = 1;
    const uint64_t grid =
        std::max<uint64_t>(1, std::min<uint64_t>({p.ngroups, (uint64_t)h->sm_count * occ, grid_cap}));
    k_adj_group<P, XS><<<(unsigned)grid, 1 << P::TBITS, smem, h->stream>>>(
        (typename P::S*)phi, (typename P::S*)lam, p, partial);
    QGPU_CHECK_LAUNCH("k_adj_group");
    h->launches++;
    h->h2d_bytes += sizeof(p);
    return QGPU_OK;
}

int adj_group_tile_bits(int precision) {
    return (precision == QGPU_C64 ? AgF32::TBITS : AgFF::TBITS) + AG_RBITS;
}

int adj_group_pass(qgpu_handle* h, void* phi, void* lam, uint64_t mask,
                   const std::vector<AdjGroupWire>& wires, int row_i, double* partial, int nb,
                   double* drift) {
    AgParams p;
    std::memset(&p, 0, sizeof(p));
    for (int b = 0; b < 64; ++b)
        if ((mask >> b) & 1ull) p.bits[p.nbits++] = b;
    p.ngroups = h->dim >> p.nbits;
    for (int b = 0, at = 0; b < h->n_qubits; ++b) {
        if ((mask >> b) & 1ull) continue;
        if (p.nfields == 0 || b == 0 || ((mask >> (b - 1)) & 1ull)) {
            p.src[p.nfields] = at;
            p.dst[p.nfields++] = b;
        }
        p.field[p.nfields - 1] |= 1ull << b;
        ++at;
    }
    p.nb = nb;
    p.row_i = row_i;
    p.zsum = row_i >= 0;
    p.nwires = (int)wires.size();
    for (int c = 0; c < p.nwires; ++c) {
        const AdjGroupWire& s = wires[c];
        AgWire& w = p.w[c];
        w.lb = (int)(std::find(p.bits, p.bits + p.nbits, s.bit) - p.bits);
        for (int m = 0; m < 3; ++m) w.row[m] = s.row[m];
        w.rho1 = ff_of(s.frame.rho1);
        w.rho2 = ff_of(s.frame.rho2);
        p.d1 = p.d1 || s.frame.rho1 != cd(1.0, 0.0);
        p.d2 = p.d2 || s.frame.rho2 != cd(1.0, 0.0);
        p.xsum = p.xsum || s.row[0] >= 0;
        p.zsum = p.zsum || s.row[2] >= 0;
        // c^2 + s^2 and the moduli of rho differ from 1 by f64 rounding, with a bias that 200 rotations
        // turned into 1.5e-14 of both vectors' norms: the next rotation takes the drift out
        const double c0 = s.frame.c - s.frame.c * *drift, s0 = s.frame.s - s.frame.s * *drift;
        *drift += 0.5 * square_off(c0, s0) + 0.25 * square_off(s.frame.rho1.real(), s.frame.rho1.imag()) +
                  0.25 * square_off(s.frame.rho2.real(), s.frame.rho2.imag());
        real_term(w.c + 0, c0);
        real_term(w.c + 4, -s0);
        real_term(w.c + 8, s0);
        real_term(w.c + 12, c0);
    }
    const int tbits = h->precision == QGPU_C64 ? AgF32::TBITS : AgFF::TBITS;
    // D1's factors in f64: as products of float pairs on the device their rounding added up over
    // the layers of a circuit
    std::vector<cd> dt((size_t)1 << tbits, cd(1.0, 0.0));
    for (int c = 0; c < p.nwires && p.d1; ++c)
        if (p.w[c].lb < tbits)
            for (size_t t = 0; t < dt.size(); ++t)
                if ((t >> p.w[c].lb) & 1) dt[t] *= wires[c].frame.rho1;
    for (size_t t = 0; t < dt.size(); ++t) p.dt1[t] = ff_of(dt[t]);
    const int R = h->precision == QGPU_C64 ? AgF32::R : AgFF::R;
    p.tile = std::max(p.nbits, R);
    p.nrounds = (p.nwires + R - 1) / R;
    for (int r = 0; r < p.nrounds; ++r) {  // a short last round is filled up with other bits
        int* ins = p.ins + r * R;
        for (int m = 0; m < R; ++m) {
            const int c = r * R + m;
            for (int b = 0; c >= p.nwires && b < p.tile; ++b)
                if (std::find(ins, ins + m, b) == ins + m) {
                    p.w[c].lb = b;
                    break;
                }
            ins[m] = p.w[c].lb;
        }
        std::sort(ins, ins + R);
    }
    const uint64_t cap = (uint64_t)nb;
    if (h->precision == QGPU_C64)
        return p.xsum ? launch<AgF32, true>(h, phi, lam, p, partial, cap)
                      : launch<AgF32, false>(h, phi, lam, p, partial, cap);
    return p.xsum ? launch<AgFF, true>(h, phi, lam, p, partial, cap)
                  : launch<AgFF, false>(h, phi, lam, p, partial, cap);
}

}  // namespace qgpu
