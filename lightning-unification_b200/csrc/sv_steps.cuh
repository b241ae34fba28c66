// sv_steps.cuh — gates applied in registers to shared-memory tiles of a state.
//
// Shared by the batched level engine (sv_batch_tiles.cuh) and the single-state fused engine
// (sv_fused.cu); the host side that plans segments and phases is sv_plan.hpp.  A segment is a run of
// steps whose bits fit one tile of 2^kt amplitudes; a phase is a set of its steps whose targets lie in
// the a register bits, the bits in which the A = 2^a amplitudes of a thread differ.
#pragma once

#include "sv_device.cuh"

namespace b200sv {
namespace steps {

// Step codes; + register bit, or + index of a register bit pair (pair_index).
enum TCode : uint16_t {
    T_DIAG_T = 0,    // diagonal table on thread bits: one factor for the thread
    T_PAR_T = 1,     // parity on thread bits
    T_DIAG = 2,      // diagonal table on any bits
    T_PAR = 3,       // parity on any bits
    T_SIGN_T = 4,    // -1 where every control bit (all thread bits) is set
    T_DIAG1 = 8,     // table whose lowest index bit is the register bit, the others thread bits
    T_SIGN1 = 12,    // -1: one register bit and thread bits
    T_DENSE = 16,    // 2x2 on the register bit
    T_DENSEC = 20,   // with controls
    T_CX_T = 24,     // swap along the register bit, controls all thread bits
    T_CX_G = 28,     // swap along the register bit, any controls
    T_SIGN2 = 32,    // -1: two register bits and thread bits
    T_SWAP = 40,     // exchange of a pair of register bits, any controls
    T_CX_R = 48,     // + target * 4 + control: swap along target, control one register bit (and thread bits)
    T_SPLIT = 64,    // real 2x2 on the register bit and a diagonal on it (complex128)
    T_DENSE2 = 72,   // dense matrix on a register pair, any controls (FP64 coefficients)
    T_DENSE3 = 80,   // dense matrix on three register bits (trip_mask), any controls (FP64 coefficients)
    T_PAIR2 = 88,    // 2x2 block on rows 01, 10 of a register pair, gamma on the others
    T_PAIR4 = 96,    // 2x2 block on registers 3 and 12, gamma on the others
};

struct alignas(16) TOp {
    uint16_t code, coef;   // coef: position in the segment's coefficients
    uint16_t creg;         // controls among the register bits
    uint16_t grad;         // 1 + gradient row of the segment, 0: not differentiated
    uint32_t cthr;         // controls among the thread bits (tile positions)
    uint32_t pm;           // parity: tile bits
    uint64_t pmg;          // parity: state bits outside the tile
    uint8_t p0, p1, p2;
    uint8_t pad;           // T_PAIR2, T_PAIR4: gamma is not 1; T_SPLIT: the diagonal comes first
    uint32_t dsign;        // T_DIAG with a gradient: generator entry of index i in bits 2i (1: +1, 2: -1)
};
// CNOT and SWAP steps move no data.  A segment keeps a GF(2)-linear map from the tile position of an
// amplitude to the place where it lies in shared memory; a CNOT between phases replaces the column of
// its control bit by (control column XOR target column), and the tile's store reads through the last
// map.  A phase loads and stores its amplitudes through its map: places, not positions, so no thread
// touches another's amplitudes and no extra barrier is needed.
struct TPhase {
    uint16_t op_begin, nops;
    uint8_t rt[4];     // tile position of register bit j
    uint16_t tval[8];  // tile bit of each thread index bit: the planner orders them so that the lanes
                       // of one shared-memory wavefront fall on different banks
    uint16_t tcol[8];  // its place (swizzled, bytes)
    uint16_t rcol[4];  // place of each register bit (swizzled, bytes)
    uint32_t signs;    // some step is a sign on thread bits (T_SIGN_T)
    uint32_t pad;
};
static_assert(sizeof(TPhase) == 56, "phases are staged in 8-byte words");
struct alignas(16) TSeg {
    uint32_t ph_begin, nph, op_begin, nops;
    uint32_t coef_begin, ncoef, ngrad;
    uint8_t lbits[16];
    uint8_t gbits[32];
    uint16_t fcol[12];  // places of the tile bits when the tile is stored (swizzled, bytes)
    uint8_t ng, kt, pad[2];
};
// tile buffers of a CTA: one per state, and a second one for complex64 forward (32 KiB tiles), which loads
// the next tile while the current one is worked on (200 gates on 27 qubits 25.7 -> 24.7 ms, 512 circuits of
// 8-12 qubits 138 -> 101 us; two buffers of the 64 KiB tiles would leave one CTA an SM)
template <typename R, bool REV> constexpr int tile_buffers() { return REV || sizeof(R) == 4 ? 2 : 1; }
template <typename R, bool REV> struct TGeo;
template <> struct TGeo<float, false> { static constexpr int kt = 12, a = 4, A = 16, reserve = 4, minb = 3; };
template <> struct TGeo<float, true> { static constexpr int kt = 12, a = 4, A = 16, reserve = 4, minb = 2; };
template <> struct TGeo<double, false> { static constexpr int kt = 12, a = 4, A = 16, reserve = 3, minb = 2; };
template <> struct TGeo<double, true> { static constexpr int kt = 11, a = 3, A = 8, reserve = 3, minb = 2; };
constexpr int kTThreads = 256;
constexpr int kTWarps = kTThreads / 32;
constexpr int kMaxTOps = 160, kMaxTCoefs = 640, kMaxTGrads = 64;
// Shared-memory position of tile amplitude l (linear over XOR): the lowest bits take the XOR of the
// next six, so lanes that differ in any five tile bits spread over the banks for nearly every choice
// of register bits.  complex64 keeps bit 0 in place: 16-byte pairs stay together.
template <typename R> __host__ __device__ __forceinline__ uint32_t tswz(uint32_t l) {
    if constexpr (sizeof(R) == 8) return l ^ ((l >> 3) & 7u) ^ ((l >> 6) & 7u);
    else return l ^ (((l >> 4) & 7u) << 1) ^ (((l >> 7) & 7u) << 1);
}

__host__ __device__ constexpr int pair_mask(int i) {
    return i == 0 ? 3 : i == 1 ? 5 : i == 2 ? 6 : i == 3 ? 9 : i == 4 ? 10 : 12;
}
__host__ __device__ constexpr int low_of(int m) { return m & -m; }

// single complex product m * v (FMA-formed components)
template <typename R> __device__ __forceinline__ C<R> cmul1(C<R> m, C<R> v) {
    return mk<R>(fma(m.x, v.x, -(m.y * v.y)), fma(m.x, v.y, m.y * v.x));
}

// ---- steps in registers ----------------------------------------------------------------------
template <typename R> __device__ __forceinline__ C<R> tprod(C<R> m, C<R> v) { return cmul1<R>(m, v); }
template <> __device__ __forceinline__ float2 tprod<float>(float2 m, float2 v) { return cmul2(m, v); }

template <typename R> __device__ __forceinline__ C<R> flip_sign(C<R> v, uint32_t neg) {  // neg: 0 or 1 << 31
    if constexpr (sizeof(R) == 4) {
        return make_float2(__uint_as_float(__float_as_uint(v.x) ^ neg), __uint_as_float(__float_as_uint(v.y) ^ neg));
    } else {
        const int h = (int)neg;
        return make_double2(__hiloint2double(__double2hiint(v.x) ^ h, __double2loint(v.x)),
                            __hiloint2double(__double2hiint(v.y) ^ h, __double2loint(v.y)));
    }
}

// Two FP32 values in one 64-bit register (the paired FP32 instructions' operand).  As float2 the halves
// are separate registers to the compiler, which then moved the whole state on every step (335 moves a
// step); a 64-bit value keeps its pair from step to step.
using pair2 = unsigned long long;
__device__ __forceinline__ pair2 pk(float x, float y) {
    pair2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpk(pair2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ pair2 mul2(pair2 a, pair2 b) {
    pair2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair2 fma2(pair2 a, pair2 b, pair2 c) {
    pair2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// A thread's amplitudes.  complex64 keeps real and imaginary parts apart and packs the two
// amplitudes that differ in register bit 0, so that the paired FP32 instructions work on two
// amplitude pairs at once without swapping or broadcasting any amplitude part; steps on register
// bit 0 itself use scalar FMAs (the planner gives that bit to the wire with the fewest steps).  Per
// differentiated 2x2 step on 16 + 16 amplitudes: 128 paired FMAs for both states and 60 for the four
// sums, against 128 + 64 register swaps and 112 scalar operations with (re, im) pairs; with CNOTs in the
// address map the 1024-circuit step went from 28.5 to 23.9 ms.
template <typename R, int A> struct Regs {
    C<R> v[A];
    __device__ __forceinline__ C<R> get(int g) const { return v[g]; }
    __device__ __forceinline__ void set(int g, C<R> x) { v[g] = x; }
};
template <int A> struct Regs<float, A> {
    pair2 re[A / 2], im[A / 2];
    __device__ __forceinline__ float2 get(int g) const {
        const float2 r = unpk(re[g >> 1]), i = unpk(im[g >> 1]);
        return (g & 1) ? make_float2(r.y, i.y) : make_float2(r.x, i.x);
    }
    __device__ __forceinline__ void set(int g, float2 x) {
        const float2 r = unpk(re[g >> 1]), i = unpk(im[g >> 1]);
        re[g >> 1] = (g & 1) ? pk(r.x, x.x) : pk(x.x, r.y);
        im[g >> 1] = (g & 1) ? pk(i.x, x.y) : pk(x.y, i.y);
    }
};

// ys = M (x, y) on every pair of the register bit; four roundings a component
template <typename R, int A, int BIT, bool CTL>
__device__ __forceinline__ void t_dense(Regs<R, A> &v, uint32_t creg, const C<R> (&m)[4]) {
    constexpr int B = 1 << BIT;
    if constexpr (sizeof(R) == 4 && BIT > 0 && !CTL) {
        pair2 mr[4], mi[4], mn[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            mr[i] = pk(m[i].x, m[i].x);
            mi[i] = pk(m[i].y, m[i].y);
            mn[i] = pk(-m[i].y, -m[i].y);
        }
#pragma unroll
        for (int h = 0; h < A / 2; ++h) {
            if (h & (B >> 1)) continue;
            const int k = h | (B >> 1);
            const pair2 xr = v.re[h], xi = v.im[h], yr = v.re[k], yi = v.im[k];
            v.re[h] = fma2(mn[1], yi, fma2(mr[1], yr, fma2(mn[0], xi, mul2(mr[0], xr))));
            v.im[h] = fma2(mi[1], yr, fma2(mr[1], yi, fma2(mi[0], xr, mul2(mr[0], xi))));
            v.re[k] = fma2(mn[3], yi, fma2(mr[3], yr, fma2(mn[2], xi, mul2(mr[2], xr))));
            v.im[k] = fma2(mi[3], yr, fma2(mr[3], yi, fma2(mi[2], xr, mul2(mr[2], xi))));
        }
    } else {
#pragma unroll
        for (int g = 0; g < A; ++g) {
            if (g & B) continue;
            if (CTL && ((uint32_t)g & creg) != creg) continue;
            const C<R> x = v.get(g), y = v.get(g | B);
            C<R> p, q;
            p.x = fma(-m[1].y, y.y, fma(m[1].x, y.x, fma(-m[0].y, x.y, m[0].x * x.x)));
            p.y = fma(m[1].y, y.x, fma(m[1].x, y.y, fma(m[0].y, x.x, m[0].x * x.y)));
            q.x = fma(-m[3].y, y.y, fma(m[3].x, y.x, fma(-m[2].y, x.y, m[2].x * x.x)));
            q.y = fma(m[3].y, y.x, fma(m[3].x, y.y, fma(m[2].y, x.x, m[2].x * x.y)));
            v.set(g, p);
            v.set(g | B, q);
        }
    }
}
// A real 2x2 r and a diagonal d on every pair of the register bit, one after the other: as many operations as
// their product takes, and the gates' own rounding on each amplitude, where the product's is the same on
// all of them.
template <int A, int BIT>
__device__ __forceinline__ void t_split(Regs<double, A> &v, const double2 (&r)[2], double2 d0, double2 d1, bool first) {
    constexpr int B = 1 << BIT;
#pragma unroll
    for (int g = 0; g < A; ++g) {
        if (g & B) continue;
        double2 x = v.get(g), y = v.get(g | B);
        if (first) {
            x = cmul1<double>(d0, x);
            y = cmul1<double>(d1, y);
        }
        double2 p = make_double2(fma(r[0].y, y.x, r[0].x * x.x), fma(r[0].y, y.y, r[0].x * x.y));
        double2 q = make_double2(fma(r[1].y, y.x, r[1].x * x.x), fma(r[1].y, y.y, r[1].x * x.y));
        if (!first) {
            p = cmul1<double>(d0, p);
            q = cmul1<double>(d1, q);
        }
        v.set(g, p);
        v.set(g | B, q);
    }
}
// The four sums of a differentiated step on register bit BIT, in FP64.  EXACT: so are the products, of
// widened amplitudes; otherwise complex64 forms each pair's value in FP32 first (runs of two and more gates
// in the batch engine, whose one-gate steps take the controlled form: with both forms behind T_DENSE the
// 1024-circuit step took 22.5 ms instead of 22.3).
template <typename R, int A, int BIT, bool CTL, bool EXACT>
__device__ __forceinline__ void t_cross(const Regs<R, A> &v, const Regs<R, A> &w, uint32_t creg, double (&s)[4]) {
    constexpr int B = 1 << BIT;
    if constexpr (sizeof(R) == 4 && BIT > 0 && !CTL && !EXACT) {
        const pair2 minus = pk(-1.0f, -1.0f);
#pragma unroll
        for (int h = 0; h < A / 2; ++h) {
            if (h & (B >> 1)) continue;
            const int k = h | (B >> 1);
            const pair2 a0r = v.re[h], a0i = v.im[h], a1r = v.re[k], a1i = v.im[k];
            const pair2 b0r = w.re[h], b0i = w.im[h], b1r = w.re[k], b1i = w.im[k];
            const pair2 n0i = mul2(b0i, minus), n1i = mul2(b1i, minus), n1r = mul2(b1r, minus);
            const float2 x1 = unpk(fma2(b0r, a0i, mul2(n0i, a0r)));
            const float2 x2 = unpk(fma2(b1r, a1i, mul2(n1i, a1r)));
            const float2 s1 = unpk(fma2(n1i, a0r, fma2(b1r, a0i, fma2(n0i, a1r, mul2(b0r, a1i)))));
            const float2 s2 = unpk(fma2(n1i, a0i, fma2(n1r, a0r, fma2(b0i, a1i, mul2(b0r, a1r)))));
            s[0] += (double)x1.x;
            s[1] += (double)x2.x;
            s[2] += (double)s1.x;
            s[3] += (double)s2.x;
            s[0] += (double)x1.y;
            s[1] += (double)x2.y;
            s[2] += (double)s1.y;
            s[3] += (double)s2.y;
        }
    } else {
#pragma unroll
        for (int g = 0; g < A; ++g) {
            if (g & B) continue;
            if (CTL && ((uint32_t)g & creg) != creg) continue;
            auto sums = [&](auto a0, auto a1, auto b0, auto b1) {
                s[0] += (double)fma(b0.x, a0.y, -(b0.y * a0.x));
                s[1] += (double)fma(b1.x, a1.y, -(b1.y * a1.x));
                s[2] += (double)fma(-b1.y, a0.x, fma(b1.x, a0.y, fma(-b0.y, a1.x, b0.x * a1.y)));
                s[3] += (double)fma(-b1.y, a0.y, fma(-b1.x, a0.x, fma(b0.y, a1.y, b0.x * a1.x)));
            };
            const C<R> a0 = v.get(g), a1 = v.get(g | B), b0 = w.get(g), b1 = w.get(g | B);
            if constexpr (EXACT) sums(widen<R>(a0), widen<R>(a1), widen<R>(b0), widen<R>(b1));
            else sums(a0, a1, b0, b1);
        }
    }
}
// Im(conj(b) a) in FP64
template <typename R> __device__ __forceinline__ double im_product(C<R> b, C<R> a) {
    const double2 p = widen<R>(b), q = widen<R>(a);
    return fma(p.x, q.y, -(p.y * q.x));
}
template <typename R, int A, int BIT>
__device__ __forceinline__ void t_diag1(Regs<R, A> &v, C<R> f0, C<R> f1) {
#pragma unroll
    for (int g = 0; g < A; ++g) v.set(g, tprod<R>((g >> BIT) & 1 ? f1 : f0, v.get(g)));
}
template <typename R, int A, int MASK> __device__ __forceinline__ void t_sign(Regs<R, A> &v, uint32_t neg) {
#pragma unroll
    for (int g = 0; g < A; ++g)
        if ((g & MASK) == MASK) v.set(g, flip_sign<R>(v.get(g), neg));
}
template <typename R, int A, int BIT, int CMASK> __device__ __forceinline__ void t_cx(Regs<R, A> &v, bool on) {
    constexpr int B = 1 << BIT;
#pragma unroll
    for (int g = 0; g < A; ++g) {
        if ((g & B) || (g & CMASK) != CMASK) continue;
        const C<R> x = v.get(g), y = v.get(g | B);
        v.set(g, on ? y : x);
        v.set(g | B, on ? x : y);
    }
}
template <typename R, int A, int BIT>
__device__ __forceinline__ void t_cxg(Regs<R, A> &v, uint32_t creg, bool on) {
    constexpr int B = 1 << BIT;
#pragma unroll
    for (int g = 0; g < A; ++g) {
        if (g & B) continue;
        const bool d = on && ((uint32_t)g & creg) == creg;
        const C<R> x = v.get(g), y = v.get(g | B);
        v.set(g, d ? y : x);
        v.set(g | B, d ? x : y);
    }
}
template <typename R, int A, int MASK>
__device__ __forceinline__ void t_swap(Regs<R, A> &v, uint32_t creg, bool on) {
    constexpr int LO = low_of(MASK), HI = MASK ^ LO;
#pragma unroll
    for (int g = 0; g < A; ++g) {
        if (g & MASK) continue;
        const bool d = on && ((uint32_t)g & creg) == creg;
        const C<R> x = v.get(g | LO), y = v.get(g | HI);
        v.set(g | LO, d ? y : x);
        v.set(g | HI, d ? x : y);
    }
}


// ---- wider steps (single-state engine) ---------------------------------------------------------
__host__ __device__ constexpr int trip_mask(int i) { return i == 0 ? 7 : i == 1 ? 11 : i == 2 ? 13 : 14; }
__host__ __device__ constexpr int bits_of(int m) { return m == 0 ? 0 : (m & 1) + bits_of(m >> 1); }
// c's bits deposited into the set bits of mask (ascending)
__host__ __device__ constexpr int spread_c(int mask, int c) {
    int r = 0, j = 0;
    for (int b = 0; b < 8; ++b)
        if ((mask >> b) & 1) {
            if ((c >> j) & 1) r |= 1 << b;
            ++j;
        }
    return r;
}
// Dense matrix on two or three register bits, summed in FP64 for both precisions (coefficients are
// doubles): complex64 rounds each output once, where sums of rounded products compensated in FP32
// pairs took three times the instructions and rounded every product.
template <typename R, int A, int MASK>
__device__ __forceinline__ void t_dense_wide(Regs<R, A> &v, uint32_t creg, const double2 *__restrict__ m) {
    constexpr int D = 1 << bits_of(MASK);
#pragma unroll
    for (int g = 0; g < A; ++g) {
        if (g & MASK) continue;
        if (((uint32_t)g & creg) != creg) continue;
        double2 x[D];
#pragma unroll
        for (int c = 0; c < D; ++c) x[c] = widen<R>(v.get(g | spread_c(MASK, c)));
#pragma unroll
        for (int r = 0; r < D; ++r) {
            double re = 0.0, im = 0.0;
#pragma unroll
            for (int c = 0; c < D; ++c) {
                const double2 k = m[r * D + c];
                re = fma(-k.y, x[c].y, fma(k.x, x[c].x, re));
                im = fma(k.y, x[c].x, fma(k.x, x[c].y, im));
            }
            v.set(g | spread_c(MASK, r), mk<R>((R)re, (R)im));
        }
    }
}
// 2x2 block on registers ia, ib
template <typename R, int A> __device__ __forceinline__ void t_block(Regs<R, A> &v, int ia, int ib, const C<R> (&m)[4]) {
    const C<R> x = v.get(ia), y = v.get(ib);
    C<R> p, q;
    p.x = fma(-m[1].y, y.y, fma(m[1].x, y.x, fma(-m[0].y, x.y, m[0].x * x.x)));
    p.y = fma(m[1].y, y.x, fma(m[1].x, y.y, fma(m[0].y, x.x, m[0].x * x.y)));
    q.x = fma(-m[3].y, y.y, fma(m[3].x, y.x, fma(-m[2].y, x.y, m[2].x * x.x)));
    q.y = fma(m[3].y, y.x, fma(m[3].x, y.y, fma(m[2].y, x.x, m[2].x * x.y)));
    v.set(ia, p);
    v.set(ib, q);
}
// excitations: the block on rows 01 and 10 of a register pair, gamma on the others
template <typename R, int A, int MASK>
__device__ __forceinline__ void t_pair2(Regs<R, A> &v, const C<R> *__restrict__ cf, bool rest) {
    constexpr int LO = low_of(MASK), HI = MASK ^ LO;
    const C<R> m[4] = {cf[0], cf[1], cf[2], cf[3]};
    const C<R> gm = cf[4];
#pragma unroll
    for (int g = 0; g < A; ++g) {
        if (g & MASK) continue;
        t_block<R, A>(v, g | LO, g | HI, m);
        if (rest) {
            v.set(g, tprod<R>(gm, v.get(g)));
            v.set(g | MASK, tprod<R>(gm, v.get(g | MASK)));
        }
    }
}
// double excitations: register index = row (the planner orders the registers so)
template <typename R, int A>
__device__ __forceinline__ void t_pair4(Regs<R, A> &v, const C<R> *__restrict__ cf, bool rest) {
    if constexpr (A >= 16) {
        const C<R> m[4] = {cf[0], cf[1], cf[2], cf[3]};
        const C<R> gm = cf[4];
        t_block<R, A>(v, 3, 12, m);
        if (rest) {
#pragma unroll
            for (int g = 0; g < 16; ++g)
                if (g != 3 && g != 12) v.set(g, tprod<R>(gm, v.get(g)));
        }
    }
}

// Sum of each of four values over the warp, with the exchange halving what each lane carries: lane
// 16 p + 8 q (+ 0..7) ends with the sum of value 2 p + q.  Fixed order.
__device__ __forceinline__ double reduce4(const double (&s)[4]) {
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16, hq = lane & 8;
    double k0 = hi ? s[2] : s[0], k1 = hi ? s[3] : s[1];
    k0 += __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[2], 16);
    k1 += __shfl_xor_sync(0xffffffffu, hi ? s[1] : s[3], 16);
    double r = hq ? k1 : k0;
    r += __shfl_xor_sync(0xffffffffu, hq ? k0 : k1, 8);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
    return r;
}
__device__ __forceinline__ void add_sums(double *sacc, uint32_t row, const double (&s)[4]) {
    const double r = reduce4(s);
    const int lane = threadIdx.x & 31;
    if ((lane & 7) == 0) sacc[(row * 4 + (lane >> 3)) * kTWarps + (threadIdx.x >> 5)] += r;
}

// The register bits b for which a step code exists in this geometry (a of the four).
#define TILE_EACH_BIT(X) X(0) X(1) X(2) X(3)
#define TILE_EACH_PAIR(X) X(0) X(1) X(2) X(3) X(4) X(5)

// One step on the thread's amplitudes of NS states.  WIDE: with the steps on two and more register
// bits that only the single-state engine has.
template <typename R, int A, int NS, bool WIDE>
__device__ __forceinline__ void t_step(Regs<R, A> &v, Regs<R, A> &w, const TOp &op, const C<R> *__restrict__ scf,
                                       double *sacc, uint32_t base, uint64_t tbase, const uint32_t (&rbit)[4], C<R> &tf,
                                       bool &has_tf, uint32_t &neg) {
    const C<R> *cf = scf + op.coef;
    const bool on = (base & op.cthr) == op.cthr;
    auto position = [&](int g) {  // tile position of register g
        uint32_t l = base;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((g >> j) & 1) l |= rbit[j];
        return l;
    };
    // the codes nearly every step has, ahead of the others: a two-level branch instead of a search
    // through the whole table
    if ((op.code & ~3) == T_DENSE) {
        const C<R> m[4] = {cf[0], cf[1], cf[2], cf[3]};
        const bool grad = NS == 2 && op.grad;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
#define TILE_DENSE(b)                                                                                          \
    if constexpr ((1 << b) < A) {                                                                              \
        if (grad) t_cross<R, A, b, false, WIDE>(v, w, 0, s);                                                   \
        t_dense<R, A, b, false>(v, 0, m);                                                                      \
        if (NS == 2) t_dense<R, A, b, false>(w, 0, m);                                                         \
    }
        if (op.code & 2) {
            if (op.code & 1) { TILE_DENSE(3) } else { TILE_DENSE(2) }
        } else {
            if (op.code & 1) { TILE_DENSE(1) } else { TILE_DENSE(0) }
        }
#undef TILE_DENSE
        if (grad) add_sums(sacc, op.grad - 1u, s);
        return;
    }
#define TILE_SPLIT(b)                                                                                          \
    if constexpr (sizeof(R) == 8 && (1 << b) < A) {                                                            \
        if (grad) t_cross<R, A, b, false, true>(v, w, 0, s);                                                   \
        t_split<A, b>(v, r, d0, d1, first);                                                                    \
        if (NS == 2) t_split<A, b>(w, r, d0, d1, first);                                                       \
    }
    // ahead of the others in the batch engine, whose ansatz layers are such runs; a single state's lists of
    // all kinds ran 0.7 % slower with this test before the table (26 qubits, 200 gates)
    if constexpr (sizeof(R) == 8 && !WIDE) {
        if ((op.code & ~3) == T_SPLIT) {
            const double2 r[2] = {cf[0], cf[1]}, d0 = cf[2], d1 = cf[3];
            const bool grad = NS == 2 && op.grad, first = op.pad != 0;
            double s[4] = {0.0, 0.0, 0.0, 0.0};
            if (op.code & 2) {
                if (op.code & 1) { TILE_SPLIT(3) } else { TILE_SPLIT(2) }
            } else {
                if (op.code & 1) { TILE_SPLIT(1) } else { TILE_SPLIT(0) }
            }
            if (grad) add_sums(sacc, op.grad - 1u, s);
            return;
        }
    }
    switch (op.code) {
    case T_DIAG_T: {
        const uint32_t idx = (((base >> op.p0) & 1u) << 2) | (((base >> op.p1) & 1u) << 1) | ((base >> op.p2) & 1u);
        tf = has_tf ? tprod<R>(cf[idx], tf) : cf[idx];
        has_tf = true;
        break;
    }
    case T_PAR_T: {
        const int par = (__popcll(tbase & op.pmg) + __popc(base & op.pm)) & 1;
        tf = has_tf ? tprod<R>(cf[par], tf) : cf[par];
        has_tf = true;
        break;
    }
    case T_SIGN_T: neg ^= on ? 0x80000000u : 0u; break;
    case T_DIAG: {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        const bool grad = NS == 2 && op.grad;
#pragma unroll
        for (int g = 0; g < A; ++g) {
            const uint32_t x = position(g);
            const uint32_t idx = (((x >> op.p0) & 1u) << 2) | (((x >> op.p1) & 1u) << 1) | ((x >> op.p2) & 1u);
            if (grad) {
                const uint32_t d = (op.dsign >> (2 * idx)) & 3u;
                const double im = im_product<R>(w.get(g), v.get(g));
                s[0] += d == 1u ? im : d == 2u ? -im : 0.0;
            }
            const C<R> f = cf[idx];
            v.set(g, tprod<R>(f, v.get(g)));
            if (NS == 2) w.set(g, tprod<R>(f, w.get(g)));
        }
        if (grad) add_sums(sacc, op.grad - 1u, s);
        break;
    }
    case T_PAR: {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        const bool grad = NS == 2 && op.grad;
        const int tp = __popcll(tbase & op.pmg) & 1;
        const C<R> f0 = cf[0], f1 = cf[1];
#pragma unroll
        for (int g = 0; g < A; ++g) {
            const bool odd = ((__popc(position(g) & op.pm) + tp) & 1) != 0;
            if (grad) {
                const double im = im_product<R>(w.get(g), v.get(g));
                s[0] += odd ? -im : im;
            }
            const C<R> f = odd ? f1 : f0;
            v.set(g, tprod<R>(f, v.get(g)));
            if (NS == 2) w.set(g, tprod<R>(f, w.get(g)));
        }
        if (grad) add_sums(sacc, op.grad - 1u, s);
        break;
    }
#define TILE_BIT_CASES(b)                                                                                      \
    case T_SPLIT + b:                                                                                          \
        if constexpr (sizeof(R) == 8 && WIDE) {                                                                \
            const double2 r[2] = {cf[0], cf[1]}, d0 = cf[2], d1 = cf[3];                                       \
            const bool grad = NS == 2 && op.grad, first = op.pad != 0;                                         \
            double s[4] = {0.0, 0.0, 0.0, 0.0};                                                                \
            TILE_SPLIT(b)                                                                                      \
            if (grad) add_sums(sacc, op.grad - 1u, s);                                                         \
        }                                                                                                      \
        break;                                                                                                 \
    case T_DIAG1 + b:                                                                                          \
        if constexpr ((1 << b) < A) {                                                                          \
            const uint32_t i = ((((base >> op.p0) & 1u) << 1) | ((base >> op.p1) & 1u)) * 2u;                  \
            const C<R> f0 = cf[i], f1 = cf[i + 1];                                                             \
            t_diag1<R, A, b>(v, f0, f1);                                                                       \
            if (NS == 2) t_diag1<R, A, b>(w, f0, f1);                                                          \
        }                                                                                                      \
        break;                                                                                                 \
    case T_SIGN1 + b:                                                                                          \
        if constexpr ((1 << b) < A) {                                                                          \
            const uint32_t sg = on ? 0x80000000u : 0u;                                                         \
            t_sign<R, A, 1 << b>(v, sg);                                                                       \
            if (NS == 2) t_sign<R, A, 1 << b>(w, sg);                                                          \
        }                                                                                                      \
        break;                                                                                                 \
    case T_DENSEC + b:                                                                                         \
        if constexpr ((1 << b) < A) {                                                                          \
            const C<R> m[4] = {cf[0], cf[1], cf[2], cf[3]};                                                    \
            if (NS == 2 && op.grad) {                                                                          \
                double s[4] = {0.0, 0.0, 0.0, 0.0};                                                            \
                if (on) t_cross<R, A, b, true, true>(v, w, op.creg, s);                                        \
                add_sums(sacc, op.grad - 1u, s);                                                               \
            }                                                                                                  \
            if (on) {                                                                                          \
                t_dense<R, A, b, true>(v, op.creg, m);                                                         \
                if (NS == 2) t_dense<R, A, b, true>(w, op.creg, m);                                            \
            }                                                                                                  \
        }                                                                                                      \
        break;                                                                                                 \
    case T_CX_T + b:                                                                                           \
        if constexpr ((1 << b) < A) {                                                                          \
            t_cx<R, A, b, 0>(v, on);                                                                           \
            if (NS == 2) t_cx<R, A, b, 0>(w, on);                                                              \
        }                                                                                                      \
        break;                                                                                                 \
    case T_CX_G + b:                                                                                           \
        if constexpr ((1 << b) < A) {                                                                          \
            t_cxg<R, A, b>(v, op.creg, on);                                                                    \
            if (NS == 2) t_cxg<R, A, b>(w, op.creg, on);                                                       \
        }                                                                                                      \
        break;
        TILE_EACH_BIT(TILE_BIT_CASES)
#undef TILE_BIT_CASES
#undef TILE_SPLIT
#define TILE_PAIR_CASES(i)                                                                                     \
    case T_SIGN2 + i:                                                                                          \
        if constexpr (pair_mask(i) < A) {                                                                      \
            const uint32_t sg = on ? 0x80000000u : 0u;                                                         \
            t_sign<R, A, pair_mask(i)>(v, sg);                                                                 \
            if (NS == 2) t_sign<R, A, pair_mask(i)>(w, sg);                                                    \
        }                                                                                                      \
        break;                                                                                                 \
    case T_SWAP + i:                                                                                           \
        if constexpr (pair_mask(i) < A) {                                                                      \
            t_swap<R, A, pair_mask(i)>(v, op.creg, on);                                                        \
            if (NS == 2) t_swap<R, A, pair_mask(i)>(w, op.creg, on);                                           \
        }                                                                                                      \
        break;
        TILE_EACH_PAIR(TILE_PAIR_CASES)
#undef TILE_PAIR_CASES
#define TILE_CX_CASE(t, c)                                                                                     \
    case T_CX_R + t * 4 + c:                                                                                   \
        if constexpr (t != c && (1 << t) < A && (1 << c) < A) {                                                \
            t_cx<R, A, t, 1 << c>(v, on);                                                                      \
            if (NS == 2) t_cx<R, A, t, 1 << c>(w, on);                                                         \
        }                                                                                                      \
        break;
#define TILE_CX_CASES(t) TILE_CX_CASE(t, 0) TILE_CX_CASE(t, 1) TILE_CX_CASE(t, 2) TILE_CX_CASE(t, 3)
        TILE_EACH_BIT(TILE_CX_CASES)
#undef TILE_CX_CASES
#undef TILE_CX_CASE
    default:
        if constexpr (WIDE) {
            const double2 *cd = reinterpret_cast<const double2 *>(cf);
            switch (op.code) {
#define TILE_DENSE2(i)                                                                                         \
            case T_DENSE2 + i:                                                                                 \
                if constexpr (pair_mask(i) < A) {                                                              \
                    if (on) {                                                                                  \
                        t_dense_wide<R, A, pair_mask(i)>(v, op.creg, cd);                                      \
                        if (NS == 2) t_dense_wide<R, A, pair_mask(i)>(w, op.creg, cd);                         \
                    }                                                                                          \
                }                                                                                              \
                break;                                                                                         \
            case T_PAIR2 + i:                                                                                  \
                if constexpr (pair_mask(i) < A) {                                                              \
                    t_pair2<R, A, pair_mask(i)>(v, cf, op.pad != 0);                                           \
                    if (NS == 2) t_pair2<R, A, pair_mask(i)>(w, cf, op.pad != 0);                              \
                }                                                                                              \
                break;
                TILE_EACH_PAIR(TILE_DENSE2)
#undef TILE_DENSE2
#define TILE_DENSE3(i)                                                                                         \
            case T_DENSE3 + i:                                                                                 \
                if constexpr (trip_mask(i) < A) {                                                              \
                    if (on) {                                                                                  \
                        t_dense_wide<R, A, trip_mask(i)>(v, op.creg, cd);                                      \
                        if (NS == 2) t_dense_wide<R, A, trip_mask(i)>(w, op.creg, cd);                         \
                    }                                                                                          \
                }                                                                                              \
                break;
                TILE_EACH_BIT(TILE_DENSE3)
#undef TILE_DENSE3
            case T_PAIR4:
                t_pair4<R, A>(v, cf, op.pad != 0);
                if (NS == 2) t_pair4<R, A>(w, cf, op.pad != 0);
                break;
            default: break;
            }
        }
        break;
    }
}

__device__ __forceinline__ uint64_t spread(uint64_t x, const uint8_t *pos, int nbits) {
    uint64_t r = 0;
    for (int i = 0; i < nbits; ++i) r |= ((x >> i) & 1u) << pos[i];
    return r;
}
template <typename T> __device__ __forceinline__ void copy_words(T *dst, const T *src, uint32_t n) {
    static_assert(sizeof(T) % 8 == 0, "records are whole 8-byte words");
    const uint2 *s = reinterpret_cast<const uint2 *>(src);
    uint2 *d = reinterpret_cast<uint2 *>(dst);
    for (uint32_t i = threadIdx.x; i < n * (uint32_t)(sizeof(T) / 8); i += blockDim.x) d[i] = s[i];
}


// The segment's phases on tiles t0, t0 + stride, ... below t1.  Forward: one state (a_in read, a_out
// written); REV: lambda, and the bra in place.  fresh: the state is |0..0> and is not read; store:
// the tiles are written (lambda only where a_out is given).  The two or three CTAs an SM holds overlap
// one another's tile moves and barriers.
template <typename R, bool REV, bool WIDE>
__device__ __forceinline__ void run_tiles(const TSeg &sg, C<R> *sl, C<R> *sb, const TOp *sop, const C<R> *scf,
                                          const TPhase *sph, double *sacc, uint64_t t0, uint64_t t1, uint64_t stride,
                                          bool fresh, bool store, const C<R> *a_in, C<R> *a_out, C<R> *b,
                                          uint64_t namp) {
    using G = TGeo<R, REV>;
    constexpr int A = G::A, NS = REV ? 2 : 1;
    constexpr int V = 16 / (int)sizeof(C<R>);
    constexpr int PER = A / V;
    // 16-byte chunk j of a thread: chunk threadIdx.x + j * blockDim.x of the tile.  Everything that
    // depends on j alone comes from one 16-byte broadcast, everything that depends on the thread alone
    // is formed once, and the tile's base is one bit per lane, so a chunk's move takes about six
    // instructions besides the access (27 before: a quarter of a light segment's instructions).
    constexpr int LV = V == 2 ? 1 : 0;
    struct alignas(16) Chunk {
        uint64_t off;     // bytes in the state
        uint32_t sw, f;   // bytes in the tile: when loaded, and where the last map puts it
    };
    __shared__ Chunk s_ch[PER];
    const uint32_t NT = blockDim.x, lane = threadIdx.x & 31;
    const int lt = 31 - __clz((int)NT);
    const bool padded = namp < (uint64_t(1) << sg.kt);
    if (threadIdx.x < PER) {
        const uint32_t l = threadIdx.x * NT * V;
        Chunk c;
        c.off = spread(l, sg.lbits, sg.kt) * sizeof(C<R>);
        c.sw = tswz<R>(l) * (uint32_t)sizeof(C<R>);
        c.f = 0;
        for (int i = 0; (1 << i) < PER; ++i)
            if ((threadIdx.x >> i) & 1) c.f ^= sg.fcol[LV + lt + i];
        s_ch[threadIdx.x] = c;
    }
    const uint64_t lo = spread((uint64_t)threadIdx.x * V, sg.lbits, sg.kt);
    const uint32_t sw0 = tswz<R>(threadIdx.x * V) * (uint32_t)sizeof(C<R>);
    uint32_t f0 = 0;
    for (int i = 0; i < lt; ++i) f0 ^= (threadIdx.x >> i) & 1u ? sg.fcol[LV + i] : 0u;
    const uint32_t gpos = (int)lane < (int)sg.ng ? sg.gbits[lane] : 0u;
    char *const cb = reinterpret_cast<char *>(sb);
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    constexpr bool AHEAD = !REV && tile_buffers<R, REV>() == 2;
    auto base_of = [&](uint64_t t) {
        const uint64_t mine = (int)lane < (int)sg.ng ? ((t >> lane) & 1u) << gpos : 0u;
        return (uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)mine) |
               (uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(mine >> 32)) << 32;
    };
    uint32_t cur = 0;
    if (AHEAD && !fresh && !padded && t0 < t1) {
        const char *src = reinterpret_cast<const char *>(a_in + (base_of(t0) | lo));
#pragma unroll
        for (int j = 0; j < PER; ++j) cp_async16(reinterpret_cast<char *>(sl) + (sw0 ^ s_ch[j].sw), src + s_ch[j].off);
        cp_async_commit();
    }
    for (uint64_t t = t0; t < t1; t += stride) {
        char *const cl = reinterpret_cast<char *>(sl) + (AHEAD ? cur * NT * A * (uint32_t)sizeof(C<R>) : 0u);
        const uint64_t tbase = base_of(t);
        const uint64_t start = tbase | lo;
        // beyond the state in a tile padded to a warp's share
        auto outside = [&](const Chunk &c) { return padded && start + c.off / sizeof(C<R>) >= namp; };
        if (fresh && t != 0) {  // |0..0> has no amplitude here, and a segment keeps zeros
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const Chunk c = s_ch[j];
                if (!outside(c)) *reinterpret_cast<float4 *>(reinterpret_cast<char *>(a_out + start) + c.off) = z4;
            }
            continue;
        }
        if (AHEAD && !fresh && !padded) {
            const uint64_t tn = t + stride;
            if (tn < t1) {
                const char *src = reinterpret_cast<const char *>(a_in + (base_of(tn) | lo));
                char *const dst = reinterpret_cast<char *>(sl) + (cur ^ 1u) * NT * A * (uint32_t)sizeof(C<R>);
#pragma unroll
                for (int j = 0; j < PER; ++j) cp_async16(dst + (sw0 ^ s_ch[j].sw), src + s_ch[j].off);
            }
            cp_async_commit();
            cp_async_wait1();
        } else {
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const Chunk c = s_ch[j];
                const uint32_t at = sw0 ^ c.sw;
                if (!fresh && !outside(c)) {
                    cp_async16(cl + at, reinterpret_cast<const char *>(a_in + start) + c.off);
                    if (REV) cp_async16(cb + at, reinterpret_cast<const char *>(b + start) + c.off);
                } else {
                    *reinterpret_cast<float4 *>(cl + at) = z4;
                    if (REV) *reinterpret_cast<float4 *>(cb + at) = z4;
                }
            }
            cp_async_commit();
            cp_async_wait0();
        }
        if (fresh && threadIdx.x == 0) *reinterpret_cast<C<R> *>(cl) = mk<R>(1, 0);  // thread 0 zeroed position 0 itself
        __syncthreads();
        for (uint32_t p = 0; p < sg.nph; ++p) {
            const TPhase ph = sph[p];
            uint32_t base = 0, sbase = 0, rbit[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < G::a; ++j) rbit[j] = 1u << ph.rt[j];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool one = (threadIdx.x >> j) & 1u;
                base |= one ? ph.tval[j] : 0u;
                sbase ^= one ? ph.tcol[j] : 0u;
            }
            auto at = [&](int g) {
                uint32_t x = sbase;
#pragma unroll
                for (int j = 0; j < G::a; ++j)
                    if ((g >> j) & 1) x ^= ph.rcol[j];
                return x;
            };
            auto amp = [](char *t, uint32_t x) -> C<R> & { return *reinterpret_cast<C<R> *>(t + x); };
            Regs<R, A> v, w;
            if constexpr (sizeof(R) == 4) {
#pragma unroll
                for (int g = 0; g < A; g += 2) {
                    const C<R> x = amp(cl, at(g)), y = amp(cl, at(g + 1));
                    v.re[g / 2] = pk(x.x, y.x);
                    v.im[g / 2] = pk(x.y, y.y);
                    if (REV) {
                        const C<R> p = amp(cb, at(g)), q = amp(cb, at(g + 1));
                        w.re[g / 2] = pk(p.x, q.x);
                        w.im[g / 2] = pk(p.y, q.y);
                    }
                }
            } else {
#pragma unroll
                for (int g = 0; g < A; ++g) {
                    v.set(g, amp(cl, at(g)));
                    if (REV) w.set(g, amp(cb, at(g)));
                }
            }
            C<R> tf = mk<R>(1, 0);
            bool has_tf = false;
            uint32_t neg = 0;
            for (uint32_t o = ph.op_begin, oe = ph.op_begin + ph.nops; o < oe; ++o)
                t_step<R, A, NS, WIDE>(v, w, sop[o], scf, sacc, base, tbase, rbit, tf, has_tf, neg);
            if (has_tf) {
#pragma unroll
                for (int g = 0; g < A; ++g) {
                    v.set(g, tprod<R>(tf, v.get(g)));
                    if (REV) w.set(g, tprod<R>(tf, w.get(g)));
                }
            }
            if (ph.signs) {
#pragma unroll
                for (int g = 0; g < A; ++g) {
                    v.set(g, flip_sign<R>(v.get(g), neg));
                    if (REV) w.set(g, flip_sign<R>(w.get(g), neg));
                }
            }
#pragma unroll
            for (int g = 0; g < A; ++g) {
                amp(cl, at(g)) = v.get(g);
                if (REV) amp(cb, at(g)) = w.get(g);
            }
            __syncthreads();
        }
        if (store) {
            auto chunk = [&](const char *t, uint32_t f) {
                if constexpr (V == 2) {
                    const C<R> x = *reinterpret_cast<const C<R> *>(t + f);
                    const C<R> y = *reinterpret_cast<const C<R> *>(t + (f ^ sg.fcol[0]));
                    return make_float4(x.x, x.y, y.x, y.y);
                } else {
                    return *reinterpret_cast<const float4 *>(t + f);
                }
            };
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const Chunk c = s_ch[j];
                if (outside(c)) continue;
                const uint32_t f = f0 ^ c.f;
                if (a_out) *reinterpret_cast<float4 *>(reinterpret_cast<char *>(a_out + start) + c.off) = chunk(cl, f);
                if (REV) *reinterpret_cast<float4 *>(reinterpret_cast<char *>(b + start) + c.off) = chunk(cb, f);
            }
        }
        __syncthreads();  // the buffer is refilled next
        if (AHEAD && !fresh && !padded) cur ^= 1u;
    }
}

}  // namespace steps
}  // namespace b200sv
