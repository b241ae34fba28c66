// sv_batch_tiles.cuh — batched circuits run level by level over shared-memory tiles in registers.
//
// Part of sv_batch.cu (included there once).  Serves every batch without two-wire dense gates,
// double excitations or matrices on two and more wires; those run in k_batch.
//
// Each circuit is cut into segments, runs of steps whose bits fit one tile of 2^kt amplitudes,
// with look-ahead over commuting steps.  Segment l of every circuit belongs to level l, and one
// launch runs a level: a CTA takes a few tiles of one circuit's segment, so a launch holds
// (circuits x tiles) independent pieces of work and nothing waits on another CTA.  One wide
// circuit spreads over the whole GPU this way: a training step over 192 circuits of 10-18 qubits,
// complex128, went from 121.5 ms (one CTA per circuit: the widest circuits' chains of tiles ran alone
// at the end) to 7.4 ms, and the 1024-circuit step of 16 qubits, complex64, from 70.2 to 23.9 ms (fewer
// barriers and shared-memory passes between steps, three 256-thread CTAs an SM instead of one of 512).
// Circuits narrower than a tile are one tile of their own size in CTAs of fewer threads,
// launched beside the wide ones.
//
// Inside a tile the steps run in registers: a thread holds A = 2^a amplitudes (of lambda and of
// the bra in the reverse sweep) that differ in the phase's a register bits, a phase takes every
// ready step whose target fits those bits, and only the hand-over between phases goes through the
// XOR-swizzled tile.  Adjacent single-wire gates on one wire are one step, their product formed in
// FP64 per launch (k_tile_coefs).  A differentiated step's generator products all come from four
// sums over its amplitude pairs, S = (sum Im b0* a0, sum Im b1* a1, sum Im b0* a1 + Im b1* a0,
// sum Re b0* a1 - Re b1* a0), accumulated in FP64: member k of the step has
// Im<b|G_k|a> = h_k . S with h_k = (h00, h11, Re h01, Im h01) of the Hermitian
// H_k = A_k^dagger G_k A_k, A_k the product of the inverses undone before it.

namespace tiles {

// One gate of one circuit, as its coefficients are formed (per circuit; the plan is shared by all
// circuits of the same structure).
struct Mem {
    uint8_t form, gate, inv, nt;
    int32_t pslot, gslot;
    uint32_t cidx;
};

enum SKind : uint8_t { S_RUN = 0, S_DIAGRUN = 1, S_DENSE = 2, S_DIAG = 3, S_PARITY = 4, S_NONE = 5 };
// How a step's coefficients are formed: members in op order, index into the plan's member list.
struct CoefStep {
    uint32_t mem_begin, coef;  // coef: position in the circuit's coefficient array of this direction
    uint16_t nmem;
    uint8_t kind, nt, nbits;   // S_DIAG: target count, index bits
    uint8_t src[3];            // S_DIAG: index bit (2 - j) of the table is the gate's bit src[j] (255: none)
};

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
};

struct alignas(16) TOp {
    uint16_t code, coef;   // coef: position in the segment's coefficients
    uint16_t creg;         // controls among the register bits
    uint16_t grad;         // 1 + gradient row of the segment, 0: not differentiated
    uint32_t cthr;         // controls among the thread bits (tile positions)
    uint32_t pm;           // parity: tile bits
    uint64_t pmg;          // parity: state bits outside the tile
    uint8_t p0, p1, p2, pad;
    uint32_t dsign;        // T_DIAG with a gradient: generator entry of index i in bits 2i (1: +1, 2: -1)
};
// CNOT and SWAP steps move no data.  A segment keeps a GF(2)-linear map from the tile position of an
// amplitude to the place where it lies in shared memory; a CNOT between phases replaces the column of
// its control bit by (control column XOR target column), and the tile's store reads through the last
// map.  A phase loads and stores its amplitudes through its map: places, not positions, so no thread
// touches another's amplitudes and no extra barrier is needed.
struct TPhase {
    uint16_t op_begin, nops;
    uint8_t rb[4];     // register bits (tile positions, ascending)
    uint8_t rt[4];     // tile position of register bit j
    uint16_t tcol[8];  // place of each thread index bit (swizzled)
    uint16_t rcol[4];  // place of each register bit (swizzled)
    uint32_t pad;
};
struct alignas(16) TSeg {
    uint32_t ph_begin, nph, op_begin, nops;
    uint32_t coef_begin, ncoef, ngrad;
    uint8_t lbits[16];
    uint8_t gbits[32];
    uint16_t fcol[12];  // places of the tile bits when the tile is stored (swizzled)
    uint8_t ng, kt, pad[2];
};
struct alignas(16) Job {
    uint32_t seg, circ;
    uint32_t tile0, ntiles;
    uint32_t nparts, part;
    uint32_t flags;    // 1: the state is |0..0> before this segment; 2: nothing reads the tiles afterwards
    uint32_t pad;
    uint64_t gpart;    // first partial sum of the segment
};
struct TCirc {
    uint64_t off;              // first amplitude in either pool
    uint64_t coef[2];          // first coefficient, forward / reverse
    uint32_t n;
    uint32_t term_begin, nterms, nobs, out_begin;
};

template <typename R, bool REV> struct TGeo;
template <> struct TGeo<float, false> { static constexpr int kt = 12, a = 4, A = 16, reserve = 4, minb = 3; };
template <> struct TGeo<float, true> { static constexpr int kt = 12, a = 4, A = 16, reserve = 4, minb = 2; };
template <> struct TGeo<double, false> { static constexpr int kt = 12, a = 4, A = 16, reserve = 3, minb = 2; };
template <> struct TGeo<double, true> { static constexpr int kt = 11, a = 3, A = 8, reserve = 3, minb = 2; };
constexpr int kTThreads = 256;
constexpr int kTWarps = kTThreads / 32;
constexpr int kMaxTOps = 160, kMaxTCoefs = 640, kMaxTGrads = 64;
constexpr int kChunkBits = 12;  // amplitudes of one block of the measurement kernels: 16 a thread

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

struct TArgs {
    const Job *jobs;
    const TCirc *circs;
    const TSeg *segs;
    const TPhase *phases;
    const TOp *ops;
    const void *coefs;
    void *pool_a, *pool_b;
    double *gpart;
    const int *skip;  // forward inside a VJP: nonzero when pool A already holds the states
};

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
// the four sums of a differentiated step on register bit BIT: each pair's values in the state's
// precision, the sums in FP64
template <typename R, int A, int BIT, bool CTL>
__device__ __forceinline__ void t_cross(const Regs<R, A> &v, const Regs<R, A> &w, uint32_t creg, double (&s)[4]) {
    constexpr int B = 1 << BIT;
    if constexpr (sizeof(R) == 4 && BIT > 0 && !CTL) {
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
            const C<R> a0 = v.get(g), a1 = v.get(g | B), b0 = w.get(g), b1 = w.get(g | B);
            s[0] += (double)fma(b0.x, a0.y, -(b0.y * a0.x));
            s[1] += (double)fma(b1.x, a1.y, -(b1.y * a1.x));
            s[2] += (double)fma(-b1.y, a0.x, fma(b1.x, a0.y, fma(-b0.y, a1.x, b0.x * a1.y)));
            s[3] += (double)fma(-b1.y, a0.y, fma(-b1.x, a0.x, fma(b0.y, a1.y, b0.x * a1.x)));
        }
    }
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

// One step on the thread's amplitudes of NS states (w is v where there is one state).
template <typename R, int A, int NS>
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
        if (grad) t_cross<R, A, b, false>(v, w, 0, s);                                                         \
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
                const C<R> a = v.get(g), b = w.get(g);
                const double im = (double)fma(b.x, a.y, -(b.y * a.x));
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
                const C<R> a = v.get(g), b = w.get(g);
                const double im = (double)fma(b.x, a.y, -(b.y * a.x));
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
                if (on) t_cross<R, A, b, true>(v, w, op.creg, s);                                              \
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
    default: break;
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

// One job: a few tiles of one circuit's segment.  Forward: one state; REV: lambda (pool A) and the
// bra (pool B).  256 threads (fewer for narrow circuits) and one tile buffer per state; the two or
// three CTAs an SM holds overlap one another's tile moves, staging and barriers.
template <typename R, bool REV>
__global__ void __launch_bounds__(kTThreads, TGeo<R, REV>::minb) k_tiles(TArgs args) {
    using G = TGeo<R, REV>;
    constexpr int A = G::A, NS = REV ? 2 : 1;
    constexpr int V = 16 / (int)sizeof(C<R>);
    constexpr int PER = A / V;
    if (args.skip && *args.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TSeg sg;
    __shared__ uint64_t s_hi[PER];
    const Job jb = args.jobs[blockIdx.x];
    if (threadIdx.x < sizeof(TSeg) / 8)
        reinterpret_cast<uint64_t *>(&sg)[threadIdx.x] = reinterpret_cast<const uint64_t *>(args.segs + jb.seg)[threadIdx.x];
    __syncthreads();
    const uint32_t NT = blockDim.x, TN = NT * A;
    C<R> *const sl = reinterpret_cast<C<R> *>(smem_raw);
    C<R> *const sb = sl + TN;
    TOp *const sop = reinterpret_cast<TOp *>(smem_raw + NS * sizeof(C<R>) * TN);
    C<R> *const scf = reinterpret_cast<C<R> *>(sop + sg.nops);
    TPhase *const sph = reinterpret_cast<TPhase *>(scf + sg.ncoef);
    double *const sacc = reinterpret_cast<double *>(sph + sg.nph);
    const TCirc &circ = args.circs[jb.circ];
    const uint64_t off = circ.off, namp = uint64_t(1) << circ.n;
    copy_words(sop, args.ops + sg.op_begin, sg.nops);
    copy_words(scf, static_cast<const C<R> *>(args.coefs) + circ.coef[REV ? 1 : 0] + sg.coef_begin, sg.ncoef);
    copy_words(sph, args.phases + sg.ph_begin, sg.nph);
    if (REV)
        for (uint32_t i = threadIdx.x; i < sg.ngrad * 4 * kTWarps; i += NT) sacc[i] = 0.0;
    if (threadIdx.x < PER) s_hi[threadIdx.x] = spread((uint64_t)threadIdx.x * NT * V, sg.lbits, sg.kt);
    const uint64_t lo = spread((uint64_t)threadIdx.x * V, sg.lbits, sg.kt);
    C<R> *const ga = static_cast<C<R> *>(args.pool_a) + off;
    C<R> *const gb = REV ? static_cast<C<R> *>(args.pool_b) + off : nullptr;
    auto sw = [&](int j) { return tswz<R>((threadIdx.x + (uint32_t)j * NT) * V); };
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    for (uint32_t t = jb.tile0; t < jb.tile0 + jb.ntiles; ++t) {
        const uint64_t tbase = spread(t, sg.gbits, sg.ng);
        const bool fresh = !REV && (jb.flags & 1u);
        if (fresh && t != 0) {  // |0..0> has no amplitude here, and a segment keeps zeros
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const uint64_t x = tbase | lo | s_hi[j];
                if (x < namp) *reinterpret_cast<float4 *>(ga + x) = z4;
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint64_t x = tbase | lo | s_hi[j];  // beyond the state in a tile padded to a warp's share
            if (!fresh && x < namp) {
                cp_async16(sl + sw(j), ga + x);
                if (REV) cp_async16(sb + sw(j), gb + x);
            } else {
                *reinterpret_cast<float4 *>(sl + sw(j)) = z4;
                if (REV) *reinterpret_cast<float4 *>(sb + sw(j)) = z4;
            }
        }
        cp_async_commit();
        cp_async_wait0();
        if (fresh && threadIdx.x == 0) sl[0] = mk<R>(1, 0);  // thread 0 zeroed position 0 itself
        __syncthreads();
        for (uint32_t p = 0; p < sg.nph; ++p) {
            const TPhase ph = sph[p];
            uint32_t base = threadIdx.x, sbase = 0, rbit[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < G::a; ++j) {
                rbit[j] = 1u << ph.rt[j];
                const uint32_t low = base & ((1u << ph.rb[j]) - 1u);
                base = ((base ^ low) << 1) | low;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) sbase ^= (threadIdx.x >> j) & 1u ? ph.tcol[j] : 0u;
            auto at = [&](int g) {
                uint32_t x = sbase;
#pragma unroll
                for (int j = 0; j < G::a; ++j)
                    if ((g >> j) & 1) x ^= ph.rcol[j];
                return x;
            };
            Regs<R, A> v, w;
            if constexpr (sizeof(R) == 4) {
#pragma unroll
                for (int g = 0; g < A; g += 2) {
                    const C<R> x = sl[at(g)], y = sl[at(g + 1)];
                    v.re[g / 2] = pk(x.x, y.x);
                    v.im[g / 2] = pk(x.y, y.y);
                    if (REV) {
                        const C<R> p = sb[at(g)], q = sb[at(g + 1)];
                        w.re[g / 2] = pk(p.x, q.x);
                        w.im[g / 2] = pk(p.y, q.y);
                    }
                }
            } else {
#pragma unroll
                for (int g = 0; g < A; ++g) {
                    v.set(g, sl[at(g)]);
                    if (REV) w.set(g, sb[at(g)]);
                }
            }
            C<R> tf = mk<R>(1, 0);
            bool has_tf = false;
            uint32_t neg = 0;
            for (uint32_t o = ph.op_begin, oe = ph.op_begin + ph.nops; o < oe; ++o)
                t_step<R, A, NS>(v, w, sop[o], scf, sacc, base, tbase, rbit, tf, has_tf, neg);
            if (has_tf) {
#pragma unroll
                for (int g = 0; g < A; ++g) {
                    v.set(g, tprod<R>(tf, v.get(g)));
                    if (REV) w.set(g, tprod<R>(tf, w.get(g)));
                }
            }
#pragma unroll
            for (int g = 0; g < A; ++g) {
                sl[at(g)] = flip_sign<R>(v.get(g), neg);
                if (REV) sb[at(g)] = flip_sign<R>(w.get(g), neg);
            }
            __syncthreads();
        }
        if (!(jb.flags & 2u)) {
            constexpr int LV = V == 2 ? 1 : 0;
            const int lt = 31 - __clz((int)NT);
            uint32_t f0 = 0;
            for (int i = 0; i < lt; ++i) f0 ^= (threadIdx.x >> i) & 1u ? sg.fcol[LV + i] : 0u;
            auto chunk = [&](const C<R> *t, uint32_t f) {
                if constexpr (V == 2) {
                    const C<R> x = t[f], y = t[f ^ sg.fcol[0]];
                    return make_float4(x.x, x.y, y.x, y.y);
                } else {
                    return *reinterpret_cast<const float4 *>(t + f);
                }
            };
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const uint64_t x = tbase | lo | s_hi[j];
                uint32_t f = f0;
#pragma unroll
                for (int i = 0; (1 << i) < PER; ++i)
                    if ((j >> i) & 1) f ^= sg.fcol[LV + lt + i];
                if (x < namp) {
                    *reinterpret_cast<float4 *>(ga + x) = chunk(sl, f);
                    if (REV) *reinterpret_cast<float4 *>(gb + x) = chunk(sb, f);
                }
            }
        }
        __syncthreads();  // the buffer is refilled next
    }
    if (REV) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < sg.ngrad * 4; i += NT) {
            double s = 0.0;
            for (uint32_t k = 0; k < (NT >> 5); ++k) s += sacc[i * kTWarps + k];
            args.gpart[jb.gpart + (uint64_t)i * jb.nparts + jb.part] = s;
        }
    }
}

// ---- coefficients of one launch ---------------------------------------------------------------
struct CoefArgs {
    const CoefStep *steps;       // of every plan
    const uint32_t *mem_list;    // op indices of the steps' members
    const uint32_t *step_begin;  // per circuit: first step of its plan and direction
    const uint32_t *step_count;
    const uint64_t *mem_base;    // per circuit: first Mem
    const Mem *mems;
    const TCirc *circs;
    const double4 *cs;
    const double2 *consts;
    void *coefs;
    double4 *h;                  // REV: per gradient slot
    uint32_t ncirc;
    int rev;
};
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ void mul22(const double2 (&x)[4], const double2 (&y)[4], double2 (&r)[4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) r[i * 2 + j] = zadd(zmul(x[i * 2], y[j]), zmul(x[i * 2 + 1], y[2 + j]));
}
// h of generator code 1 X, 2 Y, 3 Z, 4 |1><1| seen through A (H = A^dagger G A)
__device__ __forceinline__ double4 gen_row(int code, const double2 (&Am)[4]) {
    const double2 z = make_double2(0, 0), one = make_double2(1, 0);
    double2 Gm[4] = {z, z, z, z};
    if (code == 1) Gm[1] = Gm[2] = one;
    else if (code == 2) { Gm[1] = make_double2(0, -1); Gm[2] = make_double2(0, 1); }
    else if (code == 3) { Gm[0] = one; Gm[3] = make_double2(-1, 0); }
    else Gm[3] = one;
    double2 GA[4];
    mul22(Gm, Am, GA);
    const double2 h01 = zadd(zmul(zconj(Am[0]), GA[1]), zmul(zconj(Am[2]), GA[3]));
    return make_double4(zadd(zmul(zconj(Am[0]), GA[0]), zmul(zconj(Am[2]), GA[2])).x,
                        zadd(zmul(zconj(Am[1]), GA[1]), zmul(zconj(Am[3]), GA[3])).x, h01.x, h01.y);
}
__device__ __forceinline__ int gen_code(uint8_t gate) {
    switch (gate) {
    case B200SV_RX: case B200SV_CRX: return 1;
    case B200SV_RY: case B200SV_CRY: return 2;
    case B200SV_RZ: return 3;
    case B200SV_PhaseShift: return 4;
    default: return 0;
    }
}

template <typename R> __global__ void k_tile_coefs(CoefArgs a) {
    const bool rev = a.rev != 0;
    for (uint32_t c = blockIdx.y; c < a.ncirc; c += gridDim.y) {
        const Mem *mems = a.mems + a.mem_base[c];
        C<R> *out = static_cast<C<R> *>(a.coefs) + a.circs[c].coef[a.rev];
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.step_count[c]; i += gridDim.x * blockDim.x) {
            const CoefStep st = a.steps[a.step_begin[c] + i];
            const uint32_t *list = a.mem_list + st.mem_begin;
            C<R> *o = out + st.coef;
            if (st.kind == S_RUN || st.kind == S_DIAGRUN) {
                double2 P[4] = {make_double2(1, 0), make_double2(0, 0), make_double2(0, 0), make_double2(1, 0)};
                for (int k = 0; k < st.nmem; ++k) {
                    const Mem &m = mems[list[rev ? st.nmem - 1 - k : k]];
                    if (rev && m.gslot >= 0) a.h[m.gslot] = gen_row(gen_code(m.gate), P);
                    C<double> q[4];
                    member_mat<double>(m, a.cs, a.consts, rev, q);
                    double2 N[4];
                    mul22(q, P, N);
                    for (int e = 0; e < 4; ++e) P[e] = N[e];
                }
                if (st.kind == S_RUN) {
                    for (int e = 0; e < 4; ++e) o[e] = mk<R>((R)P[e].x, (R)P[e].y);
                } else {  // a table whose lowest index bit is the run's bit
                    for (int e = 0; e < 8; ++e) o[e] = mk<R>((R)P[(e & 1) * 3].x, (R)P[(e & 1) * 3].y);
                }
                continue;
            }
            if (st.kind == S_NONE) continue;
            const Mem &m = mems[list[0]];
            C<double> t[4];
            op_coeffs<double, 4>(m, a.cs, a.consts, rev, t);
            if (st.kind == S_DENSE) {
                if (rev && m.gslot >= 0) {
                    const double2 id[4] = {make_double2(1, 0), make_double2(0, 0), make_double2(0, 0), make_double2(1, 0)};
                    a.h[m.gslot] = gen_row(gen_code(m.gate), id);
                }
                for (int e = 0; e < 4; ++e) o[e] = mk<R>((R)t[e].x, (R)t[e].y);
                continue;
            }
            if (rev && m.gslot >= 0) a.h[m.gslot] = make_double4(1, 0, 0, 0);
            if (st.kind == S_PARITY) {
                for (int e = 0; e < 2; ++e) o[e] = mk<R>((R)t[e].x, (R)t[e].y);
                continue;
            }
            // S_DIAG: targets first in the gate's bit list, then controls (entry 1 where one is clear)
            for (int e = 0; e < 8; ++e) {
                uint32_t v = 0;
                for (int j = 0; j < 3; ++j)
                    if (((e >> (2 - j)) & 1) && st.src[j] < 3) v |= 1u << st.src[j];
                int row = 0;
                bool all = true;
                for (int j = 0; j < st.nbits; ++j) {
                    if (j < st.nt) row = row * 2 + (int)((v >> j) & 1u);
                    else all = all && ((v >> j) & 1u);
                }
                o[e] = all ? mk<R>((R)t[row].x, (R)t[row].y) : mk<R>(1, 0);
            }
        }
    }
}

// gradw[g] = h_g . (sums of its step over the segment's parts)
struct GradRef {
    uint64_t base;
    uint32_t nparts, pad;
};
__global__ void k_tile_grads(const GradRef *__restrict__ refs, const double4 *__restrict__ h,
                             const double *__restrict__ gpart, uint32_t n, double *__restrict__ gradw) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        const GradRef r = refs[g];
        double s[4];
        for (int v = 0; v < 4; ++v) {
            s[v] = 0.0;
            for (uint32_t p = 0; p < r.nparts; ++p) s[v] += gpart[r.base + (uint64_t)v * r.nparts + p];
        }
        const double4 q = h[g];
        gradw[g] = q.x * s[0] + q.y * s[1] + q.z * s[2] + q.w * s[3];
    }
}

// ---- measurement and bra ------------------------------------------------------------------------
// Walsh-Hadamard transform of 16 register values (index bit j <-> register bit j).
__device__ __forceinline__ void wht16(double (&x)[16]) {
#pragma unroll
    for (int s = 1; s < 16; s <<= 1)
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (!(i & s)) {
                const double u = x[i], w = x[i | s];
                x[i] = u + w;
                x[i | s] = u - w;
            }
}

// A block takes a chunk of up to 4096 amplitudes of one circuit, thread t the amplitudes t + 256 r.
// Diagonal words: the transform of the thread's 16 probabilities over r holds sum_r (-1)^{z.r} p_r
// for every z, so a word costs one shared-memory read per thread instead of 16 signed additions.
// Words with X factors read their partners from the state.  part[term * chunks + chunk].
struct ChunkJob {
    uint32_t circ, chunk, nchunks, pad;
    uint64_t part;
};
template <typename R>
__global__ void __launch_bounds__(kTThreads) k_tile_expval(const ChunkJob *__restrict__ jobs, const TCirc *__restrict__ circs,
                                                           const DTerm *__restrict__ terms, const void *pool,
                                                           double *__restrict__ part) {
    __shared__ double hat[16][kTThreads];
    __shared__ double s_w[4][kTWarps];
    const ChunkJob jb = jobs[blockIdx.x];
    const TCirc c = circs[jb.circ];
    const C<R> *psi = static_cast<const C<R> *>(pool) + c.off;
    const uint64_t namp = uint64_t(1) << c.n, base = (uint64_t)jb.chunk << kChunkBits;
    double x[16];
    C<R> v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const uint64_t i = base + threadIdx.x + ((uint64_t)r << 8);
        v[r] = i < namp ? psi[i] : mk<R>(0, 0);
        const double2 a = widen<R>(v[r]);
        x[r] = a.x * a.x + a.y * a.y;
    }
    wht16(x);
#pragma unroll
    for (int r = 0; r < 16; ++r) hat[r][threadIdx.x] = x[r];
    const uint64_t mine = base + threadIdx.x;
    const DTerm *T = terms + c.term_begin;
    for (uint32_t t0 = 0; t0 < c.nterms; t0 += 4) {
        double s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            s[k] = 0.0;
            if (t0 + k >= c.nterms) continue;
            const DTerm tm = T[t0 + k];
            if (tm.xmask == 0) {
                const double p = hat[(tm.zmask >> 8) & 15u][threadIdx.x];
                s[k] = (__popcll(mine & (tm.zmask & ~uint64_t(0xf00))) & 1) ? -p : p;
                continue;
            }
            double acc = 0.0;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const uint64_t i = mine + ((uint64_t)r << 8);
                if (i >= namp) continue;
                // Re conj(psi_{i^X}) i^ny (-1)^{|i&Z|} psi_i
                const double2 vi = widen<R>(v[r]), vj = widen<R>(psi[i ^ tm.xmask]);
                const double q = (tm.ny & 1) ? vj.y * vi.x - vj.x * vi.y : vj.x * vi.x + vj.y * vi.y;
                acc += (__popcll(i & tm.zmask) & 1) ? -q : q;
            }
            // i^ny: ny = 0 Re, 1 -Im, 2 -Re, 3 Im; q above is Re or -Im
            s[k] = (tm.ny & 2) ? -acc : acc;
        }
        const double r = reduce4(s);
        const int lane = threadIdx.x & 31;
        if ((lane & 7) == 0) s_w[lane >> 3][threadIdx.x >> 5] = r;
        __syncthreads();
        if (threadIdx.x < 4 && t0 + threadIdx.x < c.nterms) {
            double sum = 0.0;
            for (int k = 0; k < kTWarps; ++k) sum += s_w[threadIdx.x][k];
            part[jb.part + (uint64_t)(t0 + threadIdx.x) * jb.nchunks + jb.chunk] = sum;
        }
        __syncthreads();
    }
}
// out[obs] = sum over its terms of coeff * (sum over chunks), terms and chunks in order
struct ObsRef {
    uint64_t part;        // first partial of the circuit
    uint32_t circ, obs, nchunks, pad;
};
__global__ void k_tile_outputs(const ObsRef *__restrict__ refs, uint32_t n, const TCirc *__restrict__ circs,
                               const DTerm *__restrict__ terms, const double *__restrict__ part,
                               double *__restrict__ out) {
    for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += gridDim.x * (blockDim.x >> 5)) {
        const ObsRef r = refs[i];  // one warp per output
        const TCirc &c = circs[r.circ];
        double sum = 0.0;
        for (uint32_t t = threadIdx.x & 31; t < c.nterms; t += 32) {
            const DTerm &tm = terms[c.term_begin + t];
            if (tm.obs != r.obs) continue;
            double s = 0.0;
            for (uint32_t k = 0; k < r.nchunks; ++k) s += part[r.part + (uint64_t)t * r.nchunks + k];
            sum += tm.coeff * s;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if ((threadIdx.x & 31) == 0) out[c.out_begin + r.obs] = sum;
    }
}

// bra_j = sum_t w_t (P_t psi)_j, w_t = coeff * dy of the term's output.  The diagonal words' factor
// sum_t +-w_t of a thread's 16 amplitudes is formed in the transform's index (one addition per word)
// and transformed back.
template <typename R>
__global__ void __launch_bounds__(kTThreads) k_tile_bra(const ChunkJob *__restrict__ jobs, const TCirc *__restrict__ circs,
                                                        const DTerm *__restrict__ terms, const void *pool, void *pool_b,
                                                        const double *__restrict__ dy) {
    __shared__ double hat[16][kTThreads];
    const ChunkJob jb = jobs[blockIdx.x];
    const TCirc c = circs[jb.circ];
    const C<R> *psi = static_cast<const C<R> *>(pool) + c.off;
    C<R> *bra = static_cast<C<R> *>(pool_b) + c.off;
    const uint64_t namp = uint64_t(1) << c.n, mine = ((uint64_t)jb.chunk << kChunkBits) + threadIdx.x;
    const DTerm *T = terms + c.term_begin;
    const double *d = dy + c.out_begin;
#pragma unroll
    for (int r = 0; r < 16; ++r) hat[r][threadIdx.x] = 0.0;
    bool flips = false;
    for (uint32_t t = 0; t < c.nterms; ++t) {
        const DTerm tm = T[t];
        if (tm.xmask != 0) {
            flips = true;
            continue;
        }
        const double w = tm.coeff * d[tm.obs];
        if (w == 0.0) continue;
        hat[(tm.zmask >> 8) & 15u][threadIdx.x] += (__popcll(mine & (tm.zmask & ~uint64_t(0xf00))) & 1) ? -w : w;
    }
    double x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = hat[r][threadIdx.x];
    wht16(x);
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const uint64_t j = mine + ((uint64_t)r << 8);
        if (j >= namp) continue;
        const double2 p = widen<R>(psi[j]);
        // no factor, no contribution: an unused output leaves the bra at zero whatever psi holds
        double br = x[r] != 0.0 ? x[r] * p.x : 0.0, bi = x[r] != 0.0 ? x[r] * p.y : 0.0;
        if (flips) {
            for (uint32_t t = 0; t < c.nterms; ++t) {
                const DTerm tm = T[t];
                if (tm.xmask == 0) continue;
                const double w = tm.coeff * d[tm.obs];
                if (w == 0.0) continue;
                const uint64_t i = j ^ tm.xmask;
                const double2 q = widen<R>(psi[i]);
                const double f = (__popcll(i & tm.zmask) & 1) ? -w : w;
                switch (tm.ny & 3) {
                case 0: br += f * q.x; bi += f * q.y; break;
                case 1: br -= f * q.y; bi += f * q.x; break;
                case 2: br -= f * q.x; bi -= f * q.y; break;
                default: br += f * q.y; bi -= f * q.x; break;
                }
            }
        }
        bra[j] = mk<R>((R)br, (R)bi);
    }
}

// The device program of a batch: plans shared by circuits of one structure, per-circuit tables,
// and one list of jobs per launch.
struct Launch {
    uint32_t first, njobs, threads, smem, level;
};
struct Program {
    TCirc *circs = nullptr;
    TSeg *segs = nullptr;
    TPhase *phases = nullptr;
    TOp *ops = nullptr;
    Job *jobs = nullptr;
    Mem *mems = nullptr;
    uint64_t *mem_base = nullptr;
    CoefStep *steps = nullptr;
    uint32_t *mem_list = nullptr, *step_begin[2] = {}, *step_count[2] = {};
    void *coefs[2] = {};
    double4 *h = nullptr;
    double *gpart = nullptr, *opart = nullptr;
    GradRef *grefs = nullptr;
    ChunkJob *chunks = nullptr;
    ObsRef *orefs = nullptr;
    uint32_t nchunks = 0, max_steps[2] = {};
    std::vector<Launch> launches[2];  // forward, reverse: level by level
};

}  // namespace tiles
