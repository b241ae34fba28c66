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
// at the end) to 6.35 ms, and the 1024-circuit step of 16 qubits, complex64, from 70.2 to 22.3 ms (fewer
// barriers and shared-memory passes between steps, two 256-thread CTAs an SM, three in the complex64
// forward sweep, instead of one of 512).
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
using namespace steps;

// One gate of one circuit, as its coefficients are formed (per circuit; the plan is shared by all
// circuits of the same structure).
struct Mem {
    uint8_t form, gate, inv, nt;
    int32_t pslot, gslot;
    uint32_t cidx;
};

// How a step's coefficients are formed: members in op order, index into the plan's member list.
struct CoefStep {
    uint32_t mem_begin, nmem;  // a run has any number of members
    uint32_t coef;             // position in the circuit's coefficient array of this direction
    uint8_t kind, nt, nbits;   // S_DIAG: target count, index bits
    uint8_t src[3];            // S_DIAG: index bit (2 - j) of the table is the gate's bit src[j] (255: none)
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

constexpr int kChunkBits = 12;  // amplitudes of one block of the measurement kernels: 16 a thread

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

// One job: a few tiles of one circuit's segment.  Forward: one state; REV: lambda (pool A) and the
// bra (pool B).  256 threads (fewer for narrow circuits); the two or three CTAs an SM holds overlap one
// another's tile moves, staging and barriers.
template <typename R, bool REV>
__global__ void __launch_bounds__(kTThreads, TGeo<R, REV>::minb) k_tiles(TArgs args) {
    using G = TGeo<R, REV>;
    constexpr int A = G::A;
    if (args.skip && *args.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TSeg sg;
    const Job jb = args.jobs[blockIdx.x];
    if (threadIdx.x < sizeof(TSeg) / 8)
        reinterpret_cast<uint64_t *>(&sg)[threadIdx.x] = reinterpret_cast<const uint64_t *>(args.segs + jb.seg)[threadIdx.x];
    __syncthreads();
    const uint32_t NT = blockDim.x, TN = NT * A;
    C<R> *const sl = reinterpret_cast<C<R> *>(smem_raw);
    C<R> *const sb = sl + TN;
    TOp *const sop = reinterpret_cast<TOp *>(smem_raw + tile_buffers<R, REV>() * sizeof(C<R>) * TN);
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
    C<R> *const ga = static_cast<C<R> *>(args.pool_a) + off;
    C<R> *const gb = REV ? static_cast<C<R> *>(args.pool_b) + off : nullptr;
    __syncthreads();
    run_tiles<R, REV, false>(sg, sl, sb, sop, scf, sph, sacc, jb.tile0, uint64_t(jb.tile0) + jb.ntiles, 1,
                             !REV && (jb.flags & 1u), !(jb.flags & 2u), ga, ga, gb, namp);
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
// A 2x2 matrix in twice FP64's length, h + l.  complex128 runs are multiplied so and rounded once (as the
// single-state engine does on the host, sv_fused.cu): what their coefficients miss is the same on every
// amplitude and adds up in the values.
struct Mat2 {
    double2 h[4], l[4];
};
struct Twofold {  // sum of products with its low part
    double h, l;
    __device__ __forceinline__ void add(double a, double al, double b, double bl) {
        const double p = a * b, u = h + p, z = u - h;
        l += ((h - (u - z)) + (p - z)) + fma(a, b, -p) + fma(a, bl, al * b);
        h = u;
    }
};
__device__ __forceinline__ void mul22(const Mat2 &x, Mat2 &y) {  // y = x y
    Mat2 r;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            Twofold re{0.0, 0.0}, im{0.0, 0.0};
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const double2 a = x.h[i * 2 + k], al = x.l[i * 2 + k], b = y.h[k * 2 + j], bl = y.l[k * 2 + j];
                re.add(a.x, al.x, b.x, bl.x);
                re.add(-a.y, -al.y, b.y, bl.y);
                im.add(a.x, al.x, b.y, bl.y);
                im.add(a.y, al.y, b.x, bl.x);
            }
            r.h[i * 2 + j] = make_double2(re.h + re.l, im.h + im.l);
            r.l[i * 2 + j] = make_double2(re.l - (r.h[i * 2 + j].x - re.h), im.l - (r.h[i * 2 + j].y - im.h));
        }
    y = r;
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
            if (st.kind == S_RUN || st.kind == S_SPLIT || st.kind == S_DIAGRUN) {
                const double2 zero = make_double2(0, 0), one = make_double2(1, 0);
                Mat2 run{{one, zero, zero, one}, {zero, zero, zero, zero}};
                double2(&P)[4] = run.h;
                for (uint32_t k = 0; k < st.nmem; ++k) {
                    const Mem &m = mems[list[rev ? st.nmem - 1 - k : k]];
                    if (rev && m.gslot >= 0) a.h[m.gslot] = gen_row(gen_code(m.gate), P);
                    Mat2 q{{}, {zero, zero, zero, zero}};
                    member_mat<double>(m, a.cs, a.consts, rev, q.h);
                    if (st.kind == S_SPLIT) {
                        if (m.form == F_DIAG) {
                            o[2] = mk<R>((R)q.h[0].x, (R)q.h[0].y);
                            o[3] = mk<R>((R)q.h[3].x, (R)q.h[3].y);
                        } else {
                            o[0] = mk<R>((R)q.h[0].x, (R)q.h[1].x);
                            o[1] = mk<R>((R)q.h[2].x, (R)q.h[3].x);
                        }
                    }
                    if constexpr (sizeof(R) == 8) {
                        mul22(q, run);
                    } else {
                        double2 N[4];
                        mul22(q.h, P, N);
                        for (int e = 0; e < 4; ++e) P[e] = N[e];
                    }
                }
                if (st.kind == S_RUN) {
                    for (int e = 0; e < 4; ++e) o[e] = mk<R>((R)P[e].x, (R)P[e].y);
                } else if (st.kind == S_DIAGRUN) {  // a table whose lowest index bit is the run's bit
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

// gradw[g] = h_g . (sums of its step over the segment's parts) for the gradients of a group; eight lanes a
// gradient, fixed order
struct GradRef {
    uint64_t base;
    uint32_t nparts, group;
};
__global__ void k_tile_grads(const GradRef *__restrict__ refs, const double4 *__restrict__ h,
                             const double *__restrict__ gpart, uint32_t n, uint32_t group, double *__restrict__ gradw) {
    const uint32_t sub = threadIdx.x & 7;
    for (uint32_t g0 = blockIdx.x * (blockDim.x >> 3); g0 < n; g0 += gridDim.x * (blockDim.x >> 3)) {
        const uint32_t g = g0 + (threadIdx.x >> 3);
        double s = 0.0;
        const GradRef r = g < n ? refs[g] : GradRef{0, 0, ~0u};
        const bool mine = g < n && r.group == group;
        if (mine) {
            const double4 q = h[g];
            const double hv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                double t = 0.0;
                for (uint32_t p = sub; p < r.nparts; p += 8) t += gpart[r.base + (uint64_t)v * r.nparts + p];
                s += hv[v] * t;
            }
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (mine && sub == 0) gradw[g] = s;
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
// Words with X factors read their partners from the chunk in shared memory, or from the state where
// the mask leaves the chunk.  A word's sign splits into one for the thread and a bit per r.  Words are
// summed four at a time over the warp and written per 64, so the block synchronises twice per 64 words
// (with a barrier per four words and partners from the state: 0.60 ms for 192 circuits of 10-18 qubits
// complex128, now 0.37; the bra 0.90 -> 0.40).  part[term * chunks + chunk].
struct ChunkJob {
    uint32_t circ, chunk, nchunks, pad;
    uint64_t part;
};
constexpr int kWordGroup = 64;
template <typename R> constexpr size_t chunk_smem() {
    return (sizeof(C<R>) << kChunkBits) + 16 * kTThreads * sizeof(double);
}
// A group of words in shared memory, each coefficient times its output's dy where dy is given (read from
// global memory, every word cost its latency); the block synchronises before and after.
__device__ __forceinline__ uint32_t stage_words(DTerm *dst, const DTerm *src, uint32_t n, const double *dy) {
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
        DTerm x = src[t];
        if (dy) x.coeff *= dy[x.obs];
        dst[t] = x;
    }
    __syncthreads();
    return n;
}
// bit r: parity of the word's bits 8..11 on r
__device__ __forceinline__ uint32_t row_signs(uint64_t z) {
    const uint32_t q = (uint32_t)(z >> 8) & 15u;
    return (q & 1u ? 0xAAAAu : 0u) ^ (q & 2u ? 0xCCCCu : 0u) ^ (q & 4u ? 0xF0F0u : 0u) ^ (q & 8u ? 0xFF00u : 0u);
}
__device__ __forceinline__ double signed_by(double x, uint32_t bit) {  // bit: 0 or 1
    return __hiloint2double(__double2hiint(x) ^ (int)(bit << 31), __double2loint(x));
}
// the chunk into shared memory, zeros beyond a narrow state
template <typename R>
__device__ __forceinline__ void load_chunk(C<R> *tile, const C<R> *psi, uint64_t base, uint64_t namp) {
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const uint32_t j = threadIdx.x + ((uint32_t)r << 8);
        tile[j] = base + j < namp ? psi[base + j] : mk<R>(0, 0);
    }
}
template <typename R>
__global__ void __launch_bounds__(kTThreads, 2) k_tile_expval(const ChunkJob *__restrict__ jobs, const TCirc *__restrict__ circs,
                                                           const DTerm *__restrict__ terms, const void *pool,
                                                           double *__restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_w[kWordGroup][kTWarps];
    __shared__ DTerm s_t[kWordGroup];
    C<R> *const tile = reinterpret_cast<C<R> *>(smem_raw);
    double (*const hat)[kTThreads] = reinterpret_cast<double (*)[kTThreads]>(tile + (1 << kChunkBits));
    const ChunkJob jb = jobs[blockIdx.x];
    const TCirc c = circs[jb.circ];
    const C<R> *psi = static_cast<const C<R> *>(pool) + c.off;
    const uint64_t namp = uint64_t(1) << c.n, base = (uint64_t)jb.chunk << kChunkBits;
    load_chunk<R>(tile, psi, base, namp);
    double x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const double2 a = widen<R>(tile[threadIdx.x + (r << 8)]);
        x[r] = a.x * a.x + a.y * a.y;
    }
    wht16(x);
#pragma unroll
    for (int r = 0; r < 16; ++r) hat[r][threadIdx.x] = x[r];
    const uint64_t mine = base + threadIdx.x;
    const DTerm *T = terms + c.term_begin;
    for (uint32_t g0 = 0; g0 < c.nterms; g0 += kWordGroup) {
        const uint32_t g1 = g0 + stage_words(s_t, T + g0, min(c.nterms - g0, (uint32_t)kWordGroup), nullptr);
        for (uint32_t t0 = g0; t0 < g1; t0 += 4) {
            double s[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s[k] = 0.0;
                if (t0 + k >= g1) continue;
                const DTerm &tm = s_t[t0 - g0 + k];
                const uint32_t neg = (uint32_t)__popcll(mine & (tm.zmask & ~uint64_t(0xf00))) & 1u;
                if (tm.xmask == 0) {
                    s[k] = signed_by(hat[(tm.zmask >> 8) & 15u][threadIdx.x], neg);
                    continue;
                }
                // Re conj(psi_{i^X}) i^ny (-1)^{|i&Z|} psi_i; i^ny takes the real part, or minus the
                // imaginary part, with the sign of ny's second bit
                const uint32_t rows = row_signs(tm.zmask), xl = (uint32_t)tm.xmask & ((1u << kChunkBits) - 1);
                const bool inside = (tm.xmask >> kChunkBits) == 0;
                const C<R> *other = psi + ((base ^ tm.xmask) & ~uint64_t((1 << kChunkBits) - 1));
                double acc = 0.0;
#pragma unroll 8
                for (int r = 0; r < 16; ++r) {
                    const uint32_t j = threadIdx.x + ((uint32_t)r << 8), o = j ^ xl;
                    if (j >= namp) break;  // a narrow state ends here for every later row
                    const double2 vi = widen<R>(tile[j]), vj = widen<R>(inside ? tile[o] : other[o]);
                    const double q = (tm.ny & 1) ? vj.y * vi.x - vj.x * vi.y : vj.x * vi.x + vj.y * vi.y;
                    acc += signed_by(q, (rows >> r) & 1u);
                }
                s[k] = signed_by(acc, neg ^ ((uint32_t)(tm.ny >> 1) & 1u));
            }
            const double r = reduce4(s);
            const int lane = threadIdx.x & 31;
            if ((lane & 7) == 0) s_w[t0 - g0 + (lane >> 3)][threadIdx.x >> 5] = r;
        }
        __syncthreads();
        if (threadIdx.x < g1 - g0) {
            double sum = 0.0;
            for (int k = 0; k < kTWarps; ++k) sum += s_w[threadIdx.x][k];
            part[jb.part + (uint64_t)(g0 + threadIdx.x) * jb.nchunks + jb.chunk] = sum;
        }
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
// and transformed back; words with X factors add their partners, word by word, to sums in registers.
template <typename R>
__global__ void __launch_bounds__(kTThreads, 2) k_tile_bra(const ChunkJob *__restrict__ jobs, const TCirc *__restrict__ circs,
                                                        const DTerm *__restrict__ terms, const void *pool, void *pool_b,
                                                        const double *__restrict__ dy) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C<R> *const tile = reinterpret_cast<C<R> *>(smem_raw);
    double (*const hat)[kTThreads] = reinterpret_cast<double (*)[kTThreads]>(tile + (1 << kChunkBits));
    const ChunkJob jb = jobs[blockIdx.x];
    const TCirc c = circs[jb.circ];
    const C<R> *psi = static_cast<const C<R> *>(pool) + c.off;
    C<R> *bra = static_cast<C<R> *>(pool_b) + c.off;
    const uint64_t namp = uint64_t(1) << c.n, base = (uint64_t)jb.chunk << kChunkBits, mine = base + threadIdx.x;
    const DTerm *T = terms + c.term_begin;
    const double *d = dy + c.out_begin;
    __shared__ DTerm s_t[kWordGroup];
    load_chunk<R>(tile, psi, base, namp);
#pragma unroll
    for (int r = 0; r < 16; ++r) hat[r][threadIdx.x] = 0.0;
    bool flips = false;
    for (uint32_t g0 = 0; g0 < c.nterms; g0 += kWordGroup) {
        const uint32_t n = stage_words(s_t, T + g0, min(c.nterms - g0, (uint32_t)kWordGroup), d);
        for (uint32_t t = 0; t < n; ++t) {
            const DTerm &tm = s_t[t];
            if (tm.xmask != 0) flips = true;
            else if (tm.coeff != 0.0)
                hat[(tm.zmask >> 8) & 15u][threadIdx.x] +=
                    signed_by(tm.coeff, (uint32_t)__popcll(mine & (tm.zmask & ~uint64_t(0xf00))) & 1u);
        }
    }
    double br[16], bi[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) br[r] = hat[r][threadIdx.x];
    wht16(br);
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        // no factor, no contribution: an unused output leaves the bra at zero whatever psi holds
        const double2 p = widen<R>(tile[threadIdx.x + (r << 8)]);
        const double x = br[r];
        br[r] = x != 0.0 ? x * p.x : 0.0;
        bi[r] = x != 0.0 ? x * p.y : 0.0;
    }
    for (uint32_t g0 = 0; flips && g0 < c.nterms; g0 += kWordGroup) {
        const uint32_t n = c.nterms <= kWordGroup ? c.nterms  // still staged
                                                  : stage_words(s_t, T + g0, min(c.nterms - g0, (uint32_t)kWordGroup), d);
        for (uint32_t t = 0; t < n; ++t) {
            const DTerm &tm = s_t[t];
            const double w = tm.coeff;
            if (w == 0.0 || tm.xmask == 0) continue;
            // i^ny (-1)^{|i&Z|} psi_i of the partner i = j ^ X: the sign is that of j times the one of X & Z
            const uint32_t neg = (uint32_t)__popcll((mine ^ tm.xmask) & (tm.zmask & ~uint64_t(0xf00))) & 1u;
            const uint32_t rows = row_signs(tm.zmask) ^ (__popcll(tm.xmask & tm.zmask & 0xf00u) & 1 ? 0xffffu : 0u);
            const uint32_t xl = (uint32_t)tm.xmask & ((1u << kChunkBits) - 1);
            const bool inside = (tm.xmask >> kChunkBits) == 0, odd = tm.ny & 1;
            const C<R> *other = psi + ((base ^ tm.xmask) & ~uint64_t((1 << kChunkBits) - 1));
            const double f = signed_by(w, neg ^ ((uint32_t)(tm.ny >> 1) & 1u));
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const uint32_t j = threadIdx.x + ((uint32_t)r << 8), o = j ^ xl;
                if (j >= namp) continue;
                const double2 q = widen<R>(inside ? tile[o] : other[o]);
                const double g = signed_by(f, (rows >> r) & 1u);
                if (odd) {  // i psi
                    br[r] -= g * q.y;
                    bi[r] += g * q.x;
                } else {
                    br[r] += g * q.x;
                    bi[r] += g * q.y;
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const uint32_t j = threadIdx.x + ((uint32_t)r << 8);
        if (j < namp) bra[base + j] = mk<R>((R)br[r], (R)bi[r]);
    }
}

// The device program of a batch: plans shared by circuits of one structure, per-circuit tables,
// and one list of jobs per launch.
struct Launch {
    uint32_t first, njobs, threads, smem, level;
};
// Reverse levels from `level` on; reduce: the gradients' partial sums are reduced first, their place is needed.
struct Span {
    uint32_t level;
    bool reduce;
};
// Circuits whose states are in the pools together.
struct Wave {
    std::vector<Launch> launches[2];  // forward, reverse: level by level
    std::vector<Span> spans;
    uint32_t chunk0 = 0, nchunks = 0;
    bool kept = true;                 // no other wave takes its places
};
constexpr uint64_t kNarrowPool = uint64_t(256) << 20;
constexpr uint64_t kMaxGradSums = uint64_t(32) << 20;  // 256 MiB
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
    uint32_t max_steps[2] = {};
    std::vector<Wave> waves;
};

}  // namespace tiles
