// sv_fused.cu — one pass over a single state for a run of gates.
//
// The per-gate kernels (sv_gates.cu) read and write the whole state once per gate.  Here gates whose
// wires fit in one shared-memory tile form a segment (sv_plan.hpp): a CTA takes tiles, applies the
// segment's gates to them in registers (sv_steps.cuh) and writes them back.  Consecutive gates on one
// wire are one step, CNOTs and SWAPs only change the tile's address map.  The reverse sweep of the
// adjoint method runs the same way over lambda and a bra, with every differentiated step's generator
// products formed from four FP64 sums.
//
// Against the previous kernels (512-thread CTAs, one per SM, tiles double-buffered, CNOTs exchanged in
// registers, complex64 sums compensated in FP32 pairs, products per member in FP64): 200 random gates on
// 26 qubits complex128 21.8 -> 17.9 ms and on 27 qubits complex64 39.0 -> 24.7 ms (error against 64 bits
// 6.2e-7 -> 5.3e-7), the 600-parameter Jacobian of 20 qubits 6.2 -> 4.1 ms a call.
#include <algorithm>
#include <cstring>
#include <functional>
#include <type_traits>
#include <vector>

#include "sv_device.cuh"
#include "sv_internal.hpp"
#include "sv_plan.hpp"
#include "sv_steps.cuh"

namespace b200sv {
namespace {

using namespace steps;

constexpr int kMaxStateCoefs = 1024;
// Partial sums of a sweep's gradients (64 MiB; a step has four per CTA and bra, 38 KB on a wide state): they are
// reduced when the next segment's would not fit, so the workspace does not grow with the parameters.
constexpr uint64_t kMaxGradSums = uint64_t(8) << 20;

struct StateArgs {
    const TSeg *seg;
    const TPhase *phases;
    const TOp *ops;
    const void *coefs;
    double *gpart;  // REV: partial sums [bra][row][4][CTA]
    uint64_t ntiles, namp;
};

// One segment over the tiles of one state, or (REV) of lambda and the bra of blockIdx.y: every bra's
// CTAs take lambda's tiles through the segment again beside their own bra's, reading lam_in; those of
// blockIdx.y 0 write lam_out (a second buffer where one launch takes several bras) unless it is null.
template <typename R, bool REV>
__global__ void __launch_bounds__(kTThreads, 2) k_state(const C<R> *lam_in, C<R> *lam_out, C<R> *const *__restrict__ bras,
                                                        StateArgs a) {
    using G = TGeo<R, REV>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TSeg sg;
    if (threadIdx.x < sizeof(TSeg) / 8)
        reinterpret_cast<uint64_t *>(&sg)[threadIdx.x] = reinterpret_cast<const uint64_t *>(a.seg)[threadIdx.x];
    __syncthreads();
    const uint32_t NT = blockDim.x, TN = NT * G::A;
    C<R> *const sl = reinterpret_cast<C<R> *>(smem_raw);
    C<R> *const sb = sl + TN;
    TOp *const sop = reinterpret_cast<TOp *>(smem_raw + tile_buffers<R, REV>() * sizeof(C<R>) * TN);
    C<R> *const scf = reinterpret_cast<C<R> *>(sop + sg.nops);
    TPhase *const sph = reinterpret_cast<TPhase *>(scf + sg.ncoef);
    double *const sacc = reinterpret_cast<double *>(sph + sg.nph);
    copy_words(sop, a.ops + sg.op_begin, sg.nops);
    copy_words(scf, static_cast<const C<R> *>(a.coefs) + sg.coef_begin, sg.ncoef);
    copy_words(sph, a.phases + sg.ph_begin, sg.nph);
    if (REV)
        for (uint32_t i = threadIdx.x; i < sg.ngrad * 4 * kTWarps; i += NT) sacc[i] = 0.0;
    run_tiles<R, REV, true>(sg, sl, sb, sop, scf, sph, sacc, blockIdx.x, a.ntiles, gridDim.x, false, true, lam_in,
                            !REV || blockIdx.y == 0 ? lam_out : nullptr, REV ? bras[blockIdx.y] : nullptr, a.namp);
    if (REV) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < sg.ngrad * 4; i += NT) {
            double s = 0.0;
            for (uint32_t k = 0; k < (NT >> 5); ++k) s += sacc[i * kTWarps + k];
            a.gpart[((uint64_t)blockIdx.y * sg.ngrad * 4 + i) * gridDim.x + blockIdx.x] = s;
        }
    }
}

// One differentiated gate: h of its step's sums, -2 scale, its Jacobian column, and where the sums lie.
struct GradItem {
    double4 h;
    double alpha;
    int64_t col;
    uint64_t base, bra_stride;  // first partial of its row for bra 0; distance between bras
};
// jac[col * nobs + bra] = alpha * h . (sums over the nb CTAs); one block per item and bra (bra0 on), fixed order
__global__ void k_state_grads(const GradItem *__restrict__ items, const double *__restrict__ gpart, int nb,
                              unsigned bra0, unsigned nobs, double *__restrict__ jac) {
    __shared__ double sm[4 * 32];
    const GradItem it = items[blockIdx.x];
    const unsigned bra = bra0 + blockIdx.y;
    const double *p = gpart + it.base + it.bra_stride * bra;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < nb; b += blockDim.x)
#pragma unroll
        for (int v = 0; v < 4; ++v) s[v] += p[(size_t)v * nb + b];
    block_reduce<4>(s, sm);
    if (threadIdx.x == 0)
        jac[it.col * nobs + bra] = it.alpha * (it.h.x * s[0] + it.h.y * s[1] + it.h.z * s[2] + it.h.w * s[3]);
}

// apply g to a vector over the state bits pb (small index bit k-1-j <-> state bit pb[j])
void apply_small(const GateDesc &g, const std::vector<uint32_t> &pb, std::vector<cd> &v) {
    const int k = (int)pb.size();
    auto small = [&](uint32_t sb) {
        for (int j = 0; j < k; ++j)
            if (pb[j] == sb) return 1u << (k - 1 - j);
        return 0u;
    };
    uint32_t cm = 0, tall = 0;
    for (auto c : g.cbits) cm |= small(c);
    const int kg = (int)g.tbits.size();
    std::vector<uint32_t> tm(kg);
    for (int j = 0; j < kg; ++j) tall |= (tm[j] = small(g.tbits[j]));
    auto off = [&](uint32_t r) {
        uint32_t o = 0;
        for (int j = 0; j < kg; ++j)
            if ((r >> (kg - 1 - j)) & 1u) o |= tm[j];
        return o;
    };
    const uint32_t D = 1u << kg;
    for (uint32_t base = 0; base < (1u << k); ++base) {
        if ((base & cm) != cm || (base & tall) != 0) continue;
        switch (g.kind) {
        case Kind::Dense: {
            std::vector<cd> u(D), w(D, cd(0, 0));
            for (uint32_t r = 0; r < D; ++r) u[r] = v[base | off(r)];
            for (uint32_t r = 0; r < D; ++r)
                for (uint32_t c = 0; c < D; ++c) w[r] += g.m[r * D + c] * u[c];
            for (uint32_t r = 0; r < D; ++r) v[base | off(r)] = w[r];
            break;
        }
        case Kind::Diag:
            for (uint32_t r = 0; r < D; ++r) v[base | off(r)] *= g.m[r];
            break;
        case Kind::Swap:
            std::swap(v[base | off(g.sa)], v[base | off(g.sb)]);
            break;
        case Kind::Pair: {
            const cd a = v[base | off(g.pa)], b = v[base | off(g.pb)];
            v[base | off(g.pa)] = g.m2[0] * a + g.m2[1] * b;
            v[base | off(g.pb)] = g.m2[2] * a + g.m2[3] * b;
            for (uint32_t r = 0; r < D; ++r)
                if (r != g.pa && r != g.pb) v[base | off(r)] *= g.gamma;
            break;
        }
        default: break;
        }
    }
}

// Tile form of a descriptor; false when it has to run on its own (wide dense matrices and the like).
bool has_tile_form(const GateDesc &g, int a) {
    const size_t bits = g.tbits.size() + g.cbits.size();
    switch (g.kind) {
    case Kind::Noop: case Kind::Parity: return true;
    case Kind::Dense: return g.k >= 1 && g.k <= 3 && g.k <= a && bits <= 8;
    case Kind::Diag: return bits >= 1 && bits <= 3;
    case Kind::Swap: return g.k >= 1 && g.k <= 2 && bits <= 8;
    case Kind::Pair: return g.cbits.empty() && (g.k == 1 || g.k == 2 || (g.k == 4 && a >= 4));
    default: return false;
    }
}
bool one_bit(const GateDesc &g) {
    return g.tbits.size() + g.cbits.size() == 1 &&
           (g.kind == Kind::Dense || g.kind == Kind::Diag || g.kind == Kind::Swap || g.kind == Kind::Pair);
}
// 2x2 matrix of a one-bit descriptor
void one_bit_matrix(const GateDesc &g, cd (&m)[4]) {
    const uint32_t b = g.tbits.empty() ? g.cbits[0] : g.tbits[0];
    for (int col = 0; col < 2; ++col) {
        std::vector<cd> e(2, cd(0, 0));
        e[col] = cd(1, 0);
        apply_small(g, {b}, e);
        m[col] = e[0];
        m[2 + col] = e[1];
    }
}

// Product of a run's gates, rounded once: its rounding is the same on every amplitude and so adds up in the
// values, where the rounding of single amplitudes averages out.  complex128 products are formed in extended
// precision (600-parameter Jacobian of 20 qubits: error 2.1e-15 -> 1.3e-15 against gate by gate in 64 bits).
template <typename R>
void run_product(const std::vector<const GateDesc *> &gs, const std::vector<uint32_t> &mems, cd (&P)[4]) {
    using L = std::conditional_t<sizeof(R) == 8, long double, double>;
    if (mems.size() == 1) return one_bit_matrix(*gs[mems[0]], P);
    L pr[4] = {1, 0, 0, 1}, pi[4] = {0, 0, 0, 0};
    for (uint32_t i : mems) {
        cd m[4];
        one_bit_matrix(*gs[i], m);
        L mr[4], mi[4], nr[4], ni[4];
        for (int e = 0; e < 4; ++e) {
            mr[e] = m[e].real();
            mi[e] = m[e].imag();
        }
        for (int r = 0; r < 4; r += 2)
            for (int c = 0; c < 2; ++c) {
                nr[r + c] = mr[r] * pr[c] - mi[r] * pi[c] + mr[r + 1] * pr[2 + c] - mi[r + 1] * pi[2 + c];
                ni[r + c] = mr[r] * pi[c] + mi[r] * pr[c] + mr[r + 1] * pi[2 + c] + mi[r + 1] * pr[2 + c];
            }
        for (int e = 0; e < 4; ++e) {
            pr[e] = nr[e];
            pi[e] = ni[e];
        }
    }
    for (int e = 0; e < 4; ++e) P[e] = cd((double)pr[e], (double)pi[e]);
}

// Steps of a gate list in order.  `extra(i, step)` completes the step of gate i (gradients) and says
// whether the gate may use a tile form.
template <typename F>
std::vector<Step> make_steps(const std::vector<const GateDesc *> &gs, uint32_t n, int a, F &&extra) {
    std::vector<Step> out;
    std::vector<int> last(n, -1);  // latest step on each bit
    for (uint32_t i = 0; i < gs.size(); ++i) {
        const GateDesc &g = *gs[i];
        if (g.kind == Kind::Noop) continue;
        Step s;
        s.mems = {i};
        for (auto b : g.tbits) s.mask |= uint64_t(1) << b;
        for (auto b : g.cbits) s.mask |= uint64_t(1) << b;
        s.mask |= g.pmask;
        s.ctl = g.cbits;
        s.tgt = g.tbits;
        s.flip = g.kind == Kind::Diag || g.kind == Kind::Parity ? 0 : s.mask;
        bool tile = has_tile_form(g, a);
        if (tile && one_bit(g)) {
            s.kind = g.kind == Kind::Diag ? S_DIAGRUN : S_RUN;
            s.tgt = {g.tbits.empty() ? g.cbits[0] : g.tbits[0]};
            s.ctl.clear();
        } else if (tile) {
            for (auto b : g.cbits) s.flip &= ~(uint64_t(1) << b);
            switch (g.kind) {
            case Kind::Dense:
                s.kind = g.k == 1 ? S_DENSE : S_WIDE;
                break;
            case Kind::Pair:
                if (g.k == 2 && !(g.pa == 1 && g.pb == 2)) tile = false;
                if (g.k == 4 && !(g.pa == 3 && g.pb == 12)) tile = false;
                s.kind = g.k == 2 ? S_PAIR2 : S_PAIR4;
                s.gamma = g.gamma != cd(1, 0);
                break;
            case Kind::Swap: {
                const bool x = g.k == 1 && g.sa + g.sb == 1, sw = g.k == 2 && g.sa + g.sb == 3 && g.sa != 0 && g.sb != 0;
                if (!x && !sw) tile = false;
                s.swap = true;
                s.linear = tile && g.tbits.size() + g.cbits.size() == 2;
                break;
            }
            case Kind::Parity:
                s.kind = S_PARITY;
                for (uint32_t b = 0; b < n; ++b)
                    if ((g.pmask >> b) & 1) s.tgt.push_back(b);
                break;
            default: {  // Diag: a sign where every bit is set?
                bool sign = s.tgt.size() + s.ctl.size() == 2 && g.m.back() == cd(-1, 0);
                for (size_t r = 0; r + 1 < g.m.size(); ++r) sign = sign && g.m[r] == cd(1, 0);
                if (sign) s.sign = true;
                else s.kind = S_DIAG;
            }
            }
            if (!s.linear && s.flip)
                for (auto b : g.tbits) s.targets |= uint64_t(1) << b;
        }
        if (!tile || !extra(i, s)) {
            s.single = true;
            s.linear = false;
            s.flip = s.mask;
        }
        const bool run = !s.single && (s.kind == S_RUN || s.kind == S_DIAGRUN);
        if (run) {
            const int l = last[s.tgt[0]];
            if (l >= 0 && !out[l].single && (out[l].kind == S_RUN || out[l].kind == S_DIAGRUN)) {
                Step &r = out[l];  // nothing touched the bit since: the gate joins the run
                r.mems.push_back(i);
                if (s.kind == S_RUN) r.kind = S_RUN;
                r.flip |= s.flip;
                r.grad = r.grad || s.grad;
                continue;
            }
        }
        for (uint32_t b = 0; b < n; ++b)
            if ((s.mask >> b) & 1) last[b] = (int)out.size();
        out.push_back(std::move(s));
    }
    for (Step &s : out)
        if (!s.single && s.kind == S_RUN) {
            s.targets = s.mask;
            if (s.mems.size() == 2) {
                auto real = [&](int k) {
                    cd m[4];
                    one_bit_matrix(*gs[s.mems[k]], m);
                    return m[0].imag() == 0 && m[1].imag() == 0 && m[2].imag() == 0 && m[3].imag() == 0;
                };
                if (gs[s.mems[1]]->kind == Kind::Diag && real(0)) s.split = 1;
                else if (gs[s.mems[0]]->kind == Kind::Diag && real(1)) s.split = 2;
            }
        }
    return out;
}

// Coefficients of a step's record, in the positions plan_segments gave it.
template <typename R>
void put_coefs(std::vector<C<R>> &out, const std::vector<const GateDesc *> &gs, const Step &s, SKind kind, TOp &o,
               const uint8_t *src, const int *tr, uint32_t at) {
    auto put = [&](uint32_t i, cd z) {
        if (out.size() <= at + i) out.resize(at + i + 1, mk<R>(0, 0));
        out[at + i] = mk<R>((R)z.real(), (R)z.imag());
    };
    const GateDesc &g = *gs[s.mems[0]];
    switch (kind) {
    case S_RUN: case S_DIAGRUN: {
        cd P[4];
        run_product<R>(gs, s.mems, P);
        if (kind == S_RUN) for (uint32_t e = 0; e < 4; ++e) put(e, P[e]);
        else for (uint32_t e = 0; e < 8; ++e) put(e, P[(e & 1) * 3]);
        break;
    }
    case S_SPLIT: {  // the gates are in the order that they run in
        cd r[4], d[4];
        o.pad = s.split == 2;
        one_bit_matrix(*gs[s.mems[s.split - 1]], r);
        one_bit_matrix(*gs[s.mems[2 - s.split]], d);
        put(0, cd(r[0].real(), r[1].real()));
        put(1, cd(r[2].real(), r[3].real()));
        put(2, d[0]);
        put(3, d[3]);
        break;
    }
    case S_DENSE:
        for (uint32_t e = 0; e < 4; ++e) put(e, g.m[e]);
        break;
    case S_DIAG: {
        const int nt = (int)s.tgt.size(), nb = nt + (int)s.ctl.size();
        for (uint32_t e = 0; e < 8; ++e) {
            uint32_t v = 0;
            for (int j = 0; j < 3; ++j)
                if (((e >> (2 - j)) & 1) && src[j] < 3) v |= 1u << src[j];
            int row = 0;
            bool all = true;
            for (int j = 0; j < nb; ++j) {
                if (j < nt) row = row * 2 + (int)((v >> j) & 1);
                else all = all && ((v >> j) & 1);
            }
            put(e, all ? g.m[row] : cd(1, 0));
        }
        break;
    }
    case S_PARITY:
        put(0, g.pphase[0]);
        put(1, g.pphase[1]);
        break;
    case S_WIDE: {
        // index bit i <-> i-th lowest register bit; entries are doubles in both precisions
        const int k = (int)s.tgt.size(), D = 1 << k;
        std::vector<int> rank(k);
        int mask = 0;
        for (int j = 0; j < k; ++j) mask |= 1 << tr[j];
        for (int j = 0; j < k; ++j) rank[j] = __builtin_popcount(mask & ((1 << tr[j]) - 1));
        auto orig = [&](int c) {
            int q = 0;
            for (int j = 0; j < k; ++j)
                if ((c >> rank[j]) & 1) q |= 1 << (k - 1 - j);
            return q;
        };
        constexpr uint32_t W = sizeof(R) == 4 ? 2 : 1;
        put(W * D * D - 1, cd(0, 0));
        double *d = reinterpret_cast<double *>(out.data() + at);
        for (int r = 0; r < D; ++r)
            for (int c = 0; c < D; ++c) {
                const cd z = g.m[orig(r) * D + orig(c)];
                std::memcpy(d + 2 * (r * D + c), &z, sizeof z);
            }
        break;
    }
    case S_PAIR2: {
        // rows 01 (tgt[0] clear, tgt[1] set) and 10; the kernel's first row has the lower register set
        const bool low = tr[1] < tr[0];
        const cd b[4] = {low ? g.m2[0] : g.m2[3], low ? g.m2[1] : g.m2[2], low ? g.m2[2] : g.m2[1], low ? g.m2[3] : g.m2[0]};
        for (uint32_t e = 0; e < 4; ++e) put(e, b[e]);
        put(4, g.gamma);
        break;
    }
    case S_PAIR4:
        for (uint32_t e = 0; e < 4; ++e) put(e, g.m2[e]);
        put(4, g.gamma);
        break;
    default: break;
    }
}

// Device copies of host arrays in one upload (freed in stream order).
struct Blob {
    std::vector<unsigned char> host;
    unsigned char *dev = nullptr;
    cudaStream_t st;
    explicit Blob(cudaStream_t s) : st(s) {}
    ~Blob() {
        if (dev) cudaFreeAsync(dev, st);
    }
    template <typename T> size_t add(const std::vector<T> &v) {
        const size_t at = (host.size() + 15) & ~size_t(15);
        host.resize(at + v.size() * sizeof(T));
        if (!v.empty()) std::memcpy(host.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
    void upload() {
        B200SV_CUDA(cudaMallocAsync((void **)&dev, std::max<size_t>(16, host.size()), st));
        B200SV_CUDA(cudaMemcpyAsync(dev, host.data(), host.size(), cudaMemcpyHostToDevice, st));
    }
    template <typename T> const T *at(size_t off) const { return reinterpret_cast<const T *>(dev + off); }
};

template <typename R, bool REV> void allow_smem() {
    constexpr size_t most = max_seg_smem<R, REV>(kMaxStateCoefs);
    static_assert(most <= 113 * 1024, "two CTAs an SM");
    B200SV_CUDA(cudaFuncSetAttribute(k_state<R, REV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
}
// CTAs of a launch: four per resident slot, so that the last ones leave few SMs idle and each stages the
// segment's records for several tiles
unsigned state_grid(uint64_t ntiles, unsigned bras) {
    return (unsigned)std::min<uint64_t>(ntiles, std::max(1u, 8u * (unsigned)sm_count() / bras));
}

template <typename R>
void run_fused(void *state, uint32_t nq, const std::vector<GateDesc> &descs,
               const std::function<void(const GateDesc &)> &apply_single, cudaStream_t st) {
    using G = TGeo<R, false>;
    std::vector<const GateDesc *> gs;
    for (const GateDesc &g : descs) gs.push_back(&g);
    const std::vector<Step> all = make_steps(gs, nq, G::a, [](uint32_t, Step &) { return true; });
    std::vector<uint32_t> order(all.size());
    for (uint32_t i = 0; i < order.size(); ++i) order[i] = i;
    Records rec;
    std::vector<C<R>> coefs;
    auto coef = [&](uint32_t si, SKind kind, TOp &o, const uint8_t *src, const int *tr, uint32_t at) {
        put_coefs<R>(coefs, gs, all[si], kind, o, src, tr, at);
    };
    const std::vector<Piece> pieces = plan_segments<R, false>(all, order, nq, 64, false, false, kMaxStateCoefs, rec, coef);
    coefs.resize(rec.ncoef + 2, mk<R>(0, 0));
    Blob blob(st);
    const size_t o_seg = blob.add(rec.segs), o_ph = blob.add(rec.phases), o_op = blob.add(rec.ops), o_cf = blob.add(coefs);
    if (!rec.segs.empty()) {
        allow_smem<R, false>();
        blob.upload();
    }
    for (const Piece &p : pieces) {
        if (p.seg < 0) {
            apply_single(descs[all[p.step].mems[0]]);
            continue;
        }
        const TSeg &s = rec.segs[p.seg];
        StateArgs a{};
        a.seg = blob.at<TSeg>(o_seg) + p.seg;
        a.phases = blob.at<TPhase>(o_ph);
        a.ops = blob.at<TOp>(o_op);
        a.coefs = blob.at<C<R>>(o_cf);
        a.namp = uint64_t(1) << nq;
        a.ntiles = (int)nq > (int)s.kt ? a.namp >> s.kt : 1;
        C<R> *psi = static_cast<C<R> *>(state);
        k_state<R, false><<<state_grid(a.ntiles, 1), 1u << (s.kt - G::a), seg_smem<R, false>(s), st>>>(psi, psi, nullptr, a);
        B200SV_CUDA(cudaGetLastError());
    }
}

// h of a 2x2 generator seen through A (the product of the inverses undone before it in its run)
double4 generator_row(const cd (&Gm)[4], const cd (&A)[4]) {
    cd GA[4], H[4];
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) GA[r * 2 + c] = Gm[r * 2] * A[c] + Gm[r * 2 + 1] * A[2 + c];
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) H[r * 2 + c] = std::conj(A[r]) * GA[c] + std::conj(A[2 + r]) * GA[2 + c];
    return make_double4(H[0].real(), H[3].real(), H[1].real(), H[1].imag());
}

// Generators with sums in the tile kernel: any 2x2 on the gate's own bit, a parity, a diagonal of 0 and
// +-1 over the gate's bits, and a controlled 2x2 on the target of a controlled gate.
bool generator_form(const AdjItem &it, Step &s, cd (&m)[4]) {
    const GateDesc &G = it.G, &u = it.adj;
    if (s.kind == S_RUN || s.kind == S_DIAGRUN) {
        if (!one_bit(G) || (G.tbits.empty() ? G.cbits[0] : G.tbits[0]) != s.tgt[0]) return false;
        if (G.kind == Kind::Pair && G.k != 1) return false;
        one_bit_matrix(G, m);
        return true;
    }
    if (s.kind == S_PARITY)
        return G.kind == Kind::Parity && G.pmask == u.pmask && G.pphase[0] == cd(1, 0) && G.pphase[1] == cd(-1, 0);
    if (s.kind == S_DIAG) {
        if (G.kind != Kind::Diag || !G.cbits.empty()) return false;
        std::vector<uint32_t> L = s.tgt;
        L.insert(L.end(), s.ctl.begin(), s.ctl.end());
        if (L.size() != G.tbits.size() || L.size() > 3) return false;
        s.dsign = 0;
        for (uint32_t e = 0; e < (1u << L.size()); ++e) {
            // e has L[0] as its most significant bit
            uint32_t r = 0;
            for (size_t q = 0; q < G.tbits.size(); ++q) {
                const auto it2 = std::find(L.begin(), L.end(), G.tbits[q]);
                if (it2 == L.end()) return false;
                r = r * 2 + ((e >> (L.size() - 1 - (size_t)(it2 - L.begin()))) & 1);
            }
            const cd z = G.m[r];
            if (z == cd(1, 0)) s.dsign |= 1u << (2 * e);
            else if (z == cd(-1, 0)) s.dsign |= 2u << (2 * e);
            else if (z != cd(0, 0)) return false;
        }
        return true;
    }
    if (s.kind == S_DENSE && s.ctl.size() == 1 && G.kind == Kind::Dense && G.k == 2 && G.cbits.empty() &&
        G.tbits[0] == s.ctl[0] && G.tbits[1] == s.tgt[0]) {
        for (int r = 0; r < 4; ++r)
            for (int c = 0; c < 4; ++c)
                if ((r < 2 || c < 2) && G.m[r * 4 + c] != cd(0, 0)) return false;
        m[0] = G.m[10];
        m[1] = G.m[11];
        m[2] = G.m[14];
        m[3] = G.m[15];
        return true;
    }
    return false;
}

template <typename R>
void run_fused_adjoint(void *&lam, void *&lam2, const std::vector<void *> &bras, uint32_t nq,
                       const std::vector<AdjItem> &items, const std::function<void(size_t)> &exec_single, double *d_jac,
                       cudaStream_t st) {
    using G = TGeo<R, true>;
    const unsigned nobs = (unsigned)bras.size();
    std::vector<const GateDesc *> gs;
    for (const AdjItem &it : items) gs.push_back(&it.adj);
    const std::vector<Step> all = make_steps(gs, nq, G::a, [&](uint32_t i, Step &s) {
        if (!items[i].diff) return true;
        cd m[4];
        if (s.sign) return false;  // no sums in a sign step
        if (!generator_form(items[i], s, m)) return false;
        s.grad = true;
        return true;
    });
    std::vector<uint32_t> order(all.size());
    for (uint32_t i = 0; i < order.size(); ++i) order[i] = i;
    Records rec;
    std::vector<C<R>> coefs;
    auto coef = [&](uint32_t si, SKind kind, TOp &o, const uint8_t *src, const int *tr, uint32_t at) {
        put_coefs<R>(coefs, gs, all[si], kind, o, src, tr, at);
    };
    const std::vector<Piece> pieces = plan_segments<R, true>(all, order, nq, 64, false, false, kMaxStateCoefs, rec, coef);
    coefs.resize(rec.ncoef + 2, mk<R>(0, 0));
    const uint64_t namp = uint64_t(1) << nq;
    const int kt = tile_bits_of<R, true>(nq, 64);
    const uint64_t ntiles = (int)nq > kt ? namp >> kt : 1;
    const bool together = nobs > 1 && lam2;  // every bra in one launch, else one launch a bra
    const unsigned grid = state_grid(ntiles, together ? nobs : 1);
    // gradient items: members in sweep order, each seen through the inverses before it in its run
    std::vector<GradItem> grads;
    std::vector<uint64_t> gbase(rec.segs.size(), 0);
    std::vector<size_t> flush(rec.segs.size(), 0);  // items whose sums are formed after the segment
    uint64_t ngpart = 0, most_gpart = 0;
    size_t flushed = 0;
    int last = -1;
    for (const Piece &p : pieces) {
        if (p.seg < 0) continue;
        const uint64_t size = (uint64_t)p.grads.size() * 4 * grid * nobs;
        if (ngpart > 0 && ngpart + size > kMaxGradSums) {
            flush[last] = grads.size() - flushed;
            flushed = grads.size();
            ngpart = 0;
        }
        last = p.seg;
        gbase[p.seg] = ngpart;
        for (size_t row = 0; row < p.grads.size(); ++row) {
            Step s = all[p.grads[row]];
            cd A[4] = {1, 0, 0, 1};
            for (uint32_t i : s.mems) {
                const AdjItem &it = items[i];
                const bool run = s.kind == S_RUN || s.kind == S_DIAGRUN;
                if (it.diff) {
                    GradItem gi{};
                    cd m[4];
                    generator_form(it, s, m);
                    gi.h = s.kind == S_PARITY || s.kind == S_DIAG ? make_double4(1, 0, 0, 0) : generator_row(m, A);
                    gi.alpha = it.alpha;
                    gi.col = it.col;
                    gi.base = ngpart + (uint64_t)row * 4 * grid;
                    gi.bra_stride = (uint64_t)p.grads.size() * 4 * grid;
                    grads.push_back(gi);
                }
                if (run) {
                    cd u[4], N[4];
                    one_bit_matrix(it.adj, u);
                    for (int r = 0; r < 2; ++r)
                        for (int c = 0; c < 2; ++c) N[r * 2 + c] = u[r * 2] * A[c] + u[r * 2 + 1] * A[2 + c];
                    for (int e = 0; e < 4; ++e) A[e] = N[e];
                }
            }
        }
        ngpart += size;
        most_gpart = std::max(most_gpart, ngpart);
    }
    if (last >= 0) flush[last] = grads.size() - flushed;
    double *gpart = nullptr;
    struct Free {
        double *&p;
        cudaStream_t s;
        ~Free() {
            if (p) cudaFreeAsync(p, s);
        }
    } fr{gpart, st};
    Blob blob(st);
    const size_t o_seg = blob.add(rec.segs), o_ph = blob.add(rec.phases), o_op = blob.add(rec.ops),
                 o_cf = blob.add(coefs), o_br = blob.add(bras), o_gr = blob.add(grads);
    if (!rec.segs.empty()) {
        allow_smem<R, true>();
        blob.upload();
        B200SV_CUDA(cudaMallocAsync((void **)&gpart, std::max<uint64_t>(1, most_gpart) * sizeof(double), st));
    }
    size_t done = 0;  // items whose sums are formed
    for (const Piece &p : pieces) {
        if (p.seg < 0) {
            exec_single(all[p.step].mems[0]);
            continue;
        }
        const TSeg &s = rec.segs[p.seg];
        StateArgs a{};
        a.seg = blob.at<TSeg>(o_seg) + p.seg;
        a.phases = blob.at<TPhase>(o_ph);
        a.ops = blob.at<TOp>(o_op);
        a.coefs = blob.at<C<R>>(o_cf);
        a.gpart = gpart + gbase[p.seg];
        a.namp = namp;
        a.ntiles = ntiles;
        const C<R> *in = static_cast<const C<R> *>(lam);
        if (together) {
            k_state<R, true><<<dim3(grid, nobs), 1u << (s.kt - G::a), seg_smem<R, true>(s), st>>>(
                in, static_cast<C<R> *>(lam2), blob.at<C<R> *>(o_br), a);
            std::swap(lam, lam2);
        } else {
            for (unsigned o = 0; o < nobs; ++o) {  // lambda moves on with the last bra, in place
                k_state<R, true><<<grid, 1u << (s.kt - G::a), seg_smem<R, true>(s), st>>>(
                    in, o + 1 == nobs ? static_cast<C<R> *>(lam) : nullptr, blob.at<C<R> *>(o_br) + o, a);
                a.gpart += (uint64_t)s.ngrad * 4 * grid;
            }
        }
        B200SV_CUDA(cudaGetLastError());
        if (const size_t n = flush[p.seg]) {
            for (unsigned o = 0; o < nobs; o += 65535)
                k_state_grads<<<dim3((unsigned)n, std::min(65535u, nobs - o)), 128, 0, st>>>(
                    blob.at<GradItem>(o_gr) + done, gpart, (int)grid, o, nobs, d_jac);
            B200SV_CUDA(cudaGetLastError());
            done += n;
        }
    }
}

}  // namespace

// A state narrower than a tile is fused from four gates on: the records' upload and the launch
// cost about as much as three gate launches.  From one tile up every call is fused.  While the stream is
// being captured every width stays on the per-gate launches, whose coefficients are kernel arguments (or
// kept with the graph, upload_matrix): a replay must not read the records from this call's host memory.
bool fused_worthwhile(int dtype, uint32_t nq, size_t ngates, cudaStream_t st) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (status != cudaStreamCaptureStatusNone) return false;
    return nq >= (uint32_t)(dtype == B200SV_C64 ? TGeo<float, false>::kt : TGeo<double, false>::kt) || ngates >= 4;
}

void apply_fused(void *state, uint32_t nq, int dtype, const std::vector<GateDesc> &descs,
                 const std::function<void(const GateDesc &)> &apply_single, cudaStream_t st) {
    if (dtype == B200SV_C64) run_fused<float>(state, nq, descs, apply_single, st);
    else run_fused<double>(state, nq, descs, apply_single, st);
}

// Several bras share launches, which needs the second lambda, while the state fits the L2 cache: the bras read
// lambda from there.  On wider states a launch per bra is faster and takes no further state (three bras,
// 22 qubits complex128 5.0 against 5.2 ms, 24 qubits 22.4 against 19.5, 26 qubits 134 against 119).
bool fused_adjoint_together(int dtype, uint32_t nq, uint32_t nobs) {
    return nobs > 1 && nobs <= 65535 && ((uint64_t)(dtype == B200SV_C64 ? 8 : 16) << nq) <= (uint64_t(128) << 20);
}

void apply_fused_adjoint(void *&lambda, void *&lambda2, const std::vector<void *> &bras, uint32_t nq, int dtype,
                         const std::vector<AdjItem> &items, const std::function<void(size_t)> &exec_single,
                         double *d_jac, cudaStream_t st) {
    if (dtype == B200SV_C64) run_fused_adjoint<float>(lambda, lambda2, bras, nq, items, exec_single, d_jac, st);
    else run_fused_adjoint<double>(lambda, lambda2, bras, nq, items, exec_single, d_jac, st);
}

}  // namespace b200sv
