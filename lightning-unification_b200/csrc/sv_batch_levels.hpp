// sv_batch_levels.hpp — host planner and launches of the level-by-level batch engine
// (sv_batch_tiles.cuh).  Part of sv_batch.cu (included there once).

namespace tiles {

constexpr int kMaxTileBits = std::max(TGeo<float, false>::kt, TGeo<double, false>::kt);

// Gates of the level engine: everything but two-wire dense gates, double excitations and matrices on
// two and more wires.
bool serves(const HostOp &h) {
    switch (h.form) {
    case F_NOOP: case F_PARITY: case F_SWAP: case F_MAT1: return true;
    case F_DIAG: return h.bits.size() <= 3;
    default: return false;
    }
}

// A one-wire gate with a real matrix.
bool is_real(const HostOp &h) {
    if (h.form != F_MAT1 || h.bits.size() != 1) return false;
    if (h.gate != kConstGate) return h.gate == B200SV_RY;
    return std::all_of(h.cmat.begin(), h.cmat.end(), [](cd z) { return z.imag() == 0; });
}

std::vector<Step> make_steps(const std::vector<HostOp> &ops, uint32_t n) {
    std::vector<Step> out;
    std::vector<int> last(n, -1);  // latest step on each bit
    for (uint32_t i = 0; i < ops.size(); ++i) {
        const HostOp &h = ops[i];
        if (h.form == F_NOOP) continue;
        if (h.bits.size() == 1 && h.form != F_PARITY) {
            const uint32_t b = h.bits[0];
            if (last[b] < 0 || (out[last[b]].kind != S_RUN && out[last[b]].kind != S_DIAGRUN)) {
                Step s;
                s.kind = S_DIAGRUN;
                s.tgt = {b};
                s.mask = uint64_t(1) << b;
                last[b] = (int)out.size();
                out.push_back(std::move(s));
            }
            Step &s = out[last[b]];
            s.mems.push_back(i);
            if (h.form != F_DIAG) {
                s.kind = S_RUN;
                s.flip = s.mask;
            }
            s.grad = s.grad || h.diff;
            continue;
        }
        Step s;
        s.mems = {i};
        s.grad = h.diff;
        const size_t nc = h.form == F_PARITY ? 0 : h.form == F_DIAG && h.nt == 0 ? h.bits.size() : h.bits.size() - h.nt;
        s.ctl.assign(h.bits.begin(), h.bits.begin() + nc);
        s.tgt.assign(h.bits.begin() + nc, h.bits.end());
        for (auto b : h.bits) s.mask |= uint64_t(1) << b;
        if (h.form == F_PARITY) {
            s.kind = S_PARITY;
        } else if (h.form == F_SWAP) {
            s.swap = true;
            for (auto b : s.tgt) s.flip |= uint64_t(1) << b;
            s.linear = s.ctl.size() + s.tgt.size() == 2;
            if (!s.linear) s.targets = s.flip;
        } else if (h.form == F_MAT1) {
            s.kind = S_DENSE;
            s.targets = s.flip = uint64_t(1) << s.tgt[0];
        } else {
            s.kind = S_DIAG;
            const bool cst = h.gate == kConstGate, all = h.nt == 0 && cst && h.cmat[0] == cd(-1, 0),
                       one = h.nt == 1 && cst && h.cmat[0] == cd(1, 0) && h.cmat[1] == cd(-1, 0);
            if (h.bits.size() == 2 && (all || one)) {  // CZ: a sign where both bits are set
                s.kind = S_NONE;
                s.sign = true;
            }
            if (h.diff) {
                // generator over (targets, controls) as the table's index: Z, |11><11| or ZZ
                auto put = [&](int idx, int sg) { s.dsign |= (uint32_t)(sg > 0 ? 1 : 2) << (2 * idx); };
                if (h.gate == B200SV_CRZ) { put(1, 1); put(3, -1); }
                else if (h.gate == B200SV_ControlledPhaseShift) put(3, 1);
                else if (h.gate == B200SV_IsingZZ) { put(0, 1); put(1, -1); put(2, -1); put(3, 1); }
                else throw Unsupported("batch: diagonal generator not supported");
            }
        }
        for (auto b : h.bits) last[b] = (int)out.size();
        out.push_back(std::move(s));
    }
    for (Step &s : out)
        if (s.kind == S_RUN) {
            s.targets = s.mask;
            if (s.mems.size() == 2) {
                const HostOp &a = ops[s.mems[0]], &b = ops[s.mems[1]];
                if (is_real(a) && b.form == F_DIAG) s.split = 1;
                else if (a.form == F_DIAG && is_real(b)) s.split = 2;
            }
        }
    return out;
}

struct PlanDir {
    std::vector<uint32_t> segs;                      // global segment indices, in launch order
    std::vector<std::vector<uint32_t>> grad_steps;   // per segment: step index of each gradient row
    uint32_t step_begin = 0, step_count = 0, ncoef = 0;
};
struct Plan {
    std::vector<Step> steps;
    PlanDir dir[2];
};

struct Builder {
    Records rec;
    std::vector<CoefStep> steps;
    std::vector<uint32_t> mem_list;
};

// Segments and phases of one direction.
template <typename R, bool REV> void plan_dir(Builder &B, Plan &P, uint32_t n, int kt_cap) {
    PlanDir &D = P.dir[REV ? 1 : 0];
    std::vector<uint32_t> order(P.steps.size());
    std::iota(order.begin(), order.end(), 0u);
    if (REV) {  // steps past the last differentiated one are not needed
        std::reverse(order.begin(), order.end());
        while (!order.empty() && !P.steps[order.back()].grad) order.pop_back();
    }
    D.step_begin = (uint32_t)B.steps.size();
    B.rec.ncoef = 0;
    auto coef = [&](uint32_t si, SKind kind, TOp &o, const uint8_t *src, const int *, uint32_t at) {
        const Step &s = P.steps[si];
        if (kind == S_SPLIT) o.pad = (s.split == 2) != REV;
        CoefStep c{};
        c.kind = kind;
        c.mem_begin = (uint32_t)B.mem_list.size();
        c.nmem = (uint32_t)s.mems.size();
        c.coef = at;
        c.nt = (uint8_t)s.tgt.size();
        c.nbits = (uint8_t)(s.tgt.size() + s.ctl.size());
        for (int j = 0; j < 3; ++j) c.src[j] = src[j];
        for (auto m : s.mems) B.mem_list.push_back(m);
        B.steps.push_back(c);
    };
    for (const Piece &p : plan_segments<R, REV>(P.steps, order, n, kt_cap, !REV, sizeof(R) == 4, kMaxTCoefs, B.rec, coef)) {
        D.segs.push_back((uint32_t)p.seg);
        D.grad_steps.push_back(p.grads);
    }
    D.ncoef = B.rec.ncoef + (B.rec.ncoef & 1);
    D.step_count = (uint32_t)B.steps.size() - D.step_begin;
}

// Circuits with equal keys share a plan: the same gates on the same bits (angles, parameter slots and
// constant values differ).
std::string structure_key(const std::vector<HostOp> &ops, uint32_t n) {
    std::string k;
    auto put = [&](uint32_t x) { k.append(reinterpret_cast<const char *>(&x), sizeof x); };
    put(n);
    for (const HostOp &h : ops) {
        const bool sign = h.form == F_DIAG && h.gate == kConstGate && h.bits.size() == 2 &&
                          ((h.nt == 0 && h.cmat[0] == cd(-1, 0)) ||
                           (h.nt == 1 && h.cmat[0] == cd(1, 0) && h.cmat[1] == cd(-1, 0)));
        put((uint32_t)h.form | (uint32_t)h.nt << 8 | (h.diff ? 1u << 16 : 0u) | (sign ? 1u << 17 : 0u) |
            (is_real(h) ? 1u << 18 : 0u));
        put(h.diff ? h.gate : 0u);
        put((uint32_t)h.bits.size());
        for (auto b : h.bits) put(b);
    }
    return k;
}

// Partial sums of the gradients given out so far: of one group, reduced together (k_tile_grads).
struct GradSums {
    uint64_t used = 0, most = 0;
    uint32_t group = 0;
};
// Launches of one direction over the circuits `members` (a wave).
template <typename R, bool REV>
void make_launches(Batch &B, Wave &W, const std::vector<uint32_t> &members, const Builder &bd,
                   const std::vector<Plan> &plans, const std::vector<uint32_t> &plan_of, std::vector<Job> &jobs,
                   std::vector<GradRef> &refs, const std::vector<std::vector<int64_t>> &gslots, GradSums &sums) {
    using G = TGeo<R, REV>;
    constexpr int dir = REV ? 1 : 0;
    size_t levels = 0;
    for (uint32_t c : members) levels = std::max(levels, plans[plan_of[c]].dir[dir].segs.size());
    for (size_t l = 0; l < levels; ++l) {
        // tiles a job takes: eight jobs for every CTA the GPU holds, so that the last ones to finish
        // leave few SMs idle, and no more, since a job stages its segment's records once
        uint64_t tiles = 0;
        for (uint32_t c : members) {
            const PlanDir &D = plans[plan_of[c]].dir[dir];
            if (l < D.segs.size()) tiles += uint64_t(1) << std::max(0, (int)B.nq[c] - (int)bd.rec.segs[D.segs[l]].kt);
        }
        uint64_t per = 1;
        while (per * 2 * 8 * (uint64_t)(sm_count() * G::minb) <= tiles) per *= 2;
        auto parts = [&](uint32_t c, const TSeg &s) {
            return ((uint64_t(1) << std::max(0, (int)B.nq[c] - (int)s.kt)) + per - 1) / per;
        };
        if (REV) {
            uint64_t need = 0;
            for (uint32_t c : members) {
                const PlanDir &D = plans[plan_of[c]].dir[dir];
                if (l >= D.segs.size()) continue;
                const TSeg &s = bd.rec.segs[D.segs[l]];
                need += (uint64_t)s.ngrad * 4 * parts(c, s);
            }
            const bool full = sums.used > 0 && sums.used + need > kMaxGradSums;
            if (full) {
                sums.used = 0;
                ++sums.group;
            }
            if (l == 0 || full) W.spans.push_back(Span{(uint32_t)l, full});
            sums.most = std::max(sums.most, sums.used + need);
        }
        struct Ref {
            Job j;
            uint32_t threads;
            size_t smem;
            uint64_t cost;
        };
        std::vector<Ref> list;
        for (uint32_t c : members) {
            const PlanDir &D = plans[plan_of[c]].dir[dir];
            if (l >= D.segs.size()) continue;
            const TSeg &s = bd.rec.segs[D.segs[l]];
            const uint64_t nt = uint64_t(1) << std::max(0, (int)B.nq[c] - (int)s.kt);
            const uint64_t nparts = parts(c, s);
            for (uint64_t p = 0; p < nparts; ++p) {
                Ref r{};
                r.j.seg = D.segs[l];
                r.j.circ = c;
                r.j.tile0 = (uint32_t)(p * per);
                r.j.ntiles = (uint32_t)std::min<uint64_t>(per, nt - p * per);
                r.j.nparts = (uint32_t)nparts;
                r.j.part = (uint32_t)p;
                r.j.flags = (!REV && l == 0 ? 1u : 0u) | (REV && l + 1 == D.segs.size() ? 2u : 0u);
                r.j.gpart = sums.used;
                r.threads = 1u << (s.kt - G::a);
                r.smem = seg_smem<R, REV>(s);
                r.cost = (uint64_t)r.j.ntiles * (s.nops + 2 * s.nph + 1);
                list.push_back(r);
            }
            if (REV) {
                const auto &rows = D.grad_steps[l];
                for (size_t k = 0; k < rows.size(); ++k)
                    for (uint32_t m : plans[plan_of[c]].steps[rows[k]].mems)
                        if (gslots[c][m] >= 0)
                            refs[gslots[c][m]] = GradRef{sums.used + (uint64_t)k * 4 * nparts, (uint32_t)nparts, sums.group};
                sums.used += (uint64_t)s.ngrad * 4 * nparts;
            }
        }
        std::stable_sort(list.begin(), list.end(), [](const Ref &a, const Ref &b) {
            return a.threads != b.threads ? a.threads > b.threads : a.cost > b.cost;
        });
        for (size_t i = 0; i < list.size();) {
            Launch L{(uint32_t)jobs.size(), 0, list[i].threads, 0, (uint32_t)l};
            const uint32_t th = list[i].threads;
            for (; i < list.size() && list[i].threads == th; ++i) {
                jobs.push_back(list[i].j);
                L.smem = std::max(L.smem, (uint32_t)list[i].smem);
                ++L.njobs;
            }
            W.launches[dir].push_back(L);
        }
    }
}

template <typename R> void build(Batch &B, Planned &P) {
    B.tp = std::make_unique<Program>();
    Program &T = *B.tp;
    Builder bd;
    std::vector<Plan> plans;
    std::vector<uint32_t> plan_of(B.ncirc);
    std::map<std::string, uint32_t> known;
    std::vector<TCirc> circs(B.ncirc);
    std::vector<Mem> mems;
    std::vector<uint64_t> mem_base(B.ncirc);
    std::vector<std::vector<int64_t>> gslots(B.ncirc);
    std::vector<uint32_t> sbegin[2], scount[2];
    uint64_t ncoef[2] = {0, 0};
    uint32_t out_begin = 0;
    const int kt_old = B.dtype == B200SV_C64 ? 13 : 12;  // the widest gate a batch takes
    // Places of the states.  k_batch holds states up to kt_old wires in shared memory, so a batch of any number
    // of narrow circuits fits; here they share kNarrowPool bytes and take turns in waves where they need
    // more (100 000 circuits of 12 qubits complex64 would take 3.3 GB in each pool).  Wider states, which
    // k_batch keeps in memory too, have places of their own.
    auto narrow = [&](uint32_t c) { return (int)B.nq[c] <= kt_old; };
    auto place = [&](uint32_t c) { return std::max<uint64_t>(2, uint64_t(1) << B.nq[c]); };  // 16-byte aligned
    constexpr uint64_t kShare = kNarrowPool / sizeof(C<R>);
    uint64_t wide = 0, narrows = 0, pool = 0;
    for (uint32_t c = 0; c < B.ncirc; ++c) (narrow(c) ? narrows : wide) += place(c);
    std::vector<std::vector<uint32_t>> members(1);  // circuits of each wave
    std::vector<uint64_t> off(B.ncirc);
    for (bool turn : {false, true}) {  // the wide states, then the narrow ones
        uint64_t at = turn ? wide : 0;
        for (uint32_t c = 0; c < B.ncirc; ++c) {
            if (narrow(c) != turn) continue;
            if (turn && narrows > kShare && (at == wide || at + place(c) > wide + kShare)) {
                if (!members.back().empty()) members.emplace_back();
                at = wide;
            }
            off[c] = at;
            at += place(c);
            pool = std::max(pool, at);
            members.back().push_back(c);
        }
    }
    for (uint32_t c = 0; c < B.ncirc; ++c) {
        const auto &ops = B.hops[c];
        const uint32_t n = B.nq[c];
        for (const HostOp &h : ops)
            if ((int)h.bits.size() > kt_old) throw Unsupported("batch: gate wider than the tile");
        const std::string key = structure_key(ops, n);
        auto it = known.find(key);
        if (it == known.end()) {
            Plan p;
            p.steps = make_steps(ops, n);
            plan_dir<R, false>(bd, p, n, B.cfg.kt);
            plan_dir<R, true>(bd, p, n, B.cfg.kt);
            it = known.emplace(key, (uint32_t)plans.size()).first;
            plans.push_back(std::move(p));
        }
        plan_of[c] = it->second;
        TCirc &tc = circs[c];
        tc.n = n;
        tc.off = off[c];
        tc.term_begin = (uint32_t)P.terms.size();
        for (auto t : B.hterms[c]) P.terms.push_back(t);
        tc.nterms = (uint32_t)B.hterms[c].size();
        tc.nobs = B.nobs[c];
        tc.out_begin = out_begin;
        DCirc dc{};
        dc.n = n;
        dc.nobs = tc.nobs;
        dc.out_begin = out_begin;
        P.circs.push_back(dc);
        out_begin += B.nobs[c];
        for (int d = 0; d < 2; ++d) {
            tc.coef[d] = ncoef[d];
            ncoef[d] += plans[plan_of[c]].dir[d].ncoef;
            sbegin[d].push_back(plans[plan_of[c]].dir[d].step_begin);
            scount[d].push_back(plans[plan_of[c]].dir[d].step_count);
            T.max_steps[d] = std::max(T.max_steps[d], scount[d].back());
        }
        mem_base[c] = mems.size();
        gslots[c].assign(ops.size(), -1);
        for (size_t i = 0; i < ops.size(); ++i) {
            const HostOp &h = ops[i];
            Mem m{};
            m.form = (uint8_t)h.form;
            m.gate = (uint8_t)h.gate;
            m.inv = h.inv ? 1 : 0;
            m.nt = (uint8_t)h.nt;
            m.pslot = (int32_t)(h.gate == kConstGate ? -1 : h.pslot);
            m.gslot = -1;
            if (h.gate == kConstGate && h.form != F_SWAP && h.form != F_NOOP) m.cidx = push_const(P, h.cmat);
            if (h.diff && h.gen >= 0) {
                double sc = 0.0;
                std::vector<uint32_t> w(h.bits.size());
                for (size_t q = 0; q < w.size(); ++q) w[q] = (uint32_t)q;
                compile_generator((uint32_t)h.gen, w.data(), (uint32_t)w.size(), 32, &sc);
                gslots[c][i] = m.gslot = (int32_t)P.gscale.size();
                P.gscale.push_back(-2.0 * sc * (h.inv ? -1.0 : 1.0));
                P.gslot_circ.push_back(c);
                P.gslot_param.push_back(h.pslot);
            }
            mems.push_back(m);
        }
    }
    std::vector<uint32_t> col(B.ncirc, 0);
    for (auto c : P.gslot_circ) P.gslot_col.push_back(col[c]++);
    P.pool_a = pool;
    P.pool_b = P.gscale.empty() ? 0 : pool;  // bras
    // jobs of every launch, and the chunks of the measurement kernels, wave by wave
    std::vector<Job> jobs;
    std::vector<GradRef> refs(P.gscale.size());
    std::vector<ChunkJob> chunks;
    std::vector<ObsRef> orefs;
    GradSums sums;
    uint64_t opart = 0;
    for (const auto &list : members) {
        Wave W;
        W.kept = members.size() == 1 || !narrow(list[0]);
        make_launches<R, false>(B, W, list, bd, plans, plan_of, jobs, refs, gslots, sums);
        make_launches<R, true>(B, W, list, bd, plans, plan_of, jobs, refs, gslots, sums);
        W.chunk0 = (uint32_t)chunks.size();
        for (uint32_t c : list) {
            const uint32_t nch = B.nq[c] > (uint32_t)kChunkBits ? 1u << (B.nq[c] - kChunkBits) : 1u;
            for (uint32_t k = 0; k < nch; ++k) chunks.push_back(ChunkJob{c, k, nch, 0, opart});
            for (uint32_t o = 0; o < B.nobs[c]; ++o) orefs.push_back(ObsRef{opart, c, o, nch, 0});
            opart += (uint64_t)circs[c].nterms * nch;
        }
        W.nchunks = (uint32_t)chunks.size() - W.chunk0;
        T.waves.push_back(std::move(W));
    }
    upload(B, T.circs, circs);
    upload(B, T.segs, bd.rec.segs);
    upload(B, T.phases, bd.rec.phases);
    upload(B, T.ops, bd.rec.ops);
    upload(B, T.jobs, jobs);
    upload(B, T.mems, mems);
    upload(B, T.mem_base, mem_base);
    upload(B, T.steps, bd.steps);
    upload(B, T.mem_list, bd.mem_list);
    for (int d = 0; d < 2; ++d) {
        upload(B, T.step_begin[d], sbegin[d]);
        upload(B, T.step_count[d], scount[d]);
        T.coefs[d] = B.dalloc<C<R>>(ncoef[d]);
    }
    upload(B, T.grefs, refs);
    upload(B, T.chunks, chunks);
    upload(B, T.orefs, orefs);
    T.h = B.dalloc<double4>(P.gscale.size());
    T.gpart = B.dalloc<double>(sums.most);
    T.opart = B.dalloc<double>(opart);
    for (const void *m : {(const void *)k_tile_expval<R>, (const void *)k_tile_bra<R>})
        B200SV_CUDA(cudaFuncSetAttribute(m, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chunk_smem<R>()));
    B200SV_CUDA(cudaFuncSetAttribute(k_tiles<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)max_seg_smem<R, false>(kMaxTCoefs)));
    B200SV_CUDA(cudaFuncSetAttribute(k_tiles<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)max_seg_smem<R, true>(kMaxTCoefs)));
}

// coefficients of a direction from this launch's trigonometry
template <typename R> void launch_coefs(Batch &B, int dir, cudaStream_t st) {
    Program &T = *B.tp;
    if (!T.max_steps[dir]) return;
    CoefArgs a{};
    a.steps = T.steps;
    a.mem_list = T.mem_list;
    a.step_begin = T.step_begin[dir];
    a.step_count = T.step_count[dir];
    a.mem_base = T.mem_base;
    a.mems = T.mems;
    a.circs = T.circs;
    a.cs = B.d_cs;
    a.consts = B.d_consts;
    a.coefs = T.coefs[dir];
    a.h = T.h;
    a.ncirc = B.ncirc;
    a.rev = dir;
    k_tile_coefs<R><<<dim3((T.max_steps[dir] + 63) / 64, std::min(B.ncirc, 65535u)), 64, 0, st>>>(a);
    B200SV_CUDA(cudaGetLastError());
    B.launched++;
}

// Levels [l0, l1) of a direction: circuits of full tiles in order on the caller's stream, the narrower
// classes (one level each, as a rule) beside them on the batch's side streams.
template <typename R, bool REV>
void launch_levels(Batch &B, const Wave &W, uint32_t l0, uint32_t l1, const int *skip, cudaStream_t st) {
    Program &T = *B.tp;
    TArgs a{};
    a.jobs = T.jobs;
    a.circs = T.circs;
    a.segs = T.segs;
    a.phases = T.phases;
    a.ops = T.ops;
    a.coefs = T.coefs[REV ? 1 : 0];
    a.pool_a = B.d_pool_a;
    a.pool_b = B.d_pool_b;
    a.gpart = T.gpart;
    a.skip = skip;
    const auto &Ls = W.launches[REV ? 1 : 0];
    auto now = [&](const Launch &L) { return L.level >= l0 && L.level < l1; };
    std::vector<uint32_t> classes;
    for (const Launch &L : Ls)
        if (now(L) && std::find(classes.begin(), classes.end(), L.threads) == classes.end())
            classes.push_back(L.threads);
    if (classes.size() > 1) B200SV_CUDA(cudaEventRecord(B.fork, st));
    for (size_t k = 0; k < classes.size(); ++k) {
        const cudaStream_t s = k == 0 ? st : B.side[k - 1];
        if (k > 0) B200SV_CUDA(cudaStreamWaitEvent(s, B.fork, 0));
        for (const Launch &L : Ls) {
            if (!now(L) || L.threads != classes[k]) continue;
            TArgs x = a;
            x.jobs = a.jobs + L.first;
            k_tiles<R, REV><<<L.njobs, L.threads, L.smem, s>>>(x);
            B200SV_CUDA(cudaGetLastError());
            B.launched++;
        }
        if (k > 0) {
            B200SV_CUDA(cudaEventRecord(B.join[k - 1], s));
            B200SV_CUDA(cudaStreamWaitEvent(st, B.join[k - 1], 0));
        }
    }
}

template <typename R> void forward(Batch &B, double *out, cudaStream_t st) {
    Program &T = *B.tp;
    launch_coefs<R>(B, 0, st);
    for (const Wave &W : T.waves) {
        launch_levels<R, false>(B, W, 0, ~0u, nullptr, st);
        if (!B.total_obs) continue;
        k_tile_expval<R><<<W.nchunks, kTThreads, chunk_smem<R>(), st>>>(T.chunks + W.chunk0, T.circs, B.d_terms,
                                                                        B.d_pool_a, T.opart);
        B200SV_CUDA(cudaGetLastError());
        B.launched++;
    }
    if (!B.total_obs) return;
    k_tile_outputs<<<(B.total_obs + 7) / 8, 256, 0, st>>>(T.orefs, B.total_obs, T.circs, B.d_terms, T.opart, out);
    B200SV_CUDA(cudaGetLastError());
    B.launched++;
}

// gradw[g] for the bra of dy, recomputing the states unless *reuse says pool A holds them (the places of a
// wave that takes turns hold another wave's)
template <typename R> void reverse(Batch &B, const double *dy, const int *reuse, cudaStream_t st) {
    Program &T = *B.tp;
    if (!B.ngslots) return;
    uint32_t group = 0;
    auto grads = [&] {
        k_tile_grads<<<std::max(1u, std::min(8192u, (B.ngslots + 15) / 16)), 128, 0, st>>>(T.grefs, T.h, T.gpart, B.ngslots,
                                                                                          group++, B.d_gradw);
        B200SV_CUDA(cudaGetLastError());
        B.launched++;
    };
    launch_coefs<R>(B, 0, st);
    launch_coefs<R>(B, 1, st);
    for (const Wave &W : T.waves) {
        launch_levels<R, false>(B, W, 0, ~0u, W.kept ? reuse : nullptr, st);
        k_tile_bra<R><<<W.nchunks, kTThreads, chunk_smem<R>(), st>>>(T.chunks + W.chunk0, T.circs, B.d_terms,
                                                                     B.d_pool_a, B.d_pool_b, dy);
        B200SV_CUDA(cudaGetLastError());
        B.launched++;
        for (size_t i = 0; i < W.spans.size(); ++i) {
            if (W.spans[i].reduce) grads();
            const uint32_t end = i + 1 < W.spans.size() ? W.spans[i + 1].level : ~0u;
            launch_levels<R, true>(B, W, W.spans[i].level, end, nullptr, st);
        }
    }
    grads();
}

}  // namespace tiles
