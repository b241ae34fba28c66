// sv_batch_levels.hpp — host planner and launches of the level-by-level batch engine
// (sv_batch_tiles.cuh).  Part of sv_batch.cu (included there once).

namespace tiles {

// Gates of the level engine: everything but two-wire dense gates, double excitations and matrices on
// two and more wires.
bool serves(const HostOp &h) {
    switch (h.form) {
    case F_NOOP: case F_PARITY: case F_SWAP: case F_MAT1: return true;
    case F_DIAG: return h.bits.size() <= 3;
    default: return false;
    }
}

// A step of a circuit: a run of single-wire gates on one bit, or one gate.
struct Step {
    SKind kind = S_NONE;
    bool swap = false, sign = false, grad = false, wide = false;
    std::vector<uint32_t> mems;     // op indices, in order
    std::vector<uint32_t> ctl, tgt; // state bits
    uint64_t mask = 0, targets = 0; // bits touched; bits that must be register bits
    uint64_t flip = 0;              // bits on which the step is not diagonal: steps commute when every
                                    // bit they share is diagonal in both
    bool linear = false;            // CNOT, SWAP: between phases, in the tile's address map
    uint32_t dsign = 0;
};

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
            s.wide = true;
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
        if (s.kind == S_RUN) s.targets = s.mask;
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
    std::vector<TSeg> segs;
    std::vector<TPhase> phases;
    std::vector<TOp> ops;
    std::vector<CoefStep> steps;
    std::vector<uint32_t> mem_list;
};

int coef_slots(const Step &s, bool rev) {
    switch (s.kind) {
    case S_RUN: case S_DENSE: return 4;
    case S_DIAGRUN: return rev && s.grad ? 4 : 8;
    case S_DIAG: return 8;
    case S_PARITY: return 2;
    default: return 0;
    }
}

// Segments and phases of one direction.  A diagonal run with a gradient is a 2x2 step of the reverse
// sweep (its sums go over register pairs).
template <typename R, bool REV> void plan_dir(Builder &B, Plan &P, uint32_t n, int kt_cap) {
    using G = TGeo<R, REV>;
    PlanDir &D = P.dir[REV ? 1 : 0];
    const int kt = std::max(std::min({(int)n, (int)G::kt, kt_cap}), G::a + 5);
    const bool tiled = (int)n > kt;
    const uint64_t low = tiled ? (uint64_t(1) << G::reserve) - 1 : 0;
    std::vector<uint32_t> order(P.steps.size());
    std::iota(order.begin(), order.end(), 0u);
    if (REV) std::reverse(order.begin(), order.end());
    const size_t ns = order.size();
    auto step = [&](size_t i) -> const Step & { return P.steps[order[i]]; };
    auto targets = [&](const Step &s) { return REV && s.kind == S_DIAGRUN && s.grad ? s.mask : s.targets; };
    std::vector<char> done(ns, 0);
    size_t left = ns, first = 0;
    if (REV) {  // steps past the last differentiated one are not needed
        size_t lastg = 0;
        for (size_t i = 0; i < ns; ++i)
            if (step(i).grad) lastg = i + 1;
        for (size_t i = lastg; i < ns; ++i) done[i] = 1;
        left = lastg;
    }
    D.step_begin = (uint32_t)B.steps.size();
    while (left > 0 || (!REV && D.segs.empty())) {
        while (first < ns && done[first]) ++first;
        // the segment: every later step that fits the tile and commutes with the steps left out
        uint64_t used = 0, any = 0, flipped = 0;  // of the steps left out
        int nops = 0, ncf = 0, ngr = 0;
        std::vector<uint32_t> take;
        for (size_t j = first; j < ns; ++j) {
            if (done[j]) continue;
            const Step &s = step(j);
            const uint64_t need = s.wide ? 0 : s.mask;
            const bool fits = !(s.flip & any) && !(s.mask & flipped) && __builtin_popcountll(used | need | low) <= kt &&
                              nops < kMaxTOps && ncf + coef_slots(s, REV) <= kMaxTCoefs &&
                              ngr + (REV && s.grad ? 1 : 0) <= kMaxTGrads;
            if (fits) {
                used |= need;
                ++nops;
                ncf += coef_slots(s, REV);
                ngr += REV && s.grad ? 1 : 0;
                take.push_back((uint32_t)j);
                done[j] = 1;
                --left;
            } else {
                any |= s.mask;
                flipped |= s.flip;
                if (flipped == (uint64_t(1) << n) - 1) break;  // everything later is blocked
            }
        }
        if (take.empty() && left > 0) throw Unsupported("batch: gate wider than the tile");
        TSeg sg{};
        std::vector<int> loc(n, -1);
        uint64_t inl = used | low;
        for (uint32_t x = 0; x < n && __builtin_popcountll(inl) < kt; ++x) inl |= uint64_t(1) << x;
        int nl = 0;
        for (uint32_t x = 0; x < n; ++x) {
            if ((inl >> x) & 1) {
                loc[x] = nl;
                sg.lbits[nl++] = (uint8_t)x;
            } else {
                sg.gbits[sg.ng++] = (uint8_t)x;
            }
        }
        for (uint32_t x = n; nl < kt; ++x) sg.lbits[nl++] = (uint8_t)x;  // padding above the state
        sg.kt = (uint8_t)kt;
        sg.ph_begin = (uint32_t)B.phases.size();
        sg.op_begin = (uint32_t)B.ops.size();
        sg.coef_begin = D.ncoef;
        std::vector<uint32_t> grads;
        // phases: the ready CNOTs and SWAPs go into the address map, then every ready step whose
        // targets fit the register bits, until nothing moves
        std::vector<char> out(take.size(), 0);
        size_t rest = take.size();
        uint16_t place[12];  // of each tile bit, before the swizzle
        for (int b = 0; b < 12; ++b) place[b] = (uint16_t)(1u << b);
        while (rest > 0) {
            uint32_t rmask = 0;
            std::vector<uint32_t> cur;
            for (bool linear : {true, false}) {
                for (bool progress = true; progress;) {
                    progress = false;
                    uint64_t la = 0, lf = 0;
                    for (size_t i = 0; i < take.size(); ++i) {
                        if (out[i]) continue;
                        const Step &s = step(take[i]);
                        uint32_t need = 0;
                        for (uint32_t x = 0; x < n; ++x)
                            if ((targets(s) >> x) & 1) need |= 1u << loc[x];
                        if (s.linear == linear && !(s.flip & la) && !(s.mask & lf) &&
                            __builtin_popcount(rmask | need) <= G::a) {
                            out[i] = 1;
                            --rest;
                            progress = true;
                            if (!linear) {
                                rmask |= need;
                                cur.push_back(take[i]);
                            } else if (s.ctl.size() == 1) {
                                place[loc[s.ctl[0]]] ^= place[loc[s.tgt[0]]];
                            } else {
                                std::swap(place[loc[s.tgt[0]]], place[loc[s.tgt[1]]]);
                            }
                        } else {
                            la |= s.mask;
                            lf |= s.flip;
                        }
                    }
                }
            }
            if (cur.empty()) continue;  // the segment ends in CNOTs
            for (int b = kt - 1; b >= 0 && __builtin_popcount(rmask) < G::a; --b) rmask |= 1u << b;
            TPhase ph{};
            ph.op_begin = (uint16_t)(B.ops.size() - sg.op_begin);
            ph.nops = (uint16_t)cur.size();
            std::vector<int> rpos(32, -1);
            std::vector<int> reg;  // register j's tile bit: fewest steps first (Regs)
            for (int b = 0, j = 0; b < kt; ++b)
                if ((rmask >> b) & 1) {
                    reg.push_back(b);
                    ph.rb[j++] = (uint8_t)b;
                }
            auto uses = [&](int b) {
                int c = 0;
                for (uint32_t j : cur) c += (int)((targets(step(j)) >> sg.lbits[b]) & 1);
                return c;
            };
            std::stable_sort(reg.begin(), reg.end(), [&](int x, int y) { return uses(x) < uses(y); });
            for (int j = 0; j < G::a; ++j) {
                rpos[reg[j]] = j;
                ph.rt[j] = (uint8_t)reg[j];
                ph.rcol[j] = (uint16_t)tswz<R>(place[reg[j]]);
            }
            for (int b = 0, j = 0; b < kt; ++b)
                if (!((rmask >> b) & 1)) ph.tcol[j++] = (uint16_t)tswz<R>(place[b]);
            B.phases.push_back(ph);
            for (uint32_t j : cur) {
                const Step &s = step(j);
                TOp o{};
                CoefStep c{};
                c.kind = s.kind;
                if (REV && s.kind == S_DIAGRUN && s.grad) c.kind = S_RUN;
                c.mem_begin = (uint32_t)B.mem_list.size();
                c.nmem = (uint16_t)s.mems.size();
                c.coef = D.ncoef;
                o.coef = (uint16_t)(D.ncoef - sg.coef_begin);
                o.p0 = o.p1 = o.p2 = 31;
                if (REV && s.grad) {
                    grads.push_back(order[j]);
                    o.grad = (uint16_t)grads.size();
                }
                auto control = [&](const std::vector<uint32_t> &bits) {
                    for (auto x : bits) {
                        if (rpos[loc[x]] >= 0) o.creg |= (uint16_t)(1 << rpos[loc[x]]);
                        else o.cthr |= 1u << loc[x];
                    }
                };
                auto pair_index = [](int m) {
                    for (int i = 0; i < 6; ++i)
                        if (pair_mask(i) == m) return i;
                    return 0;
                };
                if (s.sign) {
                    control(s.ctl);
                    control(s.tgt);
                    const int nr = __builtin_popcount(o.creg);
                    o.code = nr == 0 ? T_SIGN_T : nr == 1 ? T_SIGN1 + __builtin_ctz(o.creg) : T_SIGN2 + pair_index(o.creg);
                } else if (s.swap) {
                    control(s.ctl);
                    if (s.tgt.size() == 1) {
                        const int t = rpos[loc[s.tgt[0]]], nr = __builtin_popcount(o.creg);
                        o.code = nr == 0   ? T_CX_T + t
                                 : nr == 1 ? T_CX_R + 4 * t + __builtin_ctz(o.creg)
                                           : T_CX_G + t;
                    } else {
                        o.code = T_SWAP + pair_index((1 << rpos[loc[s.tgt[0]]]) | (1 << rpos[loc[s.tgt[1]]]));
                    }
                } else if (c.kind == S_RUN) {
                    o.code = T_DENSE + rpos[loc[s.tgt[0]]];
                } else if (s.kind == S_DENSE) {
                    control(s.ctl);
                    o.code = T_DENSEC + rpos[loc[s.tgt[0]]];
                } else if (s.kind == S_DIAGRUN) {
                    const int b = loc[s.tgt[0]];
                    if (rpos[b] >= 0) o.code = T_DIAG1 + rpos[b];
                    else o.code = T_DIAG_T;
                    o.p2 = (uint8_t)b;
                } else if (s.kind == S_PARITY) {
                    for (auto x : s.tgt) {
                        if (loc[x] >= 0) o.pm |= 1u << loc[x];
                        else o.pmg |= uint64_t(1) << x;
                    }
                    o.code = (o.pm & rmask) == 0 && !o.grad ? T_PAR_T : T_PAR;
                } else {  // S_DIAG: index over the gate's bits, targets first
                    std::vector<uint32_t> L = s.tgt;
                    L.insert(L.end(), s.ctl.begin(), s.ctl.end());
                    c.nt = (uint8_t)s.tgt.size();
                    c.nbits = (uint8_t)L.size();
                    int reg = -1, nr = 0;
                    for (size_t q = 0; q < L.size(); ++q)
                        if (rpos[loc[L[q]]] >= 0) {
                            reg = (int)q;
                            ++nr;
                        }
                    uint8_t pos[3] = {31, 31, 31};
                    c.src[0] = c.src[1] = c.src[2] = 255;
                    if (nr == 1 && !o.grad) {  // the register bit last
                        int at = 0;
                        for (size_t q = 0; q < L.size(); ++q) {
                            const int j3 = (int)q == reg ? 2 : at++;
                            pos[j3] = (uint8_t)loc[L[q]];
                            c.src[j3] = (uint8_t)q;
                        }
                        o.code = T_DIAG1 + rpos[loc[L[reg]]];
                    } else {
                        uint32_t ds = 0;
                        for (size_t q = 0; q < L.size(); ++q) {
                            pos[q] = (uint8_t)loc[L[q]];
                            c.src[q] = (uint8_t)q;
                        }
                        // the generator's index has the gate's bits lowest; the table's has them highest
                        for (int e = 0; e < 8; ++e)
                            ds |= ((s.dsign >> (2 * (e >> (3 - (int)L.size())))) & 3u) << (2 * e);
                        o.dsign = ds;
                        o.code = nr == 0 && !o.grad ? T_DIAG_T : T_DIAG;
                    }
                    o.p0 = pos[0];
                    o.p1 = pos[1];
                    o.p2 = pos[2];
                }
                for (auto m : s.mems) B.mem_list.push_back(m);
                D.ncoef += (uint32_t)coef_slots(s, REV);
                B.steps.push_back(c);
                B.ops.push_back(o);
            }
        }
        for (int b = 0; b < 12; ++b) sg.fcol[b] = (uint16_t)tswz<R>(place[b]);
        sg.nph = (uint32_t)B.phases.size() - sg.ph_begin;
        sg.nops = (uint32_t)B.ops.size() - sg.op_begin;
        sg.ncoef = D.ncoef - sg.coef_begin;
        sg.ngrad = (uint32_t)grads.size();
        D.segs.push_back((uint32_t)B.segs.size());
        D.grad_steps.push_back(grads);
        B.segs.push_back(sg);
    }
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
        put((uint32_t)h.form | (uint32_t)h.nt << 8 | (h.diff ? 1u << 16 : 0u) | (sign ? 1u << 17 : 0u));
        put(h.diff ? h.gate : 0u);
        put((uint32_t)h.bits.size());
        for (auto b : h.bits) put(b);
    }
    return k;
}

template <typename R, bool REV> size_t seg_smem(const TSeg &s) {
    return (REV ? 2 : 1) * (sizeof(C<R>) << s.kt) + s.nops * sizeof(TOp) + s.ncoef * sizeof(C<R>) +
           s.nph * sizeof(TPhase) + (REV ? (size_t)s.ngrad * 4 * kTWarps * sizeof(double) : 0);
}

template <typename R, bool REV>
void make_launches(Batch &B, Program &T, const Builder &bd, const std::vector<Plan> &plans,
                   const std::vector<uint32_t> &plan_of, std::vector<Job> &jobs, std::vector<GradRef> &refs,
                   const std::vector<std::vector<int64_t>> &gslots, uint64_t &gpart) {
    using G = TGeo<R, REV>;
    constexpr int dir = REV ? 1 : 0;
    size_t levels = 0;
    for (const Plan &p : plans) levels = std::max(levels, p.dir[dir].segs.size());
    for (size_t l = 0; l < levels; ++l) {
        // tiles a job takes: eight jobs for every CTA the GPU holds, so that the last ones to finish
        // leave few SMs idle, and no more, since a job stages its segment's records once
        uint64_t tiles = 0;
        for (uint32_t c = 0; c < B.ncirc; ++c) {
            const PlanDir &D = plans[plan_of[c]].dir[dir];
            if (l < D.segs.size()) tiles += uint64_t(1) << std::max(0, (int)B.nq[c] - (int)bd.segs[D.segs[l]].kt);
        }
        uint64_t per = 1;
        while (per * 2 * 8 * (uint64_t)(sm_count() * G::minb) <= tiles) per *= 2;
        struct Ref {
            Job j;
            uint32_t threads;
            size_t smem;
            uint64_t cost;
        };
        std::vector<Ref> list;
        for (uint32_t c = 0; c < B.ncirc; ++c) {
            const PlanDir &D = plans[plan_of[c]].dir[dir];
            if (l >= D.segs.size()) continue;
            const TSeg &s = bd.segs[D.segs[l]];
            const uint64_t nt = uint64_t(1) << std::max(0, (int)B.nq[c] - (int)s.kt);
            const uint64_t nparts = (nt + per - 1) / per;
            for (uint64_t p = 0; p < nparts; ++p) {
                Ref r{};
                r.j.seg = D.segs[l];
                r.j.circ = c;
                r.j.tile0 = (uint32_t)(p * per);
                r.j.ntiles = (uint32_t)std::min<uint64_t>(per, nt - p * per);
                r.j.nparts = (uint32_t)nparts;
                r.j.part = (uint32_t)p;
                r.j.flags = (!REV && l == 0 ? 1u : 0u) | (REV && l + 1 == D.segs.size() ? 2u : 0u);
                r.j.gpart = gpart;
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
                            refs[gslots[c][m]] = GradRef{gpart + (uint64_t)k * 4 * nparts, (uint32_t)nparts, 0};
                gpart += (uint64_t)s.ngrad * 4 * nparts;
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
            T.launches[dir].push_back(L);
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
    uint64_t pool = 0, ncoef[2] = {0, 0};
    uint32_t out_begin = 0;
    const int kt_old = B.dtype == B200SV_C64 ? 13 : 12;  // the widest gate a batch takes
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
        tc.off = pool;
        pool += std::max<uint64_t>(2, uint64_t(1) << n);  // 16-byte aligned states
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
    P.pool_a = P.pool_b = pool;
    // jobs of every launch
    std::vector<Job> jobs;
    std::vector<GradRef> refs(P.gscale.size());
    uint64_t gpart = 0;
    make_launches<R, false>(B, T, bd, plans, plan_of, jobs, refs, gslots, gpart);
    make_launches<R, true>(B, T, bd, plans, plan_of, jobs, refs, gslots, gpart);
    // chunks of the measurement kernels
    std::vector<ChunkJob> chunks;
    std::vector<ObsRef> orefs;
    uint64_t opart = 0;
    for (uint32_t c = 0; c < B.ncirc; ++c) {
        const uint32_t nch = B.nq[c] > (uint32_t)kChunkBits ? 1u << (B.nq[c] - kChunkBits) : 1u;
        for (uint32_t k = 0; k < nch; ++k) chunks.push_back(ChunkJob{c, k, nch, 0, opart});
        for (uint32_t o = 0; o < B.nobs[c]; ++o) orefs.push_back(ObsRef{opart, c, o, nch, 0});
        opart += (uint64_t)circs[c].nterms * nch;
    }
    T.nchunks = (uint32_t)chunks.size();
    upload(B, T.circs, circs);
    upload(B, T.segs, bd.segs);
    upload(B, T.phases, bd.phases);
    upload(B, T.ops, bd.ops);
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
    T.gpart = B.dalloc<double>(gpart);
    T.opart = B.dalloc<double>(opart);
    uint32_t smem[2] = {0, 0};
    for (int d = 0; d < 2; ++d)
        for (const Launch &L : T.launches[d]) smem[d] = std::max(smem[d], L.smem);
    const void *k[2] = {(const void *)k_tiles<R, false>, (const void *)k_tiles<R, true>};
    for (int d = 0; d < 2; ++d)
        if (smem[d] > 48 * 1024)
            B200SV_CUDA(cudaFuncSetAttribute(k[d], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem[d]));
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

// The levels of a direction: circuits of full tiles in order on the caller's stream, the narrower
// classes (one level each, as a rule) beside them on the batch's side streams.
template <typename R, bool REV> void launch_levels(Batch &B, const int *skip, cudaStream_t st) {
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
    const auto &Ls = T.launches[REV ? 1 : 0];
    if (Ls.empty()) return;
    std::vector<uint32_t> classes;
    for (const Launch &L : Ls)
        if (std::find(classes.begin(), classes.end(), L.threads) == classes.end()) classes.push_back(L.threads);
    if (classes.size() > 1) B200SV_CUDA(cudaEventRecord(B.fork, st));
    for (size_t k = 0; k < classes.size(); ++k) {
        const cudaStream_t s = k == 0 ? st : B.side[k - 1];
        if (k > 0) B200SV_CUDA(cudaStreamWaitEvent(s, B.fork, 0));
        for (const Launch &L : Ls) {
            if (L.threads != classes[k]) continue;
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
    launch_levels<R, false>(B, nullptr, st);
    if (!B.total_obs) return;
    k_tile_expval<R><<<T.nchunks, kTThreads, 0, st>>>(T.chunks, T.circs, B.d_terms, B.d_pool_a, T.opart);
    k_tile_outputs<<<(B.total_obs + 7) / 8, 256, 0, st>>>(T.orefs, B.total_obs, T.circs, B.d_terms, T.opart, out);
    B200SV_CUDA(cudaGetLastError());
    B.launched += 2;
}

// gradw[g] for the bra of dy, recomputing the states unless *reuse says pool A holds them
template <typename R> void reverse(Batch &B, const double *dy, const int *reuse, cudaStream_t st) {
    Program &T = *B.tp;
    launch_coefs<R>(B, 0, st);
    launch_levels<R, false>(B, reuse, st);
    if (!B.ngslots) return;
    launch_coefs<R>(B, 1, st);
    k_tile_bra<R><<<T.nchunks, kTThreads, 0, st>>>(T.chunks, T.circs, B.d_terms, B.d_pool_a, B.d_pool_b, dy);
    launch_levels<R, true>(B, nullptr, st);
    k_tile_grads<<<std::max(1u, std::min(4096u, (B.ngslots + 127) / 128)), 128, 0, st>>>(T.grefs, T.h, T.gpart, B.ngslots,
                                                                                      B.d_gradw);
    B200SV_CUDA(cudaGetLastError());
    B.launched += 2;
}

}  // namespace tiles
