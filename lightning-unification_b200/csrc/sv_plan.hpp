// sv_plan.hpp — host side of sv_steps.cuh: cuts a list of steps into tile segments and register phases.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "sv_internal.hpp"
#include "sv_steps.cuh"

namespace b200sv {
namespace steps {

enum SKind : uint8_t {
    S_RUN = 0,      // single-wire gates on one bit: their product, a 2x2
    S_DIAGRUN = 1,  // the same, all diagonal
    S_DENSE = 2,    // controlled 2x2
    S_DIAG = 3,     // diagonal on two or three bits
    S_PARITY = 4,   // phase by the parity of any number of bits
    S_NONE = 5,     // no coefficients: sign, CNOT, swaps
    S_WIDE = 6,     // dense on two or three bits
    S_PAIR2 = 7,    // excitation block on two bits
    S_PAIR4 = 8,    // excitation block on four bits
    S_SPLIT = 9,    // a run of a real 2x2 and a diagonal (complex128): both kept apart
};

constexpr int kLookAhead = 4096;  // steps a segment leaves out before it is closed

// A step of a circuit.  Two steps commute when every bit they share is diagonal in both (flip).
struct Step {
    SKind kind = S_NONE;
    bool swap = false, sign = false, grad = false;
    bool linear = false;             // CNOT, SWAP: between phases, in the tile's address map
    bool single = false;             // has no tile form: runs alone
    bool gamma = false;              // S_PAIR2, S_PAIR4: the other rows take a factor
    uint8_t split = 0;               // S_RUN of two gates, 1: a real 2x2 and then a diagonal, 2: the reverse
    std::vector<uint32_t> mems;      // caller's indices of its gates, in order
    std::vector<uint32_t> ctl, tgt;  // state bits (tgt[0] the matrix index's most significant)
    uint64_t mask = 0;               // bits touched
    uint64_t flip = 0;               // bits on which the step is not diagonal
    uint64_t targets = 0;            // bits that must be register bits
    uint32_t dsign = 0;              // diagonal generator over (targets, controls)
};

struct Records {
    std::vector<TSeg> segs;
    std::vector<TPhase> phases;
    std::vector<TOp> ops;
    uint32_t ncoef = 0;  // coefficients of the current circuit so far
};
struct Piece {
    int seg = -1;                // segment index, or
    uint32_t step = 0;           // a step that runs alone
    std::vector<uint32_t> grads; // steps of the segment's gradient rows
};

// A diagonal run with a gradient is a 2x2 step of the reverse sweep (its sums go over register pairs).
template <typename R, bool REV> SKind effective_kind(const Step &s) {
    if (sizeof(R) == 8 && s.kind == S_RUN && s.split) return S_SPLIT;
    return REV && s.kind == S_DIAGRUN && s.grad ? S_RUN : s.kind;
}
template <typename R, bool REV> int coef_slots(const Step &s) {
    switch (effective_kind<R, REV>(s)) {
    case S_RUN: case S_SPLIT: case S_DENSE: return 4;
    case S_DIAGRUN: case S_DIAG: return 8;
    case S_PARITY: return 2;
    case S_PAIR2: case S_PAIR4: return 5;
    case S_WIDE: return (1 << (2 * (int)s.tgt.size())) * (sizeof(R) == 4 ? 2 : 1) + (sizeof(R) == 4 ? 1 : 0);
    default: return 0;
    }
}
// register bits a step needs: its targets, and the bit of a differentiated diagonal run
template <bool REV> uint64_t register_targets(const Step &s) {
    return REV && s.kind == S_DIAGRUN && s.grad ? s.mask : s.targets;
}
template <typename R, bool REV> int tile_bits_of(uint32_t n, int cap) {
    using G = TGeo<R, REV>;
    return std::max(std::min({(int)n, (int)G::kt, cap}), G::a + 5);
}

// Steps order[0..] in execution order.  Each segment takes, from the first step not yet done, every
// later one that fits the tile and commutes with the steps left out; each phase first puts the ready
// CNOTs and SWAPs into the address map and then takes every ready step whose targets fit the
// register bits.  coef(step index, effective kind, record, index bit sources, register of each target,
// position) is called once per record; `even_empty` keeps one segment for a circuit without steps;
// `exact_single` gives differentiated steps of one gate the controlled form (t_cross).
template <typename R, bool REV, typename F>
std::vector<Piece> plan_segments(const std::vector<Step> &all, const std::vector<uint32_t> &order, uint32_t n, int cap,
                                 bool even_empty, bool exact_single, int max_coefs, Records &B, F &&coef) {
    using G = TGeo<R, REV>;
    const int kt = tile_bits_of<R, REV>(n, cap);
    const bool tiled = (int)n > kt;
    const uint64_t low = tiled ? (uint64_t(1) << G::reserve) - 1 : 0, every = (uint64_t(1) << n) - 1;
    const size_t ns = order.size();
    std::vector<Piece> pieces;
    std::vector<char> done(ns, 0);
    size_t left = ns, first = 0;
    while (left > 0 || (even_empty && pieces.empty())) {
        while (first < ns && done[first]) ++first;
        if (first < ns && all[order[first]].single) {
            Piece p;
            p.step = order[first];
            pieces.push_back(p);
            done[first] = 1;
            --left;
            continue;
        }
        uint64_t used = 0, any = 0, flipped = 0;  // any, flipped: of the steps left out
        int nops = 0, ncf = 0, ngr = 0, skipped = 0;
        std::vector<uint32_t> take;
        for (size_t j = first; j < ns; ++j) {
            if (done[j]) continue;
            const Step &s = all[order[j]];
            const uint64_t need = s.kind == S_PARITY ? 0 : s.mask;
            const int slots = coef_slots<R, REV>(s), rows = REV && s.grad ? 1 : 0;
            if (!s.single && !(s.flip & any) && !(s.mask & flipped) && __builtin_popcountll(used | need | low) <= kt &&
                nops < kMaxTOps && ncf + slots <= max_coefs && ngr + rows <= kMaxTGrads) {
                used |= need;
                ++nops;
                ncf += slots;
                ngr += rows;
                take.push_back((uint32_t)j);
                done[j] = 1;
                --left;
            } else {
                any |= s.mask;
                flipped |= s.flip;
                // everything later is blocked, or far away: where some bits are never touched (or all steps
                // commute) the look-ahead would read the whole list for every segment
                if (flipped == every || ++skipped == kLookAhead) break;
            }
        }
        if (take.empty() && left > 0) throw Unsupported("gate wider than the tile");
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
        if (B.ncoef & 1) ++B.ncoef;
        sg.coef_begin = B.ncoef;
        Piece piece;
        std::vector<char> out(take.size(), 0);
        std::vector<uint32_t> need_of(take.size(), 0);
        for (size_t i = 0; i < take.size(); ++i)
            for (uint64_t t = register_targets<REV>(all[order[take[i]]]); t; t &= t - 1)
                need_of[i] |= 1u << loc[__builtin_ctzll(t)];
        size_t rest = take.size();
        uint16_t place[12];  // of each tile bit, before the swizzle
        for (int b = 0; b < 12; ++b) place[b] = (uint16_t)(1u << b);
        while (rest > 0) {
            uint32_t rmask = 0;
            const Step *fixed = nullptr;  // a four-row block fixes the registers' order
            std::vector<uint32_t> cur;    // positions in take
            for (bool linear : {true, false}) {
                for (bool progress = true; progress;) {
                    progress = false;
                    uint64_t la = 0, lf = 0;
                    for (size_t i = 0; i < take.size(); ++i) {
                        if (out[i]) continue;
                        const Step &s = all[order[take[i]]];
                        const bool order_ok = s.kind != S_PAIR4 || !fixed || fixed->tgt == s.tgt;
                        if (s.linear == linear && !(s.flip & la) && !(s.mask & lf) && order_ok &&
                            __builtin_popcount(rmask | need_of[i]) <= G::a) {
                            out[i] = 1;
                            --rest;
                            progress = true;
                            if (!linear) {
                                rmask |= need_of[i];
                                if (s.kind == S_PAIR4) fixed = &s;
                                cur.push_back((uint32_t)i);
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
            if (cur.empty()) {
                if (rest > 0) throw Unsupported("phase planning made no progress");
                continue;  // the segment ends in CNOTs
            }
            for (int b = kt - 1; b >= 0 && __builtin_popcount(rmask) < G::a; --b) rmask |= 1u << b;
            TPhase ph{};
            ph.op_begin = (uint16_t)(B.ops.size() - sg.op_begin);
            ph.nops = (uint16_t)cur.size();
            int rpos[32];
            std::vector<int> reg;  // register j's tile bit: fewest steps first (Regs)
            std::vector<int> thr;  // thread bit j's tile bit
            for (int b = 0; b < kt; ++b) {
                rpos[b] = -1;
                ((rmask >> b) & 1 ? reg : thr).push_back(b);
            }
            // the thread bits within one wavefront (eight lanes of 16 bytes, sixteen of 8) first, with
            // places whose bank bits are independent: those lanes hit different banks (27-qubit complex64
            // circuit 26.4 -> 25.7 ms, 26-qubit complex128 18.9 -> 17.9 ms, against ascending order)
            {
                constexpr int q = sizeof(R) == 4 ? 4 : 3;
                std::vector<int> front, back;
                uint32_t basis[q] = {0};
                for (int b : thr) {
                    uint32_t v = tswz<R>(place[b]) & ((1u << q) - 1);
                    for (int k = q - 1; k >= 0 && v; --k)
                        if ((v >> k) & 1) {
                            if (!basis[k]) {
                                basis[k] = v;
                                break;
                            }
                            v ^= basis[k];
                        }
                    (v ? front : back).push_back(b);
                }
                thr = front;
                thr.insert(thr.end(), back.begin(), back.end());
            }
            for (size_t t = 0; t < thr.size(); ++t) {
                ph.tval[t] = (uint16_t)(1u << thr[t]);
                ph.tcol[t] = (uint16_t)(tswz<R>(place[thr[t]]) * sizeof(C<R>));
            }
            if (fixed) {
                for (int j = 0; j < G::a; ++j) reg[j] = loc[fixed->tgt[3 - j]];
            } else {
                int uses[32] = {0};
                for (uint32_t i : cur)
                    for (int b = 0; b < kt; ++b) uses[b] += (need_of[i] >> b) & 1;
                std::stable_sort(reg.begin(), reg.end(), [&](int x, int y) { return uses[x] < uses[y]; });
            }
            for (int j = 0; j < G::a; ++j) {
                rpos[reg[j]] = j;
                ph.rt[j] = (uint8_t)reg[j];
                ph.rcol[j] = (uint16_t)(tswz<R>(place[reg[j]]) * sizeof(C<R>));
            }
            const size_t at_phase = B.phases.size();
            B.phases.push_back(ph);
            for (uint32_t i : cur) {
                const uint32_t si = order[take[i]];
                const Step &s = all[si];
                const SKind kind = effective_kind<R, REV>(s);
                TOp o{};
                uint8_t src[3] = {255, 255, 255};
                int tr[4] = {-1, -1, -1, -1};
                for (size_t q = 0; q < s.tgt.size() && q < 4 && kind != S_PARITY; ++q) tr[q] = rpos[loc[s.tgt[q]]];
                if (kind == S_WIDE && (B.ncoef & 1)) ++B.ncoef;  // 16-byte aligned doubles
                o.coef = (uint16_t)(B.ncoef - sg.coef_begin);
                o.p0 = o.p1 = o.p2 = 31;
                if (REV && s.grad) {
                    piece.grads.push_back(si);
                    o.grad = (uint16_t)piece.grads.size();
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
                int rm = 0;
                for (int q = 0; q < 4; ++q)
                    if (tr[q] >= 0) rm |= 1 << tr[q];
                if (s.sign) {
                    control(s.ctl);
                    control(s.tgt);
                    const int nr = __builtin_popcount(o.creg);
                    o.code = nr == 0 ? T_SIGN_T : nr == 1 ? T_SIGN1 + __builtin_ctz(o.creg) : T_SIGN2 + pair_index(o.creg);
                } else if (s.swap) {
                    control(s.ctl);
                    if (s.tgt.size() == 1) {
                        const int nr = __builtin_popcount(o.creg);
                        o.code = nr == 0   ? T_CX_T + tr[0]
                                 : nr == 1 ? T_CX_R + 4 * tr[0] + __builtin_ctz(o.creg)
                                           : T_CX_G + tr[0];
                    } else {
                        o.code = T_SWAP + pair_index(rm);
                    }
                } else if (kind == S_SPLIT) {
                    o.code = T_SPLIT + tr[0];
                } else if (kind == S_RUN) {
                    o.code = (exact_single && o.grad && s.mems.size() == 1 ? T_DENSEC : T_DENSE) + tr[0];
                } else if (kind == S_DENSE) {
                    control(s.ctl);
                    o.code = T_DENSEC + tr[0];
                } else if (kind == S_DIAGRUN) {
                    const int b = loc[s.tgt[0]];
                    o.code = rpos[b] >= 0 ? T_DIAG1 + rpos[b] : (int)T_DIAG_T;
                    o.p2 = (uint8_t)b;
                } else if (kind == S_PARITY) {
                    for (auto x : s.tgt) {
                        if (loc[x] >= 0) o.pm |= 1u << loc[x];
                        else o.pmg |= uint64_t(1) << x;
                    }
                    o.code = (o.pm & rmask) == 0 && !o.grad ? T_PAR_T : T_PAR;
                } else if (kind == S_WIDE) {
                    control(s.ctl);
                    if (s.tgt.size() == 2) {
                        o.code = T_DENSE2 + pair_index(rm);
                    } else {
                        int t = 0;
                        while (t < 3 && trip_mask(t) != rm) ++t;
                        o.code = T_DENSE3 + t;
                    }
                } else if (kind == S_PAIR2) {
                    o.code = T_PAIR2 + pair_index(rm);
                    o.pad = s.gamma ? 1 : 0;
                } else if (kind == S_PAIR4) {
                    o.code = T_PAIR4;
                    o.pad = s.gamma ? 1 : 0;
                } else {  // S_DIAG: index over the gate's bits, targets first
                    std::vector<uint32_t> L = s.tgt;
                    L.insert(L.end(), s.ctl.begin(), s.ctl.end());
                    int reg1 = -1, nr = 0;
                    for (size_t q = 0; q < L.size(); ++q)
                        if (rpos[loc[L[q]]] >= 0) {
                            reg1 = (int)q;
                            ++nr;
                        }
                    uint8_t pos[3] = {31, 31, 31};
                    if (nr == 1 && !o.grad) {  // the register bit last
                        int at = 0;
                        for (size_t q = 0; q < L.size(); ++q) {
                            const int j3 = (int)q == reg1 ? 2 : at++;
                            pos[j3] = (uint8_t)loc[L[q]];
                            src[j3] = (uint8_t)q;
                        }
                        o.code = T_DIAG1 + rpos[loc[L[reg1]]];
                    } else {
                        for (size_t q = 0; q < L.size(); ++q) {
                            pos[q] = (uint8_t)loc[L[q]];
                            src[q] = (uint8_t)q;
                        }
                        // the generator's index has the gate's bits lowest; the table's has them highest
                        for (int e = 0; e < 8; ++e)
                            o.dsign |= ((s.dsign >> (2 * (e >> (3 - (int)L.size())))) & 3u) << (2 * e);
                        o.code = nr == 0 && !o.grad ? T_DIAG_T : T_DIAG;
                    }
                    o.p0 = pos[0];
                    o.p1 = pos[1];
                    o.p2 = pos[2];
                }
                if (o.code == T_SIGN_T) B.phases[at_phase].signs = 1;
                coef(si, kind, o, src, tr, B.ncoef);
                B.ncoef += (uint32_t)(kind == S_WIDE ? coef_slots<R, REV>(s) - (sizeof(R) == 4 ? 1 : 0)
                                                     : coef_slots<R, REV>(s));
                B.ops.push_back(o);
            }
        }
        for (int b = 0; b < 12; ++b) sg.fcol[b] = (uint16_t)(tswz<R>(place[b]) * sizeof(C<R>));
        sg.nph = (uint32_t)B.phases.size() - sg.ph_begin;
        sg.nops = (uint32_t)B.ops.size() - sg.op_begin;
        sg.ncoef = B.ncoef - sg.coef_begin;
        sg.ngrad = (uint32_t)piece.grads.size();
        piece.seg = (int)B.segs.size();
        B.segs.push_back(sg);
        pieces.push_back(std::move(piece));
    }
    return pieces;
}

template <typename R, bool REV> size_t seg_smem(const TSeg &s) {
    return tile_buffers<R, REV>() * (sizeof(C<R>) << s.kt) + s.nops * sizeof(TOp) + s.ncoef * sizeof(C<R>) +
           s.nph * sizeof(TPhase) + (REV ? (size_t)s.ngrad * 4 * kTWarps * sizeof(double) : 0);
}
// The most that any segment takes (a wide step's coefficients may start one further on, a phase holds
// at least one step).  A kernel's shared-memory limit is set to this and not to one call's or batch's
// need: the limit belongs to the function, so a later, smaller one would refuse the launches of
// programs built before it.
template <typename R, bool REV> constexpr size_t max_seg_smem(int max_coefs) {
    return tile_buffers<R, REV>() * (sizeof(C<R>) << TGeo<R, REV>::kt) + kMaxTOps * (sizeof(TOp) + sizeof(TPhase)) +
           (max_coefs + kMaxTOps) * sizeof(C<R>) + (REV ? (size_t)kMaxTGrads * 4 * kTWarps * sizeof(double) : 0);
}

}  // namespace steps
}  // namespace b200sv
