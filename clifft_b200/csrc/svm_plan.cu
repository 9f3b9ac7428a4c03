// svm_plan.cu -- host-side formation of fused blocks (see svm_plan.h).
//
// Rules (the device executes exactly what is planned here):
//   * Only the axes an opcode moves amplitudes along must be tile axes:
//     targets of CNOT / multi-CNOT / SWAP / H / U2 / U4, the new axis of an
//     EXPAND, the measured axis of an X-basis measurement. Other axes enter
//     a micro-op's condition through tile-global index bits.
//   * Tile axes are padded with the lowest free axes, and a tile is at most
//     64 contiguous runs.
//   * An EXPAND takes two micro-op slots: a renormalisation may follow it.
//   * An active measurement ends its block.

#include "svm_plan.h"

#include <cstring>

#include "svm_kernel.cuh"

namespace cgpu {

namespace {

constexpr uint32_t kNoPlan = 0xffffffffu;
// States of at most one tile are blocked only from this rank on: every
// micro-op covers the whole tile, while a sweep covers the 2^k amplitudes.
constexpr uint32_t kSingleMinRank = 9;

struct Instr {
    uint32_t op, flags, a1, a2;
    uint64_t mask;
};

Instr decode(const uint8_t* code, uint32_t pc) {
    const uint8_t* I = code + size_t(pc) * 32;
    Instr x;
    uint16_t a1, a2;
    std::memcpy(&a1, I + 4, 2);
    std::memcpy(&a2, I + 6, 2);
    std::memcpy(&x.mask, I + 8, 8);
    x.op = I[0];
    if (x.op >= CLIFFT_OP_MEAS_DORMANT_STATIC_FORCED && x.op <= CLIFFT_OP_SWAP_MEAS_INTERFERE_FORCED)
        x.op -= CLIFFT_OP_MEAS_DORMANT_STATIC_FORCED - CLIFFT_OP_MEAS_DORMANT_STATIC;
    x.flags = I[2];
    x.a1 = a1;
    x.a2 = a2;
    return x;
}

uint32_t popc(uint64_t x) { return (uint32_t)__builtin_popcountll(x); }

struct Builder {
    const uint8_t* code;
    uint32_t n;
    PlanGeometry g;
    PlanSet out;

    uint64_t tile_axes(uint64_t need, uint32_t& r) const {
        uint64_t F = need;
        for (uint32_t a = 0; popc(F) < g.bits; ++a) F |= 1ull << a;
        r = (uint32_t)__builtin_ctzll(~F);
        return F;
    }
    bool is_expand(uint32_t op) const { return op >= CLIFFT_OP_EXPAND && op <= CLIFFT_OP_EXPAND_ROT; }
    bool is_active_meas(uint32_t op) const {
        return op >= CLIFFT_OP_MEAS_ACTIVE_DIAGONAL && op <= CLIFFT_OP_SWAP_MEAS_INTERFERE;
    }
    // the opcode touches the statevector at active rank k
    bool touches(const Instr& x, uint32_t k) const {
        switch (x.op) {
            case CLIFFT_OP_ARRAY_T:
            case CLIFFT_OP_ARRAY_T_DAG:
            case CLIFFT_OP_ARRAY_ROT:
            case CLIFFT_OP_ARRAY_U2: return x.a1 < k;
            case CLIFFT_OP_EXP_VAL: return true;
            default:
                return (x.op >= CLIFFT_OP_ARRAY_CNOT && x.op <= CLIFFT_OP_EXPAND_ROT) || is_active_meas(x.op);
        }
    }

    // ---- micro-ops of a block with tile axes F
    struct Emit {
        uint64_t F;
        std::vector<PlanOp>& ops;
        uint8_t bit(uint32_t axis) const {
            return (F >> axis) & 1u ? (uint8_t)popc(F & ((1ull << axis) - 1)) : (uint8_t)0xff;
        }
        uint32_t local(uint64_t axes) const {
            uint32_t m = 0;
            for (uint64_t w = axes & F; w; w &= w - 1) m |= 1u << bit((uint32_t)__builtin_ctzll(w));
            return m;
        }
        void operator()(uint8_t kind, uint32_t a, uint32_t b, uint64_t req, uint64_t par, uint8_t flags) {
            PlanOp m{};
            m.kind = kind;
            m.a = bit(a);
            m.b = bit(b);
            m.flags = flags;
            m.req = local(req);
            m.par = local(par);
            m.greq = req & ~F;
            m.gpar = par & ~F;
            ops.push_back(m);
        }
    };
    void emit(Emit& e, const Instr& x, uint32_t k) const {
        const uint64_t b1 = 1ull << (x.a1 & 63), b2 = 1ull << (x.a2 & 63);
        switch (x.op) {
            case CLIFFT_OP_ARRAY_CNOT: e(M_CNOT, x.a2, x.a2, b1, 0, 0); break;
            case CLIFFT_OP_ARRAY_CZ: e(M_CZ, x.a1, x.a2, b1 | b2, 0, 0); break;
            case CLIFFT_OP_ARRAY_SWAP: e(M_SWAP, x.a1, x.a2, 0, 0, 0); break;
            case CLIFFT_OP_ARRAY_MULTI_CNOT: e(M_MCNOT, x.a1, x.a1, 0, x.mask & ~b1, MF_PARITY); break;
            case CLIFFT_OP_ARRAY_MULTI_CZ: e(M_MCZ, x.a1, x.a1, b1, x.mask, MF_PARITY); break;
            case CLIFFT_OP_ARRAY_H: e(M_H, x.a1, x.a1, 0, 0, 0); break;
            case CLIFFT_OP_ARRAY_S:
            case CLIFFT_OP_ARRAY_S_DAG: e(M_PHASE, x.a1, x.a1, b1, 0, 0); break;
            case CLIFFT_OP_ARRAY_T:
            case CLIFFT_OP_ARRAY_T_DAG:
            case CLIFFT_OP_ARRAY_ROT:
                if (x.a1 < k) e(M_PHASE, x.a1, x.a1, b1, 0, 0);
                break;
            case CLIFFT_OP_ARRAY_U2:
                if (x.a1 < k) e(M_U2, x.a1, x.a1, 0, 0, 0);
                break;
            case CLIFFT_OP_ARRAY_U4: e(M_U4, x.a1, x.a2, 0, 0, 0); break;
            case CLIFFT_OP_EXPAND:
            case CLIFFT_OP_EXPAND_T:
            case CLIFFT_OP_EXPAND_T_DAG:
            case CLIFFT_OP_EXPAND_ROT:
                e(M_EXPAND, x.a1, x.a1, 0, 0, x.op == CLIFFT_OP_EXPAND ? MF_COPY : 0);
                e(M_NOP, x.a1, x.a1, 0, 0, 0);  // becomes M_SCALE when the shot renormalises here
                break;
            default: break;
        }
    }

    // ---- index runs as affine maps over GF(2) (see apply_index_run)
    static bool index_map(uint8_t kind) {
        return kind == M_CNOT || kind == M_SWAP || kind == M_MCNOT || kind == M_CZ || kind == M_MCZ ||
               kind == M_PHASE;
    }
    void compile_runs(PlanOp* m, uint32_t count) const {
        for (uint32_t j = 0; j < count;) {
            uint32_t e = j;
            while (e < count && index_map(m[e].kind)) ++e;
            if (e - j < 2) {
                ++j;
                continue;
            }
            uint16_t rows[12];
            for (uint32_t i = 0; i < g.bits; ++i) rows[i] = (uint16_t)(1u << i);
            for (uint32_t q = j; q < e; ++q) {
                PlanOp& o = m[q];
                auto parity_row = [&] {
                    uint16_t x = 0;
                    for (uint32_t w = o.par; w; w &= w - 1) x ^= rows[__builtin_ctz(w)];
                    return x;
                };
                if (o.kind == M_CNOT) {
                    if (o.req) rows[o.a] ^= rows[__builtin_ctz(o.req)];
                } else if (o.kind == M_MCNOT) {
                    rows[o.a] ^= parity_row();
                } else if (o.kind == M_SWAP) {
                    std::swap(rows[o.a], rows[o.b]);
                } else {
                    uint8_t c = 0;
                    for (uint32_t w = o.req; w; w &= w - 1) o.row[c++] = rows[__builtin_ctz(w)];
                    if (o.flags & MF_PARITY) o.row[c++] = parity_row();
                    o.n_rows = c;
                }
            }
            for (uint32_t c = 0; c < g.bits; ++c) {
                uint32_t col = 0;
                for (uint32_t i = 0; i < g.bits; ++i) col |= ((rows[i] >> c) & 1u) << i;
                m[j].cols[c] = (uint16_t)col;
            }
            j = e;
        }
    }

    // The block that starts at pc with active rank k; returns the number of
    // instructions it takes, 0 for none.
    uint32_t block(uint32_t pc, uint32_t k) {
        const bool wide = g.max_ops > 1;
        const bool single = k <= g.bits;
        if (single && !(g.team && k >= kSingleMinRank)) return 0;
        uint64_t need = 0, fresh = 0;
        uint32_t slots = 0, sweeps = 0, kk = k, end = pc, term = 0, term_kind = 0;
        for (; end < n; ++end) {
            const Instr x = decode(code, end);
            uint64_t nd = 0;
            uint32_t cost = 0, tk = 0;
            bool expand = false, ok = true;
            if (frame_op(x.op)) continue;
            switch (x.op) {
                case CLIFFT_OP_ARRAY_CNOT: nd = 1ull << x.a2; cost = 1; break;
                case CLIFFT_OP_ARRAY_MULTI_CNOT: nd = 1ull << x.a1; cost = 1; break;
                case CLIFFT_OP_ARRAY_SWAP:
                case CLIFFT_OP_ARRAY_U4: nd = (1ull << x.a1) | (1ull << x.a2); cost = 1; break;
                case CLIFFT_OP_ARRAY_H: nd = 1ull << x.a1; cost = 1; break;
                case CLIFFT_OP_ARRAY_CZ:
                case CLIFFT_OP_ARRAY_MULTI_CZ:
                case CLIFFT_OP_ARRAY_S:
                case CLIFFT_OP_ARRAY_S_DAG: cost = 1; break;
                case CLIFFT_OP_ARRAY_T:
                case CLIFFT_OP_ARRAY_T_DAG:
                case CLIFFT_OP_ARRAY_ROT: cost = x.a1 < kk ? 1 : 0; break;
                case CLIFFT_OP_ARRAY_U2:
                    if (x.a1 < kk) {
                        nd = 1ull << x.a1;
                        cost = 1;
                    }
                    break;
                case CLIFFT_OP_EXPAND:
                case CLIFFT_OP_EXPAND_T:
                case CLIFFT_OP_EXPAND_T_DAG:
                case CLIFFT_OP_EXPAND_ROT:
                    ok = wide && !(single && kk == g.bits);
                    nd = 1ull << kk;
                    cost = 2;
                    expand = true;
                    break;
                case CLIFFT_OP_MEAS_ACTIVE_DIAGONAL:
                    ok = wide;
                    tk = 1;
                    if (single) nd = 1ull << (kk - 1);
                    break;
                case CLIFFT_OP_MEAS_ACTIVE_INTERFERE:
                    ok = wide;
                    tk = 2;
                    nd = 1ull << (kk - 1);
                    cost = 1;
                    break;
                case CLIFFT_OP_SWAP_MEAS_INTERFERE:
                    ok = wide;
                    tk = x.a1 != x.a2 ? 3 : 2;
                    nd = (1ull << x.a1) | (1ull << x.a2);
                    cost = tk == 3 ? 2 : 1;
                    break;
                default: ok = false;
            }
            if (!ok) break;
            const uint64_t cand = need | nd;
            if (popc(cand) > g.bits || slots + cost > g.max_ops) break;
            if (nd && !single) {
                uint32_t r;
                tile_axes(cand, r);
                if (g.bits - r > (uint32_t)kMaxRunsLog2) break;
            }
            need = cand;
            slots += cost;
            if (expand) {
                fresh |= 1ull << kk;
                kk++;
            } else if (cost && !tk) {
                sweeps++;
            }
            if (tk) {
                term = end++;
                term_kind = tk;
                break;
            }
        }
        // a block of EXPANDs alone costs more than the plain expansions
        if (sweeps < 1 && !term_kind) return 0;
        BlockPlan p{};
        p.pc = pc;
        p.n_instr = end - pc;
        p.F = tile_axes(single ? 0 : need, p.r);
        p.C = single ? 0 : ((kk == 64) ? ~0ull : ((1ull << kk) - 1)) & ~p.F;
        p.kk = kk;
        p.single = single;
        p.n_fresh = popc(fresh);
        p.term_kind = term_kind;
        p.term_pc = term;
        for (uint64_t w = fresh; w; w &= w - 1) {
            const uint32_t at = popc(p.F & ((w & (~w + 1)) - 1));
            p.fresh_local |= 1u << at;
            if (!single) p.skip |= 1u << (at - p.r);
        }
        p.first_mop = (uint32_t)out.ops.size();
        Emit e{p.F, out.ops};
        uint32_t rank = k;
        for (uint32_t q = pc; q < (term_kind ? term : end); ++q) {
            const Instr x = decode(code, q);
            emit(e, x, rank);
            if (is_expand(x.op)) rank++;
        }
        p.n_body = (uint32_t)out.ops.size() - p.first_mop;
        if (term_kind) {
            const Instr x = decode(code, term);
            const uint32_t fa = x.a1, tt = term_kind == 3 ? x.a2 : x.a1;
            if (term_kind == 3) e(M_SWAP, fa, tt, 0, 0, 0);
            if (term_kind >= 2) e(M_H, tt, tt, 0, 0, 0);
            p.red_local = (p.F >> tt) & 1u;
            p.red_bit = p.red_local ? popc(p.F & ((1ull << tt) - 1)) : tt;
        }
        p.n_mops = (uint32_t)out.ops.size() - p.first_mop;
        compile_runs(out.ops.data() + p.first_mop, p.n_mops);
        out.blocks.push_back(p);
        return end - pc;
    }

    void build() {
        uint32_t k = 0;
        for (uint32_t pc = 0; pc < n;) {
            const Instr x = decode(code, pc);
            uint32_t used = 0;
            // a CTA's control warp runs opcodes that do not touch the
            // statevector by itself; a warp offers every opcode to a block
            if (!frame_op(x.op) && (!g.cta || touches(x, k))) used = block(pc, k);
            for (uint32_t q = pc; q < pc + (used ? used : 1); ++q) {
                const uint32_t op = decode(code, q).op;
                if (is_expand(op)) ++k;
                if (is_active_meas(op)) --k;
            }
            pc += used ? used : 1;
        }
        BlockPlan last{};
        last.pc = kNoPlan;
        out.blocks.push_back(last);
    }
};

}  // namespace

PlanSet plan_blocks(const uint8_t* code, uint32_t n_code, const PlanGeometry& g) {
    Builder b{code, n_code, g, {}};
    b.build();
    return std::move(b.out);
}

}  // namespace cgpu
