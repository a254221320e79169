/*
 * Multi-row stack interpreter for fit records, forward and reverse: each
 * thread carries NR rows (f32 or f64) through one decode of every
 * instruction.
 *
 * A fit-record program (post-order records [op, kid0, kid1, slot],
 * my-version/src/fit.rs:985-1056) of a tree is evaluated on a stack exactly
 * like postfix bytecode. The host translates it once per batch into 8-byte
 * instructions: pushes of an input column or a constant slot, unary and
 * binary operators, and a binary operator fused with the push of its right
 * operand. The top of stack lives in registers (NR rows per thread),
 * deeper entries in shared-memory spill slots fixed at decode time.
 *
 * The reverse sweep is the mirror of the forward stack machine: an
 * operator's adjoint arrives on top of stack, its children's adjoints leave
 * through the same spill slot and top of stack their values used, so no
 * per-node value tape is needed. It runs over a second instruction list in
 * which every subtree without a constant is collapsed to the restore of the
 * adjoint below it (or dropped), since nothing in it has a constant to
 * differentiate. Only the local partials that lie on a path from a constant
 * to the root are kept, in a per-thread shared-memory tape. A zero adjoint
 * passes nothing to its operands, as the reference's adjoint does
 * (eval.cu:1245-1246, fit.rs:1479-1481).
 */
#pragma once

#include <cstring>
#include <vector>

#include "rc_ops.cuh"

enum FiKind {
    FI_PUSH_VAR = 0,   /* spill TOS to `spill`; TOS = x[imm]. Reverse: restore only */
    FI_PUSH_PARAM = 1, /* spill TOS; TOS = c[imm] */
    FI_PUSH_CACHE = 2, /* spill TOS; TOS = cached column imm of the candidate */
    FI_UNARY = 3,      /* TOS = op(TOS) */
    FI_BIN_S = 4,      /* TOS = op(slot[arg], TOS) */
    FI_BIN_V = 5,      /* TOS = op(TOS, x[imm]) */
    FI_BIN_P = 6,      /* TOS = op(TOS, c[imm]) */
    FI_HALT = 7
};

/* Flag bits above the kind: the left (or only) / right operand's subtree
   holds a constant, and a reverse store that adds to an earlier one. */
#define FI_KIND_MASK 7u
#define FI_HP_L 8u
#define FI_HP_R 16u
#define FI_ACC 32u

struct FIns {
    uint8_t kind;  /* FiKind | flags */
    uint8_t op;
    uint8_t arg;   /* spill slot of the left operand (FI_BIN_S) */
    uint8_t spill; /* slot a push spills TOS to, 0xff when the stack was empty */
    uint16_t imm;  /* input column or constant slot */
    uint16_t tape; /* first partial-tape slot of this instruction */
};
static_assert(sizeof(FIns) == 8, "FIns is 8 bytes");

__host__ __device__ constexpr bool fi_nonlinear(unsigned op)
{
    return op != OP_ADD && op != OP_SUB && op != OP_NEG;
}

/* Host translation of one fit-record program into the forward list `fwd`
   (ending in HALT) and the reverse list `rev` (walked last to first).
   Returns false when the records are not a tree in stack (post-) order,
   which the device path rejects.

   With `fwdc`, also the forward list in which every maximal constant-free
   subtree of two or more instructions is replaced by one push of a cached
   column (its values over all rows do not depend on the constants, so they
   are computed once per fit), and in `subs` the records of each such
   subtree, renumbered as a program of its own, in cache-column order.

   With `inputs`, the lists differentiate with respect to the inputs instead
   of the constants: the partials kept and the subtrees pruned are those on
   and off paths from an input leaf, a pruned left operand is restored by a
   push of kind FI_PUSH_CACHE, and the reverse sweep's input leaves (pushes
   and fused operands of kind FI_PUSH_VAR / FI_BIN_V) add their adjoints to
   the input's gradient (fi_reverse_x). No cached list is made. */
inline bool fi_decode(const uint32_t *rec, int m, std::vector<FIns> &fwd, std::vector<FIns> &rev,
                      int *nslots, int *ntape, std::vector<FIns> *fwdc = nullptr,
                      std::vector<std::vector<uint32_t>> *subs = nullptr, bool inputs = false)
{
    const uint32_t leaf_op = inputs ? OP_VAR : OP_CONST;
    struct Ent {
        int rec, first;
        bool hp;
    };
    std::vector<Ent> stack;
    std::vector<int> lo(m, 0), hi(m, -1), kid0(m, -1), kid1(m, -1), first_rec(m, 0);
    std::vector<char> hp(m, 0), fused(m, 0);
    int depth = 0, maxslot = -1, tape = 0;
    fwd.clear();
    rev.clear();
    for (int i = 0; i < m; ++i) {
        const uint32_t op = rec[4 * i], k0 = rec[4 * i + 1], k1 = rec[4 * i + 2],
                       slot = rec[4 * i + 3];
        FIns in;
        in.kind = 0;
        in.op = (uint8_t)op;
        in.arg = 0;
        in.spill = 0xff;
        in.imm = 0;
        in.tape = (uint16_t)tape;
        if (op == OP_CONST || op == OP_VAR) {
            if (slot > 0xffff || depth >= 250) return false;
            in.kind = op == OP_CONST ? FI_PUSH_PARAM : FI_PUSH_VAR;
            in.imm = (uint16_t)slot;
            if (depth >= 1) {
                in.spill = (uint8_t)(depth - 1);
                maxslot = maxslot > depth - 1 ? maxslot : depth - 1;
            }
            ++depth;
            hp[i] = op == leaf_op;
            first_rec[i] = i;
            lo[i] = (int)fwd.size();
            stack.push_back({i, (int)fwd.size(), op == leaf_op});
            fwd.push_back(in);
            hi[i] = lo[i];
        } else if (ft_op_binary(op)) {
            if (stack.size() < 2 || stack[stack.size() - 1].rec != (int)k1 ||
                stack[stack.size() - 2].rec != (int)k0)
                return false;
            const Ent L = stack[stack.size() - 2], R = stack[stack.size() - 1];
            stack.pop_back();
            const bool h = L.hp || R.hp;
            hp[i] = h;
            kid0[i] = (int)k0;
            kid1[i] = (int)k1;
            first_rec[i] = first_rec[k0];
            unsigned flags = 0;
            int np = 0;
            if (h) {
                flags = (L.hp ? FI_HP_L : 0u) | (R.hp ? FI_HP_R : 0u);
                if (fi_nonlinear(op)) np = (L.hp ? 1 : 0) + (R.hp ? 1 : 0);
            }
            in.kind = (uint8_t)(FI_BIN_S | flags);
            in.arg = (uint8_t)(depth - 2);
            --depth;
            FIns &prev = fwd.back();
            const unsigned pk = prev.kind & FI_KIND_MASK;
            if ((pk == FI_PUSH_VAR || pk == FI_PUSH_PARAM) && prev.spill == in.arg) {
                /* fuse "push right operand; op" */
                prev.kind = (uint8_t)((pk == FI_PUSH_VAR ? FI_BIN_V : FI_BIN_P) | flags);
                prev.op = (uint8_t)op;
                prev.spill = 0xff;
                prev.tape = (uint16_t)tape;
                fused[k1] = 1;
            } else {
                fwd.push_back(in);
            }
            tape += np;
            lo[i] = L.first;
            hi[i] = (int)fwd.size() - 1;
            stack.back() = {i, L.first, h};
        } else {
            if (stack.empty() || stack.back().rec != (int)k0) return false;
            const Ent C = stack.back();
            hp[i] = C.hp;
            kid0[i] = (int)k0;
            first_rec[i] = first_rec[k0];
            in.kind = (uint8_t)(FI_UNARY | (C.hp ? FI_HP_L : 0u));
            if (C.hp && fi_nonlinear(op)) ++tape;
            lo[i] = C.first;
            fwd.push_back(in);
            hi[i] = (int)fwd.size() - 1;
            stack.back() = {i, C.first, C.hp};
        }
        if (tape > 0xfff0) return false;
    }
    if (stack.size() != 1 || stack[0].rec != m - 1) return false;
    FIns h;
    h.kind = FI_HALT;
    h.op = 0;
    h.arg = 0;
    h.spill = 0xff;
    h.imm = 0;
    h.tape = (uint16_t)tape;
    fwd.push_back(h);
    *nslots = maxslot + 1;
    *ntape = tape;

    /* reverse list: maximal constant-free subtrees below a node with a
       constant become a restore of the adjoint below them (the left operand
       of a binary), or vanish (the right operand: its operator hands the left
       adjoint on directly; a fused leaf has no instruction of its own) */
    const int nf = (int)fwd.size() - 1;
    std::vector<int> skip_to(nf, -1);
    std::vector<char> emit(nf, 0);
    for (int i = 0; i < m; ++i) {
        if (!hp[i]) continue;
        const int kids[2] = {kid0[i], kid1[i]};
        for (int s = 0; s < 2; ++s) {
            const int k = kids[s];
            if (k < 0 || hp[k] || fused[k] || hi[k] < lo[k]) continue;
            skip_to[lo[k]] = hi[k];
            emit[lo[k]] = (s == 0 && fwd[lo[k]].spill != 0xff) ? 1 : 0;
        }
    }
    if (hp[m - 1]) {
        for (int j = 0; j < nf;) {
            if (skip_to[j] >= 0) {
                if (emit[j]) {
                    FIns r = fwd[j];
                    r.kind = inputs ? FI_PUSH_CACHE : FI_PUSH_VAR;
                    rev.push_back(r);
                }
                j = skip_to[j] + 1;
            } else {
                rev.push_back(fwd[j]);
                ++j;
            }
        }
    }
    /* a constant slot met again (in reverse order) accumulates */
    unsigned slots = 0;
    for (const FIns &r : rev) {
        const unsigned k = r.kind & FI_KIND_MASK;
        if (k == FI_PUSH_PARAM || k == FI_BIN_P) slots = slots > r.imm + 1u ? slots : r.imm + 1u;
    }
    std::vector<char> seen(slots, 0);
    for (int j = (int)rev.size() - 1; j >= 0; --j) {
        const unsigned k = rev[j].kind & FI_KIND_MASK;
        if (k == FI_PUSH_PARAM || k == FI_BIN_P) {
            if (seen[rev[j].imm]) rev[j].kind |= FI_ACC;
            seen[rev[j].imm] = 1;
        }
    }
    if (inputs) return true;
    if (fwdc) {
        /* cacheable: constant-free, its own instructions (not a fused leaf),
           two or more of them, and its parent has a constant (or it is the
           whole tree) */
        std::vector<int> parent(m, -1);
        for (int i = 0; i < m; ++i) {
            if (kid0[i] >= 0) parent[kid0[i]] = i;
            if (kid1[i] >= 0) parent[kid1[i]] = i;
        }
        std::vector<int> start_of(nf, -1);
        for (int k = 0; k < m; ++k) {
            if (hp[k] || fused[k] || hi[k] - lo[k] < 1) continue;
            if (parent[k] >= 0 && !hp[parent[k]]) continue;
            start_of[lo[k]] = k;
        }
        fwdc->clear();
        if (subs) subs->clear();
        int col = 0;
        for (int j = 0; j < nf;) {
            const int k = start_of[j];
            if (k < 0) {
                fwdc->push_back(fwd[j]);
                ++j;
                continue;
            }
            FIns c = fwd[j];
            c.kind = FI_PUSH_CACHE;
            c.op = 0;
            c.arg = 0;
            c.imm = (uint16_t)col++;
            c.tape = 0;
            fwdc->push_back(c);
            if (subs) {
                const int b = first_rec[k];
                std::vector<uint32_t> s(4 * (size_t)(k - b + 1));
                for (int r = b; r <= k; ++r) {
                    const uint32_t op = rec[4 * r];
                    const bool leaf = op == OP_CONST || op == OP_VAR;
                    const bool bin = !leaf && ft_op_binary(op);
                    s[4 * (r - b) + 0] = op;
                    s[4 * (r - b) + 1] = leaf ? rec[4 * r + 1] : rec[4 * r + 1] - (uint32_t)b;
                    s[4 * (r - b) + 2] = bin ? rec[4 * r + 2] - (uint32_t)b : rec[4 * r + 2];
                    s[4 * (r - b) + 3] = rec[4 * r + 3];
                }
                subs->push_back(std::move(s));
            }
            j = hi[k] + 1;
        }
        fwdc->push_back(fwd[nf]);
    }
    return true;
}

/* ---- device instruction words --------------------------------------------
 *
 * What bounds the sweeps is the interpreter itself: ncu shows the ALU pipe at
 * 40-52 % and the FMA and f64 pipes at 3-15 %, with most stalls fixed-latency
 * waits, so decoding costs more than the arithmetic. The device runs an
 * 8-byte form of the lists above in which the code names operator and operand
 * kind together (one dispatch reaches straight-line code), the next word is
 * loaded while the current one executes, and reverse steps that change
 * nothing (a sum's one live operand) are dropped on the host. Lists end with
 * FC_END / RC_END; a sweep may load (not run) the word after the end.
 *
 *   x: code | FO_* flags | z << 16    z: push: spill slot or FO_NONE; operator:
 *                                        tape slot of the right partial;
 *                                        FC_RARE: the operator
 *   y: operand | w << 16              operand: spill slot, input column, cache
 *                                        column or constant slot
 *                                     w: tape slot of the left / only partial */
struct FOp {
    uint32_t x, y;
};

inline FOp fi_op(unsigned code, unsigned y, unsigned z, unsigned w)
{
    return FOp{code | (z << 16), y | (w << 16)};
}

#define FO_NONE 0xffffu
#define FO_HP_L 256u  /* keep (or use) the left / only partial */
#define FO_HP_R 512u  /* keep (or use) the right partial */
#define FO_ACC 1024u  /* reverse: the constant's adjoint adds to an earlier one */
#define FO_COL 2048u  /* DIV / POW: right operand an input column */
#define FO_CON 4096u  /* DIV / POW: right operand a constant */

enum FiCode {
    FC_END = 0, FC_PUSH_V, FC_PUSH_C, FC_PUSH_P, FC_ADD_S, FC_ADD_V, FC_ADD_P, FC_SUB_S, FC_SUB_V,
    FC_SUB_P, FC_MUL_S, FC_MUL_V, FC_MUL_P, FC_DIV, FC_POW, FC_NEG, FC_SQUARE, FC_SIN, FC_COS,
    FC_EXP, FC_TANH, FC_SIG, FC_GAUSS, FC_RARE
};

enum RiCode {
    RC_END = 0,
    RC_RESTORE, /* a = slot y */
    RC_PUSH_P,  /* constant y receives a; a = slot z */
    RC_NEG,     /* a = -a */
    RC_MUL,     /* a = child(a, tape w) */
    RC_ADD2,    /* slot y = a (both operands live) */
    RC_SUB2,    /* slot y = a; a = -a */
    RC_MUL2,    /* slot y = child(a, tape w); a = child(a, tape z) */
    RC_ADD_P,   /* constant y receives a */
    RC_SUB_P,   /* constant y receives -a */
    RC_MUL_P,   /* constant y receives child(a, tape z); a = child(a, tape w), or 0 */
    RC_PUSH_X,  /* input y receives a; a = slot z */
    RC_ADD_X,   /* input y receives a */
    RC_SUB_X,   /* input y receives -a */
    RC_MUL_X    /* input y receives child(a, tape z); a = child(a, tape w), or 0 */
};

/* Append the device words of a forward list (its FI_HALT becomes FC_END). */
inline void fi_emit_forward(const std::vector<FIns> &fwd, std::vector<FOp> &out)
{
    for (const FIns &in : fwd) {
        const unsigned k = in.kind & FI_KIND_MASK;
        const unsigned fl = ((in.kind & FI_HP_L) ? FO_HP_L : 0u) | ((in.kind & FI_HP_R) ? FO_HP_R : 0u);
        if (k <= FI_PUSH_CACHE) {
            out.push_back(fi_op(k == FI_PUSH_VAR ? FC_PUSH_V : (k == FI_PUSH_PARAM ? FC_PUSH_P : FC_PUSH_C),
                                in.imm, in.spill == 0xff ? FO_NONE : in.spill, 0));
        } else if (k == FI_UNARY) {
            unsigned code = FC_RARE;
            switch (in.op) {
                case OP_NEG: code = FC_NEG; break;
                case OP_SQUARE: code = FC_SQUARE; break;
                case OP_SIN: code = FC_SIN; break;
                case OP_COS: code = FC_COS; break;
                case OP_EXP: code = FC_EXP; break;
                case OP_TANH: code = FC_TANH; break;
                case OP_SIG: code = FC_SIG; break;
                case OP_GAUSS: code = FC_GAUSS; break;
                default: break;
            }
            out.push_back(fi_op(code | fl, 0, in.op, in.tape));
        } else if (k != FI_HALT) {
            const unsigned mode = k == FI_BIN_S ? 0 : (k == FI_BIN_V ? 1 : 2);
            unsigned code;
            if (in.op == OP_DIV || in.op == OP_POW)
                code = (in.op == OP_DIV ? FC_DIV : FC_POW) |
                       (mode == 1 ? FO_COL : (mode == 2 ? FO_CON : 0u));
            else
                code = (in.op == OP_ADD ? FC_ADD_S : (in.op == OP_SUB ? FC_SUB_S : FC_MUL_S)) + mode;
            out.push_back(fi_op(code | fl, mode == 0 ? in.arg : in.imm,
                                in.tape + ((in.kind & FI_HP_L) ? 1u : 0u), in.tape));
        } else {
            out.push_back(fi_op(FC_END, 0, 0, 0));
        }
    }
}

/* Append the device words of a reverse list, in the order the device walks
   it (last to first), closed by RC_END. */
inline void fi_emit_reverse(const std::vector<FIns> &rev, bool inputs, std::vector<FOp> &out)
{
    for (int j = (int)rev.size() - 1; j >= 0; --j) {
        const FIns &in = rev[j];
        const unsigned k = in.kind & FI_KIND_MASK;
        const bool hl = in.kind & FI_HP_L, hr = in.kind & FI_HP_R;
        const unsigned acc = (in.kind & FI_ACC) ? FO_ACC : 0u;
        const unsigned spill = in.spill == 0xff ? FO_NONE : in.spill;
        const unsigned tl = in.tape, tr = in.tape + (hl ? 1u : 0u);
        if (k <= FI_PUSH_CACHE) {
            if (inputs ? k == FI_PUSH_VAR : k == FI_PUSH_PARAM)
                out.push_back(fi_op((inputs ? RC_PUSH_X : RC_PUSH_P) | acc, in.imm, spill, 0));
            else if (spill != FO_NONE)
                out.push_back(fi_op(RC_RESTORE, spill, 0, 0));
            continue;
        }
        const bool add = in.op == OP_ADD, sub = in.op == OP_SUB;
        if (k == FI_UNARY) {
            out.push_back(fi_op(in.op == OP_NEG ? RC_NEG : RC_MUL, 0, 0, tl));
        } else if (k == FI_BIN_S) {
            if (hl && hr)
                out.push_back(fi_op(add ? RC_ADD2 : (sub ? RC_SUB2 : RC_MUL2), in.arg, tr, tl));
            else if (!add && !sub)
                out.push_back(fi_op(RC_MUL, 0, 0, hr ? tr : tl));
            else if (sub && hr)
                out.push_back(fi_op(RC_NEG, 0, 0, 0));
        } else if (inputs ? k == FI_BIN_V : k == FI_BIN_P) {
            /* the right operand is a constant, or an input */
            const unsigned code = inputs ? (add ? RC_ADD_X : (sub ? RC_SUB_X : RC_MUL_X))
                                         : (add ? RC_ADD_P : (sub ? RC_SUB_P : RC_MUL_P)) | acc;
            out.push_back(fi_op(code | (hl ? FO_HP_L : 0u), in.imm, tr, tl));
        } else if (!add && !sub) {
            /* (in an adjoint list its operator has a live left operand) */
            out.push_back(fi_op(RC_MUL, 0, 0, tl));
        }
    }
    out.push_back(fi_op(RC_END, 0, 0, 0));
}

/* Local partials of one operator (ft_partials_f / ft_partials_d semantics,
   with the operator's value `r` reused where it is the same expression). A
   `pow` with a non-positive base passes nothing. */
template <typename V>
__device__ __forceinline__ void fi_partials(unsigned op, V x, V y, V r, V &d0, V &d1)
{
    d0 = V(0);
    d1 = V(0);
    switch (op) {
        case OP_EXP: d0 = r; break;
        case OP_LOG: d0 = V(1) / x; break;
        case OP_ABS: d0 = x >= V(0) ? V(1) : V(-1); break;
        case OP_SQRT: d0 = V(1) / (V(2) * r); break;
        case OP_SIN: d0 = cos(x); break;
        case OP_COS: d0 = -sin(x); break;
        case OP_TAN: {
            const V t = cos(x);
            d0 = V(1) / (t * t);
        } break;
        case OP_SINH: d0 = cosh(x); break;
        case OP_COSH: d0 = sinh(x); break;
        case OP_TANH: d0 = V(1) - r * r; break;
        case OP_SIG: d0 = r * (V(1) - r); break;
        case OP_GAUSS: d0 = (V(-2) * x) * r; break;
        case OP_SQUARE: d0 = V(2) * x; break;
        case OP_CUBE: d0 = V(3) * x * x; break;
        case OP_ERF: d0 = V(1.1283791670955126) * exp(-x * x); break;
        case OP_ERFC: d0 = V(-1.1283791670955126) * exp(-x * x); break;
        case OP_MUL: d0 = y; d1 = x; break;
        case OP_DIV: d0 = V(1) / y; d1 = -x / (y * y); break;
        case OP_POW:
            if (x > V(0)) {
                d0 = y * pow(x, y - V(1));
                d1 = r * log(x);
            }
            break;
        default: break;
    }
}

/* The rows a thread carries: NR values of type V, moved as one 4-, 8- or
   16-byte vector (spill slots, tape, column loads). */
template <typename V, int NR>
struct FiV {
    struct alignas(sizeof(V) * NR > 16 ? 16 : sizeof(V) * NR) V4 {
        V v[NR];
    };
    __device__ __forceinline__ static void unpack(const V4 &x, V *v)
    {
#pragma unroll
        for (int i = 0; i < NR; ++i) v[i] = x.v[i];
    }
    __device__ __forceinline__ static V4 pack(const V *v)
    {
        V4 x;
#pragma unroll
        for (int i = 0; i < NR; ++i) x.v[i] = v[i];
        return x;
    }
    /* read-only load of NR consecutive column values */
    __device__ __forceinline__ static void ldg(const V *p, V *v)
    {
        if constexpr (sizeof(V4) == 32) {
            FiV<V, NR / 2>::ldg(p, v);
            FiV<V, NR / 2>::ldg(p + NR / 2, v + NR / 2);
            return;
        }
        V4 x;
        if constexpr (sizeof(V4) == 16) {
            const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
            memcpy(&x, &t, 16);
        } else if constexpr (sizeof(V4) == 8) {
            const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
            memcpy(&x, &t, 8);
        } else {
            const float t = __ldg(reinterpret_cast<const float *>(p));
            memcpy(&x, &t, 4);
        }
        unpack(x, v);
    }
    __device__ __forceinline__ static V value(unsigned op, V a, V b)
    {
        if constexpr (sizeof(V) == 8) return ft_value_d(op, a, b);
        else return ft_value_f(op, a, b);
    }
};

#define FI_COPY(d, s) _Pragma("unroll") for (int i_ = 0; i_ < NR; ++i_) d[i_] = s[i_]
#define FI_CONST(d, c_)                                                            \
    do {                                                                            \
        const V fc_ = (c_);                                                         \
        _Pragma("unroll") for (int i_ = 0; i_ < NR; ++i_) d[i_] = fc_;              \
    } while (0)

template <typename V>
__device__ __forceinline__ V fi_child(V a, V d)
{
    return a == V(0) ? V(0) : a * d;
}

/* Keep the thread's partials of one operator: `d` by tape slot. */
template <typename V, int NR>
__device__ __forceinline__ void fi_keep(typename FiV<V, NR>::V4 *tape, unsigned slot, int S,
                                        const V *d)
{
    tape[slot * S] = FiV<V, NR>::pack(d);
}

/* A unary operator on the thread's rows: value, and with PARTIALS the
   partial when the word keeps it. */
#define FI_UN(OPC)                                                                     \
    {                                                                                  \
        V r[NR];                                                                       \
        _Pragma("unroll") for (int i = 0; i < NR; ++i) r[i] = F::value(OPC, t[i], V(0)); \
        if (PARTIALS && (in.x & FO_HP_L)) {                                            \
            V pl[NR], pr[NR];                                                          \
            _Pragma("unroll") for (int i = 0; i < NR; ++i)                             \
                fi_partials<V>(OPC, t[i], V(0), r[i], pl[i], pr[i]);                   \
            fi_keep<V, NR>(tape, (in.y >> 16), S, pl);                                         \
        }                                                                              \
        _Pragma("unroll") for (int i = 0; i < NR; ++i) t[i] = r[i];                    \
    }

/* t = a op b for an exact binary operator, its partials (of a product) kept. */
#define FI_BI(EXPR, PRODUCT)                                                           \
    {                                                                                  \
        if (PARTIALS && (PRODUCT)) {                                                   \
            if (in.x & FO_HP_L) fi_keep<V, NR>(tape, (in.y >> 16), S, b);                      \
            if (in.x & FO_HP_R) fi_keep<V, NR>(tape, (in.x >> 16), S, a);                      \
        }                                                                              \
        _Pragma("unroll") for (int i = 0; i < NR; ++i) t[i] = (EXPR);                  \
    }

/* Forward sweep of the thread's NR rows over a forward list. Constants from
   `cf`, inputs from `cols` (already at the thread's first row) with columns
   `npad` values apart, cached subtree values from `ccols` likewise. `stk`
   and `tape` are this thread's spill and tape row vectors, slots S apart.
   The prediction of row i is left in out[i]. */
template <typename V, int NR, bool PARTIALS>
__device__ __forceinline__ void fi_forward(const FOp *__restrict__ prog, const V *cf,
                                           const V *__restrict__ cols, unsigned npad,
                                           typename FiV<V, NR>::V4 *stk,
                                           typename FiV<V, NR>::V4 *tape, int S, V *out,
                                           const V *__restrict__ ccols = nullptr)
{
    using F = FiV<V, NR>;
    auto column = [&](const V *base, unsigned k, V *v) {
        F::ldg(base + (unsigned long long)k * npad, v);
    };
    V t[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) t[i] = V(0);
    FOp in = *prog;
    for (;;) {
        const FOp nx = *++prog;
        const unsigned code = in.x & 0xffu;
        switch (code) {
            case FC_PUSH_V:
                if ((in.x >> 16) != FO_NONE) stk[(in.x >> 16) * S] = F::pack(t);
                column(cols, (in.y & 0xffffu), t);
                break;
            case FC_PUSH_C:
                if ((in.x >> 16) != FO_NONE) stk[(in.x >> 16) * S] = F::pack(t);
                column(ccols, (in.y & 0xffffu), t);
                break;
            case FC_PUSH_P:
                if ((in.x >> 16) != FO_NONE) stk[(in.x >> 16) * S] = F::pack(t);
                FI_CONST(t, cf[(in.y & 0xffffu)]);
                break;
            case FC_ADD_S: { V a[NR], b[NR]; F::unpack(stk[(in.y & 0xffffu) * S], a); FI_COPY(b, t); FI_BI(a[i] + b[i], false) } break;
            case FC_SUB_S: { V a[NR], b[NR]; F::unpack(stk[(in.y & 0xffffu) * S], a); FI_COPY(b, t); FI_BI(a[i] - b[i], false) } break;
            case FC_MUL_S: { V a[NR], b[NR]; F::unpack(stk[(in.y & 0xffffu) * S], a); FI_COPY(b, t); FI_BI(a[i] * b[i], true) } break;
            case FC_ADD_V: { V a[NR], b[NR]; column(cols, (in.y & 0xffffu), b); FI_COPY(a, t); FI_BI(a[i] + b[i], false) } break;
            case FC_SUB_V: { V a[NR], b[NR]; column(cols, (in.y & 0xffffu), b); FI_COPY(a, t); FI_BI(a[i] - b[i], false) } break;
            case FC_MUL_V: { V a[NR], b[NR]; column(cols, (in.y & 0xffffu), b); FI_COPY(a, t); FI_BI(a[i] * b[i], true) } break;
            case FC_ADD_P: { V a[NR], b[NR]; FI_CONST(b, cf[(in.y & 0xffffu)]); FI_COPY(a, t); FI_BI(a[i] + b[i], false) } break;
            case FC_SUB_P: { V a[NR], b[NR]; FI_CONST(b, cf[(in.y & 0xffffu)]); FI_COPY(a, t); FI_BI(a[i] - b[i], false) } break;
            case FC_MUL_P: { V a[NR], b[NR]; FI_CONST(b, cf[(in.y & 0xffffu)]); FI_COPY(a, t); FI_BI(a[i] * b[i], true) } break;
            case FC_DIV:
            case FC_POW: {
                V a[NR], b[NR], r[NR];
                if (in.x & (FO_COL | FO_CON)) {
                    FI_COPY(a, t);
                    if (in.x & FO_COL) column(cols, (in.y & 0xffffu), b);
                    else FI_CONST(b, cf[(in.y & 0xffffu)]);
                } else {
                    F::unpack(stk[(in.y & 0xffffu) * S], a);
                    FI_COPY(b, t);
                }
                if (code == FC_DIV) {
#pragma unroll
                    for (int i = 0; i < NR; ++i) r[i] = F::value(OP_DIV, a[i], b[i]);
                    if (PARTIALS && (in.x & FO_HP_L)) {
                        V d[NR], e[NR];
#pragma unroll
                        for (int i = 0; i < NR; ++i) fi_partials<V>(OP_DIV, a[i], b[i], r[i], d[i], e[i]);
                        fi_keep<V, NR>(tape, (in.y >> 16), S, d);
                    }
                    if (PARTIALS && (in.x & FO_HP_R)) {
                        V d[NR], e[NR];
#pragma unroll
                        for (int i = 0; i < NR; ++i) fi_partials<V>(OP_DIV, a[i], b[i], r[i], d[i], e[i]);
                        fi_keep<V, NR>(tape, (in.x >> 16), S, e);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < NR; ++i) r[i] = F::value(OP_POW, a[i], b[i]);
                    if (PARTIALS && (in.x & (FO_HP_L | FO_HP_R))) {
                        V d[NR], e[NR];
#pragma unroll
                        for (int i = 0; i < NR; ++i) fi_partials<V>(OP_POW, a[i], b[i], r[i], d[i], e[i]);
                        if (in.x & FO_HP_L) fi_keep<V, NR>(tape, (in.y >> 16), S, d);
                        if (in.x & FO_HP_R) fi_keep<V, NR>(tape, (in.x >> 16), S, e);
                    }
                }
                FI_COPY(t, r);
            } break;
            case FC_NEG:
#pragma unroll
                for (int i = 0; i < NR; ++i) t[i] = -t[i];
                break;
            case FC_SQUARE: FI_UN(OP_SQUARE) break;
            case FC_SIN:
            case FC_COS: {
                const bool is_sin = code == FC_SIN;
                V r[NR];
                if (PARTIALS && (in.x & FO_HP_L)) {
                    V pl[NR];
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        if (sizeof(V) == 4) {
                            /* one f32 sincosf gives the value and the partial
                               (its results equal sinf / cosf bit for bit on
                               B200) */
                            float s, c;
                            sincosf((float)t[i], &s, &c);
                            r[i] = is_sin ? s : c;
                            pl[i] = is_sin ? c : -s;
                        } else if (is_sin) {
                            r[i] = F::value(OP_SIN, t[i], V(0));
                            pl[i] = cos(t[i]);
                        } else {
                            r[i] = F::value(OP_COS, t[i], V(0));
                            pl[i] = -sin(t[i]);
                        }
                    }
                    fi_keep<V, NR>(tape, (in.y >> 16), S, pl);
                } else if (is_sin) {
#pragma unroll
                    for (int i = 0; i < NR; ++i) r[i] = F::value(OP_SIN, t[i], V(0));
                } else {
#pragma unroll
                    for (int i = 0; i < NR; ++i) r[i] = F::value(OP_COS, t[i], V(0));
                }
                FI_COPY(t, r);
            } break;
            case FC_EXP: FI_UN(OP_EXP) break;
            case FC_TANH: FI_UN(OP_TANH) break;
            case FC_SIG: FI_UN(OP_SIG) break;
            case FC_GAUSS: FI_UN(OP_GAUSS) break;
            case FC_RARE:
                switch (in.x >> 16) {
                    case OP_TAN: FI_UN(OP_TAN) break;
                    case OP_LOG: FI_UN(OP_LOG) break;
                    case OP_SQRT: FI_UN(OP_SQRT) break;
                    case OP_ABS: FI_UN(OP_ABS) break;
                    case OP_CUBE: FI_UN(OP_CUBE) break;
                    case OP_SINH: FI_UN(OP_SINH) break;
                    case OP_COSH: FI_UN(OP_COSH) break;
                    case OP_ERF: FI_UN(OP_ERF) break;
                    case OP_ERFC: FI_UN(OP_ERFC) break;
                    default: FI_CONST(t, V(NAN)); break;
                }
                break;
            default: /* FC_END */
#pragma unroll
                for (int i = 0; i < NR; ++i) out[i] = t[i];
                return;
        }
        in = nx;
    }
}
#undef FI_UN
#undef FI_BI

/* Reverse sweep of the thread's rows over a reverse list. The adjoints start
   at the rows' seeds `a`. Constant adjoints are stored to g[slot * R + i * A]
   for row i (`g` is this thread's first row). Returns whether every stored
   value is finite. */
template <typename V, int NR>
__device__ __forceinline__ bool fi_reverse(const FOp *__restrict__ rev,
                                           typename FiV<V, NR>::V4 *stk,
                                           const typename FiV<V, NR>::V4 *tape, int S, V *g, int R,
                                           int A, V *a)
{
    using F = FiV<V, NR>;
    bool fin = true;
    auto give = [&](unsigned x, unsigned slot, const V *r) {
        V *gs = g + slot * R;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const V v = (x & FO_ACC) ? r[i] + gs[i * A] : r[i];
            gs[i * A] = v;
            fin = fin && isfinite(v);
        }
    };
    auto child = [&](unsigned slot, V *o) {
        V d[NR];
        F::unpack(tape[slot * S], d);
#pragma unroll
        for (int i = 0; i < NR; ++i) o[i] = fi_child(a[i], d[i]);
    };
    FOp in = *rev;
    for (;;) {
        const FOp nx = *++rev;
        switch (in.x & 0xffu) {
            case RC_RESTORE: F::unpack(stk[(in.y & 0xffffu) * S], a); break;
            case RC_PUSH_P:
                give(in.x, (in.y & 0xffffu), a);
                if ((in.x >> 16) != FO_NONE) F::unpack(stk[(in.x >> 16) * S], a);
                break;
            case RC_NEG:
#pragma unroll
                for (int i = 0; i < NR; ++i) a[i] = -a[i];
                break;
            case RC_MUL: child((in.y >> 16), a); break;
            case RC_ADD2: stk[(in.y & 0xffffu) * S] = F::pack(a); break;
            case RC_SUB2:
                stk[(in.y & 0xffffu) * S] = F::pack(a);
#pragma unroll
                for (int i = 0; i < NR; ++i) a[i] = -a[i];
                break;
            case RC_MUL2: {
                /* the left adjoint waits in its spill slot while the right
                   subtree is walked; that subtree's first push restores it */
                V l[NR];
                child((in.y >> 16), l);
                child((in.x >> 16), a);
                stk[(in.y & 0xffffu) * S] = F::pack(l);
            } break;
            case RC_ADD_P: give(in.x, (in.y & 0xffffu), a); break;
            case RC_SUB_P: {
                V r[NR];
#pragma unroll
                for (int i = 0; i < NR; ++i) r[i] = -a[i];
                give(in.x, (in.y & 0xffffu), r);
            } break;
            case RC_MUL_P: {
                V r[NR];
                child((in.x >> 16), r);
                give(in.x, (in.y & 0xffffu), r);
                if (in.x & FO_HP_L) child((in.y >> 16), a);
                else FI_CONST(a, V(0));
            } break;
            default: return fin; /* RC_END */
        }
        in = nx;
    }
}

/* Reverse sweep of the thread's rows over an input-mode reverse list (see
   fi_decode): the same stack machine as fi_reverse, seeded with a[], whose
   input leaves add their adjoints to the thread's gradient row vectors
   ig[col * S] (zeroed by the caller). Constants receive nothing. */
template <typename V, int NR>
__device__ __forceinline__ void fi_reverse_x(const FOp *__restrict__ rev,
                                             typename FiV<V, NR>::V4 *stk,
                                             const typename FiV<V, NR>::V4 *tape, int S,
                                             typename FiV<V, NR>::V4 *ig, V *a)
{
    using F = FiV<V, NR>;
    auto give = [&](unsigned col, const V *r) {
        V gv[NR];
        F::unpack(ig[col * S], gv);
#pragma unroll
        for (int i = 0; i < NR; ++i) gv[i] += r[i];
        ig[col * S] = F::pack(gv);
    };
    auto child = [&](unsigned slot, V *o) {
        V d[NR];
        F::unpack(tape[slot * S], d);
#pragma unroll
        for (int i = 0; i < NR; ++i) o[i] = fi_child(a[i], d[i]);
    };
    FOp in = *rev;
    for (;;) {
        const FOp nx = *++rev;
        switch (in.x & 0xffu) {
            case RC_RESTORE: F::unpack(stk[(in.y & 0xffffu) * S], a); break;
            case RC_PUSH_X:
                give((in.y & 0xffffu), a);
                if ((in.x >> 16) != FO_NONE) F::unpack(stk[(in.x >> 16) * S], a);
                break;
            case RC_NEG:
#pragma unroll
                for (int i = 0; i < NR; ++i) a[i] = -a[i];
                break;
            case RC_MUL: child((in.y >> 16), a); break;
            case RC_ADD2: stk[(in.y & 0xffffu) * S] = F::pack(a); break;
            case RC_SUB2:
                stk[(in.y & 0xffffu) * S] = F::pack(a);
#pragma unroll
                for (int i = 0; i < NR; ++i) a[i] = -a[i];
                break;
            case RC_MUL2: {
                V l[NR];
                child((in.y >> 16), l);
                child((in.x >> 16), a);
                stk[(in.y & 0xffffu) * S] = F::pack(l);
            } break;
            case RC_ADD_X: give((in.y & 0xffffu), a); break;
            case RC_SUB_X: {
                V r[NR];
#pragma unroll
                for (int i = 0; i < NR; ++i) r[i] = -a[i];
                give((in.y & 0xffffu), r);
            } break;
            case RC_MUL_X: {
                V r[NR];
                child((in.x >> 16), r);
                give((in.y & 0xffffu), r);
                if (in.x & FO_HP_L) child((in.y >> 16), a);
                else FI_CONST(a, V(0));
            } break;
            default: return; /* RC_END */
        }
        in = nx;
    }
}
#undef FI_COPY
#undef FI_CONST

/* D = A * B + D for one 8x8x4 f64 tile (mma.sync; A row-major, B
   column-major). Lane (g = lane / 4, t = lane % 4) holds A[g][t], B[t][g]
   and D[g][2t], D[g][2t + 1]. */
__device__ __forceinline__ void fi_dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}
