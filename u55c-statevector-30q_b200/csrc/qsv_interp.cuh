// qsv_interp.cuh -- the interpreter's phase of a tile: ops read and dispatched at run time (sweep and batch
// kernels, complex64).
//
// A consumer thread holds 2^RB slots of its tile as 64-bit registers, R = (re, re) and I = (im, im) of the two
// amplitudes of tile bit 0, from the phase's loads to its stores. Every op works on these 64-bit values whole:
// packed FP32x2 multiply-adds for register-bit targets (two amplitude pairs per instruction), for lane-bit
// targets (shuffles) and for tile bit 0 itself (the partner of an amplitude is the other half of its register).
// What bounds it: with one dispatch per op, the amplitudes are live across every branch. Held as float2 (two
// 32-bit values that the packed instructions need in an aligned pair) the branches of the dispatch left them in
// different registers and the compiler reconciled them at every join, about two moves per multiply-add; held
// as 64-bit values, updated by loops whose final multiply-adds are the last use of what they replace, they
// stay in place. What is left is the latency of the dispatch itself, so a tile is spread over 16 warps (three
// register bits), each op's path is chosen when its record is expanded, its coefficients are stored packed and
// loaded before the path's branches, and diagonal ops run wherever their target sits.
// A 27-qubit random circuit of depth 10 (31 sweeps, HBM floor 10.2 ms): 34.1 ms with float2, 22.1 ms with
// 64-bit values, 16.6 ms as it is now; a 24-qubit one with Toffolis, depth 20 (81 sweeps, floor 3.3 ms): 11.1,
// 7.3, 5.8 ms. The arithmetic is the canonical chain of qsv_device.cuh for every variant (specialised variants
// only skip exact-zero terms and unselected pairs).
#pragma once
#include "qsv_device.cuh"
#include "qsv_iop.h"
#include "qsv_ops.cuh"
#include "qsv_packed.cuh"

namespace qsv {
namespace dev {

// ---------------------------------------------------------------- op record header
struct HdrP {
    uint4 w;
    __device__ __forceinline__ uint32_t cm_thr() const { return w.x; }
    __device__ __forceinline__ uint32_t path() const { return w.y; }
    __device__ __forceinline__ uint32_t sel() const { return w.z; }
    __device__ __forceinline__ uint32_t aux() const { return w.w; }
};
__device__ __forceinline__ HdrP hdr_of(const QsvIOp *op) {
    HdrP h;
    h.w = *reinterpret_cast<const uint4 *>(op);
    return h;
}

// ---------------------------------------------------------------- ops by path
#define QSV_PAIRS for (int r = 0; r < NV; r++) if (!(r & B))
#define QSV_SEL if ((sel >> r) & 1u)

// M: the record's first matrix, loaded before the path is chosen so that the loads and the branches overlap.
template <int NV, int RBIT>
__device__ __forceinline__ void dense_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M) {
    constexpr int B = 1 << RBIT;
#pragma unroll
    QSV_PAIRS dense_p(R[r], I[r], R[r | B], I[r | B], M);
}
template <int NV, int RBIT>
__device__ __forceinline__ void dense_r0_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M) {
    constexpr int B = 1 << RBIT;
#pragma unroll
    QSV_PAIRS dense_r0_p(R[r], I[r], R[r | B], I[r | B], M);
}
template <int NV, int RBIT>
__device__ __forceinline__ void diag_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M) {
    constexpr int B = 1 << RBIT;                 // phase layout: a.re a.im -a.im b.re b.im -b.im
#pragma unroll
    QSV_PAIRS { cmul_p(R[r], I[r], M.c[0], M.c[1], M.c[2]); cmul_p(R[r | B], I[r | B], M.c[3], M.c[4], M.c[5]); }
}
template <int NV, int RBIT>
__device__ __forceinline__ void cdense_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M, uint32_t sel, bool tok) {
    constexpr int B = 1 << RBIT;
    if (tok) {
#pragma unroll
        QSV_PAIRS QSV_SEL dense_p(R[r], I[r], R[r | B], I[r | B], M);
    }
}
template <int NV, int RBIT>
__device__ __forceinline__ void swap_op(p2 (&R)[NV], p2 (&I)[NV], uint32_t sel, bool tok) {
    constexpr int B = 1 << RBIT;
    if (tok) {
#pragma unroll
        QSV_PAIRS QSV_SEL { xchg(R[r], R[r | B]); xchg(I[r], I[r | B]); }
    }
}
template <int NV, int RBIT>
__device__ __forceinline__ void half_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M, uint32_t sel, bool tok, bool swap) {
    constexpr int B = 1 << RBIT;
    if (!tok) return;
    if (swap) {
#pragma unroll
        QSV_PAIRS QSV_SEL { xchg_hi(R[r], R[r | B]); xchg_hi(I[r], I[r | B]); }
        return;
    }
    float m[8];
#pragma unroll
    for (int e = 0; e < 8; e++) m[e] = hi_of(M.c[e]);
#pragma unroll
    QSV_PAIRS QSV_SEL {
        const HalvesP a(R[r], I[r]), b(R[r | B], I[r | B]);
        float yr, yi, zr, zi;
        lin_own(yr, yi, m[0], m[1], m[2], m[3], a.rh, a.ih, b.rh, b.ih);
        lin_own(zr, zi, m[6], m[7], m[4], m[5], b.rh, b.ih, a.rh, a.ih);
        a.put(R[r], I[r], yr, yi);
        b.put(R[r | B], I[r | B], zr, zi);
    }
}
template <int NV, int RBIT>
__device__ __forceinline__ void mux_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M, const p2 *other, uint32_t sel, bool tok) {
    constexpr int B = 1 << RBIT;
    cdense_op<NV, RBIT>(R, I, M, sel, tok);
    const MatP N = load_mat(other);
    if (!tok) sel = 0;
#pragma unroll
    QSV_PAIRS if (!((sel >> r) & 1u)) dense_p(R[r], I[r], R[r | B], I[r | B], N);
}

// A factor on the slots whose index has every bit of RM: straight-line code for each mask.
template <int NV, int RM>
__device__ __forceinline__ void phase_slots(p2 (&R)[NV], p2 (&I)[NV], p2 ar, p2 ai, p2 na) {
#pragma unroll
    for (int r = 0; r < NV; r++)
        if ((r & RM) == RM) cmul_p(R[r], I[r], ar, ai, na);
}
template <int NV>
__device__ __forceinline__ void phase_op(p2 (&R)[NV], p2 (&I)[NV], p2 ar, p2 ai, p2 na, int rm) {
    static_assert(NV <= 8, "one case per mask");
    if (rm == 0) phase_slots<NV, 0>(R, I, ar, ai, na);
    else if (rm == 1) phase_slots<NV, 1>(R, I, ar, ai, na);
    else if (rm == 2) phase_slots<NV, 2>(R, I, ar, ai, na);
    else if (rm == 3) phase_slots<NV, 3>(R, I, ar, ai, na);
    else if constexpr (NV > 4) {
        if (rm == 4) phase_slots<NV, 4>(R, I, ar, ai, na);
        else if (rm == 5) phase_slots<NV, 5>(R, I, ar, ai, na);
        else if (rm == 6) phase_slots<NV, 6>(R, I, ar, ai, na);
        else phase_slots<NV, 7>(R, I, ar, ai, na);
    }
}

// The same on the high halves alone (a phase on tile bit 0, or under a control there). The low halves stay as they are:
// a packed factor of (1, 0) for them would spread an infinity or a NaN from one part of an amplitude to the other. (That
// form was 0.9 % faster on a 27-qubit random circuit and 1.9 % on a transform; straight-line code for each slot mask,
// here or beside phase_op, was no faster than this.)
template <int NV>
__device__ __forceinline__ void phase_hi_op(p2 (&R)[NV], p2 (&I)[NV], const MatP &M, uint32_t sel) {
    const float dr = hi_of(M.c[0]), di = hi_of(M.c[1]);
#pragma unroll
    for (int r = 0; r < NV; r++)
        QSV_SEL {
            const HalvesP x(R[r], I[r]);
            float yr, yi;
            diag_own(yr, yi, dr, di, x.rh, x.ih);
            x.put(R[r], I[r], yr, yi);
        }
}

// Tile-bit-0 target: the two halves of every slot are a pair; each half is own, the other half its partner.
__device__ __forceinline__ OwnP first_own(const MatP &M) { return OwnP{M.c[0], M.c[1], M.c[2], M.c[3], M.c[4], M.c[5]}; }
template <int NV>
__device__ __forceinline__ void comp_pass(p2 (&R)[NV], p2 (&I)[NV], const OwnP &M, uint32_t sel) {
#pragma unroll
    for (int r = 0; r < NV; r++)
        QSV_SEL own_p(R[r], I[r], flip(R[r]), flip(I[r]), M.ar, M.ai, M.na, M.br, M.bi, M.nb);
}

// Lane-bit target: every slot's partner is the same slot of the partner lane; own and other as above with the
// side given by the lane. Register-bit controls are uniform (slots outside them are left alone, with no
// exchange); for the others every lane takes part in the exchange and keeps its slot where they do not hold.
template <int NV>
__device__ __forceinline__ void lane_dense(p2 (&R)[NV], p2 (&I)[NV], const OwnP &M, int xm, uint32_t sel, bool keep) {
#pragma unroll
    for (int r = 0; r < NV; r++)
        QSV_SEL {
            p2 yr = R[r], yi = I[r];
            own_p(yr, yi, shfl_p(R[r], xm), shfl_p(I[r], xm), M.ar, M.ai, M.na, M.br, M.bi, M.nb);
            R[r] = keep ? R[r] : yr;
            I[r] = keep ? I[r] : yi;
        }
}
template <int NV>
__device__ __forceinline__ void lane_op_p(p2 (&R)[NV], p2 (&I)[NV], const HdrP &h, const MatP &M, const QsvIOp *op,
                                          bool tok, int lane) {
    const int xm = (int)(h.aux() & 31u);
    const bool mine = lane & xm;
    const uint32_t sel = h.sel(), path = h.path();
    const OwnP A = lane_own(M, mine);
    if (path == QSV_P_LANE_DENSE) {
        lane_dense<NV>(R, I, A, xm, 0xffffffffu, false);
    } else if (path == QSV_P_LANE_CDENSE) {
        lane_dense<NV>(R, I, A, xm, sel, !tok);
    } else if (path == QSV_P_LANE_SWAP) {
#pragma unroll
        for (int r = 0; r < NV; r++)
            QSV_SEL {
                const p2 a = shfl_p(R[r], xm), b = shfl_p(I[r], xm);
                R[r] = tok ? a : R[r];
                I[r] = tok ? b : I[r];
            }
    } else if (path == QSV_P_LANE_HALF) {
        const bool swap = h.aux() & 32u;
        const float ar = hi_of(A.ar), ai = hi_of(A.ai), br = hi_of(A.br), bi = hi_of(A.bi);
#pragma unroll
        for (int r = 0; r < NV; r++)
            QSV_SEL {
                const HalvesP x(R[r], I[r]);
                float yr = __shfl_xor_sync(0xffffffffu, x.rh, xm), yi = __shfl_xor_sync(0xffffffffu, x.ih, xm);
                if (!swap) lin_own(yr, yi, ar, ai, br, bi, x.rh, x.ih, yr, yi);
                x.put(R[r], I[r], tok ? yr : x.rh, tok ? yi : x.ih);
            }
    } else {                                     // QSV_P_LANE_MUX
        const OwnP N = lane_own(load_mat(op->b), mine);
        const OwnP S = {tok ? A.ar : N.ar, tok ? A.ai : N.ai, tok ? A.na : N.na,
                        tok ? A.br : N.br, tok ? A.bi : N.bi, tok ? A.nb : N.nb};
        lane_dense<NV>(R, I, S, xm, sel, false);
        lane_dense<NV>(R, I, N, xm, ~sel, false);
    }
}
#undef QSV_PAIRS
#undef QSV_SEL

// The path is found by a short chain of branches in order of use (a jump table was slower: 19.8 against 18.2 ms
// on a 27-qubit random circuit).
template <int NV, int RB>
__device__ __forceinline__ void apply_op_p(const HdrP &h, const QsvIOp *op, p2 (&R)[NV], p2 (&I)[NV], uint32_t tb,
                                           int lane, int vary) {
    const bool tok = (tb & h.cm_thr()) == h.cm_thr();
    const uint32_t sel = h.sel(), path = h.path();
    const MatP M = load_mat((op + vary)->a);
#define QSV_BY_RBIT(G, CALL)                                                                \
    if (RB <= 1 || path == 4 * G) { constexpr int RBIT = 0; CALL; }                         \
    else if (RB <= 2 || path == 4 * G + 1) { constexpr int RBIT = RB > 1 ? 1 : 0; CALL; }   \
    else if (RB <= 3 || path == 4 * G + 2) { constexpr int RBIT = RB > 2 ? 2 : 0; CALL; }   \
    else { constexpr int RBIT = RB > 3 ? 3 : 0; CALL; }
    if (path < 4 * (QSV_G_DENSE_R0 + 1)) {
        QSV_BY_RBIT(QSV_G_DENSE_R0, (dense_r0_op<NV, RBIT>(R, I, M)))
    } else if (path < 4 * (QSV_G_DENSE + 1)) {
        QSV_BY_RBIT(QSV_G_DENSE, (dense_op<NV, RBIT>(R, I, M)))
    } else if (path == 4 * QSV_G_PHASE) {
        if (tok) phase_op<NV>(R, I, M.c[0], M.c[1], M.c[2], h.aux());
    } else if (path < 4 * (QSV_G_SWAP + 1)) {
        QSV_BY_RBIT(QSV_G_SWAP, (swap_op<NV, RBIT>(R, I, sel, tok)))
    } else if (path >= QSV_P_LANE_DENSE) {
        if (path <= QSV_P_LANE_MUX) {
            lane_op_p<NV>(R, I, h, M, op, tok, lane);
        } else if (path == QSV_P_PHASE_HI) {
            if (tok) phase_hi_op<NV>(R, I, M, sel);
        } else if (path == QSV_P_COMP_DENSE) {
            comp_pass<NV>(R, I, first_own(M), 0xffffffffu);
        } else if (path == QSV_P_BASE_DIAG) {
            const bool one = tb & h.aux();
            phase_slots<NV, 0>(R, I, one ? M.c[3] : M.c[0], one ? M.c[4] : M.c[1], one ? M.c[5] : M.c[2]);
        } else if (path == QSV_P_COMP_SWAP) {
            if (tok) {
#pragma unroll
                for (int r = 0; r < NV; r++)
                    if ((sel >> r) & 1u) { R[r] = flip(R[r]); I[r] = flip(I[r]); }
            }
        } else if (path == QSV_P_COMP_CDENSE) {
            if (tok) comp_pass<NV>(R, I, first_own(M), sel);
        } else if (path == QSV_P_COMP_MUX) {
            if (tok) comp_pass<NV>(R, I, first_own(M), sel);
            comp_pass<NV>(R, I, load_own(op->b), tok ? ~sel : 0xffffffffu);
        }
    } else if (path < 4 * (QSV_G_DIAG + 1)) {
        QSV_BY_RBIT(QSV_G_DIAG, (diag_op<NV, RBIT>(R, I, M)))
    } else if (path < 4 * (QSV_G_CDENSE + 1)) {
        QSV_BY_RBIT(QSV_G_CDENSE, (cdense_op<NV, RBIT>(R, I, M, sel, tok)))
    } else if (path < 4 * (QSV_G_HALF + 1)) {
        QSV_BY_RBIT(QSV_G_HALF, (half_op<NV, RBIT>(R, I, M, sel, tok, h.aux())))
    } else {
        QSV_BY_RBIT(QSV_G_MUX, (mux_op<NV, RBIT>(R, I, M, op->b, sel, tok)))
    }
#undef QSV_BY_RBIT
}

// A thread's place in a phase: tile index of its base, shared-memory positions of base and register bits (base and
// register offsets are placed separately: swz128 is linear over XOR).
template <int RB>
struct PhaseAt {
    uint32_t tb, base, rbit[RB];
};
template <int RB>
__device__ __forceinline__ PhaseAt<RB> phase_at(const PhaseTab *t, int lane, int warp) {
    PhaseAt<RB> p;
    const uint32_t v = t->lane[lane] ^ t->warp[warp];
    p.tb = v & 0xffffu;
    p.base = v >> 16;
    const uint4 r = *reinterpret_cast<const uint4 *>(t->rbit);
    const uint32_t b[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int q = 0; q < RB; q++) p.rbit[q] = b[q];
    return p;
}
// the same from a phase record, for a tile stored plainly (the batch kernel, whose phases are each run once)
template <int RB, int WB, class PH>
__device__ __forceinline__ PhaseAt<RB> phase_at(const PH &Q, int lane, int warp) {
    PhaseAt<RB> p;
    p.tb = ((uint32_t)(lane & 1) << Q.lane_lo[0]) | ((uint32_t)((lane >> 1) & 1) << Q.lane_lo[1]) |
           ((uint32_t)((lane >> 2) & 1) << Q.lane_lo[2]) | ((uint32_t)((lane >> 3) & 1) << Q.lane_bits[0]) |
           ((uint32_t)((lane >> 4) & 1) << Q.lane_bits[1]);
#pragma unroll
    for (int w = 0; w < WB; w++) p.tb |= (uint32_t)((warp >> w) & 1) << Q.warp_bits[w];
    p.base = p.tb;
#pragma unroll
    for (int r = 0; r < RB; r++) p.rbit[r] = 1u << Q.reg_bits[r];
    return p;
}

// One phase of a tile in shared memory: read the thread's 2^RB slots in the phase's layout, apply ops
// [op_begin, op_end), write them back. split_in / split_out: the slots hold (re0, re1, im0, im1), the in-tile order
// between two phases (the two registers as they are), instead of the state's interleaved order (first phase in,
// last phase out).
template <int NV, int RB>
__device__ __forceinline__ void run_phase(float2 *tile, const PhaseAt<RB> &at, const QsvIOp *ops, int op_begin,
                                          int op_end, int lane, uint32_t zero, bool split_in, bool split_out) {
    const uint32_t tb = at.tb;
    auto addr = [&](int r) -> uint32_t {
        uint32_t o = at.base;
#pragma unroll
        for (int q = 0; q < RB; q++)
            if ((r >> q) & 1) o ^= at.rbit[q];
        return o;
    };
    p2 R[NV], I[NV];
    if (split_in) {
#pragma unroll
        for (int r = 0; r < NV; r++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(tile + addr(r));
            R[r] = v.x;
            I[r] = v.y;
        }
    } else {
#pragma unroll
        for (int r = 0; r < NV; r++) load_slot(tile + addr(r), R[r], I[r], zero);
    }
    if (op_begin < op_end) {
        const uint32_t vary = lane_zero();           // coefficients are read at ops + vary
        HdrP next = hdr_of(ops + op_begin);          // the next op's header is read during the current op
        for (int o = op_begin; o < op_end; o++) {
            const HdrP h = next;
            if (o + 1 < op_end) next = hdr_of(ops + o + 1);
            apply_op_p<NV, RB>(h, ops + o, R, I, tb, lane, vary);
        }
    }
    if (split_out) {
#pragma unroll
        for (int r = 0; r < NV; r++) *reinterpret_cast<ulonglong2 *>(tile + addr(r)) = make_ulonglong2(R[r], I[r]);
    } else {
#pragma unroll
        for (int r = 0; r < NV; r++) store_slot(tile + addr(r), R[r], I[r], zero);
    }
}

}  // namespace dev
}  // namespace qsv
