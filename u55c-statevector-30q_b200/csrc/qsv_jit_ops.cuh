// qsv_jit_ops.cuh -- MUX2 op application with the op's structure fixed at compile time.
//
// Used by sweep kernels specialised to one sweep structure (generated and compiled at run time by
// qsv_jit.cpp). Target slot, code variant, register-control mask and thread-control mask are template
// arguments, so per-op dispatch disappears, controls on register bits resolve at compile time (a
// controlled swap on register bits becomes a register renaming), and the phase layout's shared-memory
// offsets become immediates. The matrices stay data: packed coefficients at fixed offsets of the kernel's
// parameter block. Every update uses the interpreter's arithmetic (qsv_packed.cuh / qsv_device.cuh); forms
// that skip work only skip exact-zero terms or unselected pairs, so values equal the interpreter's and the
// CPU oracle's (up to the sign of a zero).
// What bounds it: the multiply-add pipe on sweeps with 12 dense ops, HBM on the others; every move that the
// compiler issues to that pipe counts. With the amplitudes as 64-bit values, coefficients stored packed and the
// repacking of the state's order kept off that pipe (swap_mid), the 30-qubit random-layer circuit of depth 24
// (HBM floor 220 ms) takes 273 ms where it took 283 ms, a 28-qubit random circuit on coarse kernels 28.5 instead
// of 29.3 ms (power-capped; both sides in turn).
#pragma once
#include "qsv_ops.cuh"
#include "qsv_packed.cuh"

namespace qsv {
namespace dev {

// thread base of a phase: lane bits 0-2 on tile bits L0-L2, lane bits 3-4 on tile bits LB0 / LB1
template <int L0, int L1, int L2, int LB0, int LB1>
__device__ __forceinline__ uint32_t jit_lane_base(int lane) {
    return ((uint32_t)(lane & 1) << L0) | ((uint32_t)((lane >> 1) & 1) << L1) | ((uint32_t)((lane >> 2) & 1) << L2) |
           ((uint32_t)((lane >> 3) & 1) << LB0) | ((uint32_t)((lane >> 4) & 1) << LB1);
}
template <int WBIT>
__device__ __forceinline__ uint32_t jit_warp_bit(int warp, int w) {
    return (uint32_t)((warp >> w) & 1) << WBIT;
}

// offset of register slot r in a phase whose register bits are the tile bits RBITS...
template <int... RBITS>
__device__ __forceinline__ constexpr uint32_t jit_reg_off(int r) {
    constexpr int bits[] = {RBITS...};
    uint32_t o = 0;
    for (int q = 0; q < (int)sizeof...(RBITS); q++)
        if ((r >> q) & 1) o += 1u << bits[q];
    return o;
}

// SWZ: the tile is stored with the 128-byte swizzle (swz128); the thread base and the register offsets
// (disjoint bits) are swizzled separately and combined with XOR, the offsets at compile time.
// SPLIT: the 16-byte slot holds (re0, re1, im0, im1) -- the in-tile order between two phases of a tile,
// which loads and stores straight into the (re, re) / (im, im) register pairs -- instead of the state's
// interleaved (re0, im0, re1, im1), which the first phase reads and the last phase writes.
template <int NV, int SWZ, int SPLIT, int... RBITS>
__device__ __forceinline__ void jit_load(const float2 *tile, uint32_t tb, uint32_t z, p2 (&R)[NV], p2 (&I)[NV]) {
    const uint32_t base = SWZ ? swz128(tb) : tb;
#pragma unroll
    for (int r = 0; r < NV; r++) {
        const uint32_t off = jit_reg_off<RBITS...>(r);
        const float2 *p = tile + (base ^ (SWZ ? swz128(off) : off));
        if (SPLIT) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
            R[r] = v.x;
            I[r] = v.y;
        } else {
            load_slot(p, R[r], I[r], z);
        }
    }
}
template <int NV, int SWZ, int SPLIT, int... RBITS>
__device__ __forceinline__ void jit_store(float2 *tile, uint32_t tb, uint32_t z, const p2 (&R)[NV], const p2 (&I)[NV]) {
    const uint32_t base = SWZ ? swz128(tb) : tb;
#pragma unroll
    for (int r = 0; r < NV; r++) {
        const uint32_t off = jit_reg_off<RBITS...>(r);
        float2 *p = tile + (base ^ (SWZ ? swz128(off) : off));
        if (SPLIT) {
            ulonglong2 v;
            v.x = R[r];
            v.y = I[r];
            *reinterpret_cast<ulonglong2 *>(p) = v;
        } else {
            store_slot(p, R[r], I[r], z);
        }
    }
}

// An op's coefficients C sit packed in the parameter block (layouts in qsv_iop.h) at a fixed offset: the compiler
// reads them as uniform 64-bit operands, with nothing to build per thread. (In ordinary registers, copied or loaded
// from a table in shared memory, the two-group kernels spill and take a quarter longer.)
__device__ __forceinline__ MatP jit_mat(const p2 *C) {
    MatP M;
#pragma unroll
    for (int e = 0; e < 8; e++) M.c[e] = C[e];
    M.n1 = C[8]; M.n3 = C[9]; M.n5 = C[10]; M.n7 = C[11];
    return M;
}
// controls outside the register bits hold (always, if there are none)
template <uint32_t CMTHR>
__device__ __forceinline__ bool jit_tok(uint32_t tb) {
    return CMTHR == 0u || (tb & CMTHR) == CMTHR;
}
__device__ __forceinline__ float jit_lo(p2 a) {
    float lo, hi;
    unpk(a, lo, hi);
    return lo;
}

// ---------------------------------------------------------------- register-bit target
#define QSV_PAIRS for (int r = 0; r < NV; r++) if (!(r & B))
#define QSV_CPAIRS for (int r = 0; r < NV; r++) if (!(r & B) && (r & CMREG) == CMREG)
template <int NV, int RBIT, int VAR, int CLS0, int CMREG, uint32_t CMTHR>
__device__ __forceinline__ void jit_reg(p2 (&R)[NV], p2 (&I)[NV], const p2 *C, uint32_t tb) {
    constexpr int B = 1 << RBIT;
    const bool tok = jit_tok<CMTHR>(tb);
    if constexpr (VAR == QSV_V_UNI_DENSE) {
        const MatP M = jit_mat(C);
#pragma unroll
        QSV_PAIRS dense_p(R[r], I[r], R[r | B], I[r | B], M);
    } else if constexpr (VAR == QSV_V_UNI_DENSE_R0) {
        const MatP M = jit_mat(C);
#pragma unroll
        QSV_PAIRS dense_r0_p(R[r], I[r], R[r | B], I[r | B], M);
    } else if constexpr (VAR == QSV_V_UNI_DIAG && CLS0 == QSV_M_DIAG1) {
#pragma unroll
        QSV_PAIRS cmul_p(R[r | B], I[r | B], C[0], C[1], C[2]);
    } else if constexpr (VAR == QSV_V_UNI_DIAG) {
#pragma unroll
        QSV_PAIRS { cmul_p(R[r], I[r], C[0], C[1], C[2]); cmul_p(R[r | B], I[r | B], C[3], C[4], C[5]); }
    } else if constexpr (VAR == QSV_V_CTRL_DENSE || VAR == QSV_V_CTRL_DENSE_SEL) {
        const MatP M = jit_mat(C);
        if (tok) {
#pragma unroll
            QSV_CPAIRS dense_p(R[r], I[r], R[r | B], I[r | B], M);
        }
    } else if constexpr (VAR == QSV_V_CTRL_DIAG1 || VAR == QSV_V_CTRL_DIAG1_SEL) {
        if (tok) {
#pragma unroll
            QSV_CPAIRS cmul_p(R[r | B], I[r | B], C[0], C[1], C[2]);
        }
    } else if constexpr (VAR == QSV_V_CTRL_SWAP_SEL) {
#pragma unroll
        QSV_CPAIRS {
            const p2 a = R[r], b = R[r | B], c = I[r], d = I[r | B];
            R[r] = tok ? b : a; R[r | B] = tok ? a : b;
            I[r] = tok ? d : c; I[r | B] = tok ? c : d;
        }
    } else if constexpr (VAR == QSV_V_UNI_SWAP || VAR == QSV_V_CTRL_SWAP) {
        // without controls outside the register bits this is a renaming
        if (tok) {
#pragma unroll
            QSV_CPAIRS { xchg(R[r], R[r | B]); xchg(I[r], I[r | B]); }
        }
    }
}

// QSV_V_MUX on a register bit. KIND controlled: tile bit 0 is a control, so only the high halves of the selected
// pairs change (scalar arithmetic on them). KIND general: matrix C on the selected pairs, C + 12 on the others.
template <int NV, int RBIT, int KIND, int CLS1, int CMREG, uint32_t CMTHR>
__device__ __forceinline__ void jit_reg_mux(p2 (&R)[NV], p2 (&I)[NV], const p2 *C, uint32_t tb) {
    constexpr int B = 1 << RBIT;
    const bool tok = jit_tok<CMTHR>(tb);
    if constexpr (KIND == QSV_K_MUX) {
        const MatP M = jit_mat(C), N = jit_mat(C + 12);
        if (tok) {
#pragma unroll
            QSV_CPAIRS dense_p(R[r], I[r], R[r | B], I[r | B], M);
        } else {
#pragma unroll
            QSV_CPAIRS dense_p(R[r], I[r], R[r | B], I[r | B], N);
        }
        if constexpr (CMREG != 0) {
#pragma unroll
            QSV_PAIRS if ((r & CMREG) != CMREG) dense_p(R[r], I[r], R[r | B], I[r | B], N);
        }
    } else if constexpr (CLS1 == QSV_M_XSWAP) {
#pragma unroll
        QSV_CPAIRS {
            const HalvesP a(R[r], I[r]), b(R[r | B], I[r | B]);
            a.put(R[r], I[r], tok ? b.rh : a.rh, tok ? b.ih : a.ih);
            b.put(R[r | B], I[r | B], tok ? a.rh : b.rh, tok ? a.ih : b.ih);
        }
    } else if constexpr (CLS1 != QSV_M_IDENT) {
        float m[8];
        if constexpr (CLS1 == QSV_M_DIAG1) {
            m[6] = hi_of(C[0]);
            m[7] = hi_of(C[1]);
        } else {
#pragma unroll
            for (int e = 0; e < 8; e++) m[e] = hi_of(C[e]);
        }
        if (tok) {
#pragma unroll
            QSV_CPAIRS {
                const HalvesP a(R[r], I[r]), b(R[r | B], I[r | B]);
                float x0r = a.rh, x0i = a.ih, x1r = b.rh, x1i = b.ih;
                pair_t<CLS1>(x0r, x0i, x1r, x1i, m);
                if (CLS1 != QSV_M_DIAG1) a.put(R[r], I[r], x0r, x0i);
                b.put(R[r | B], I[r | B], x1r, x1i);
            }
        }
    }
}
#undef QSV_PAIRS

// ---------------------------------------------------------------- lane-bit target (LB = lane bit 0..4)
// y = a own + b other, (a, b) = (m00, m01) on the bit-0 side and (m11, m10) on the bit-1 side
#define QSV_CSLOTS for (int r = 0; r < NV; r++) if ((r & CMREG) == CMREG)
template <int NV, int XM, int CMREG, bool ALL>
__device__ __forceinline__ void jit_lane_dense(p2 (&R)[NV], p2 (&I)[NV], const OwnP &M, bool tok) {
#pragma unroll
    QSV_CSLOTS {
        p2 yr = R[r], yi = I[r];
        own_p(yr, yi, shfl_p(R[r], XM), shfl_p(I[r], XM), M.ar, M.ai, M.na, M.br, M.bi, M.nb);
        R[r] = ALL || tok ? yr : R[r];
        I[r] = ALL || tok ? yi : I[r];
    }
}
template <int NV, int LB, int VAR, int CLS0, int CMREG, uint32_t CMTHR>
__device__ __forceinline__ void jit_lane(p2 (&R)[NV], p2 (&I)[NV], const p2 *C, uint32_t tb, int lane) {
    constexpr int XM = 1 << LB;
    const bool mine = (lane >> LB) & 1;
    const bool tok = jit_tok<CMTHR>(tb);
    if constexpr (VAR == QSV_V_UNI_DENSE || VAR == QSV_V_CTRL_DENSE || VAR == QSV_V_CTRL_DENSE_SEL) {
        jit_lane_dense<NV, XM, CMREG, CMTHR == 0u>(R, I, lane_own(jit_mat(C), mine), tok);
    } else if constexpr (VAR == QSV_V_UNI_DIAG && CLS0 != QSV_M_DIAG1) {
        const p2 ar = mine ? C[3] : C[0], ai = mine ? C[4] : C[1], na = mine ? C[5] : C[2];
#pragma unroll
        for (int r = 0; r < NV; r++) cmul_p(R[r], I[r], ar, ai, na);
    } else if constexpr (VAR == QSV_V_UNI_DIAG || VAR == QSV_V_CTRL_DIAG1 || VAR == QSV_V_CTRL_DIAG1_SEL) {
        if (mine && tok) {
#pragma unroll
            QSV_CSLOTS cmul_p(R[r], I[r], C[0], C[1], C[2]);
        }
    } else if constexpr (VAR == QSV_V_UNI_SWAP || VAR == QSV_V_CTRL_SWAP || VAR == QSV_V_CTRL_SWAP_SEL) {
#pragma unroll
        QSV_CSLOTS {
            const p2 a = shfl_p(R[r], XM), b = shfl_p(I[r], XM);
            R[r] = CMTHR == 0u || tok ? a : R[r];
            I[r] = CMTHR == 0u || tok ? b : I[r];
        }
    }
}
// QSV_V_MUX on a lane bit: as jit_reg_mux
template <int NV, int LB, int KIND, int CLS1, int CMREG, uint32_t CMTHR>
__device__ __forceinline__ void jit_lane_mux(p2 (&R)[NV], p2 (&I)[NV], const p2 *C, uint32_t tb, int lane) {
    constexpr int XM = 1 << LB;
    const bool mine = (lane >> LB) & 1;
    const bool tok = jit_tok<CMTHR>(tb);
    if constexpr (KIND == QSV_K_MUX) {
        const OwnP A = lane_own(jit_mat(C), mine), N = lane_own(jit_mat(C + 12), mine);
        const OwnP S = {tok ? A.ar : N.ar, tok ? A.ai : N.ai, tok ? A.na : N.na,
                        tok ? A.br : N.br, tok ? A.bi : N.bi, tok ? A.nb : N.nb};
        jit_lane_dense<NV, XM, CMREG, true>(R, I, S, true);
        if constexpr (CMREG != 0) {
#pragma unroll
            for (int r = 0; r < NV; r++)
                if ((r & CMREG) != CMREG)
                    own_p(R[r], I[r], shfl_p(R[r], XM), shfl_p(I[r], XM), N.ar, N.ai, N.na, N.br, N.bi, N.nb);
        }
    } else if constexpr (CLS1 == QSV_M_DIAG1) {
        if (mine && tok) {
            const float dr = hi_of(C[0]), di = hi_of(C[1]);
#pragma unroll
            QSV_CSLOTS {
                const HalvesP x(R[r], I[r]);
                float yr, yi;
                diag_own(yr, yi, dr, di, x.rh, x.ih);
                x.put(R[r], I[r], yr, yi);
            }
        }
    } else if constexpr (CLS1 != QSV_M_IDENT) {
        float ar = 0.f, ai = 0.f, br = 0.f, bi = 0.f;
        if constexpr (CLS1 != QSV_M_XSWAP) {
            const OwnP A = lane_own(jit_mat(C), mine);
            ar = hi_of(A.ar); ai = hi_of(A.ai); br = hi_of(A.br); bi = hi_of(A.bi);
        }
#pragma unroll
        QSV_CSLOTS {
            const HalvesP x(R[r], I[r]);
            float yr = __shfl_xor_sync(0xffffffffu, x.rh, XM), yi = __shfl_xor_sync(0xffffffffu, x.ih, XM);
            if (CLS1 != QSV_M_XSWAP) lin_own(yr, yi, ar, ai, br, bi, x.rh, x.ih, yr, yi);
            x.put(R[r], I[r], tok ? yr : x.rh, tok ? yi : x.ih);
        }
    }
}
#undef QSV_CSLOTS
#undef QSV_CPAIRS

// ---------------------------------------------------------------- tile-bit-0 target (halves of a slot)
// scalar arithmetic: the halves of a 64-bit register are ordinary registers, so nothing has to be exchanged
template <int NV, int KIND, int CLS0, int CLS1, int CMREG, uint32_t CMTHR>
__device__ __forceinline__ void jit_comp(p2 (&R)[NV], p2 (&I)[NV], const p2 *C, uint32_t tb) {
    constexpr bool UNI = KIND == QSV_K_UNI, CTRL = KIND == QSV_K_CTRL;
    const bool tok = jit_tok<CMTHR>(tb);
    auto mat = [](const p2 *c, float (&m)[8]) {        // own layout (qsv_iop.h)
        m[0] = jit_lo(c[0]); m[1] = jit_lo(c[1]); m[2] = jit_lo(c[3]); m[3] = jit_lo(c[4]);
        m[6] = hi_of(c[0]); m[7] = hi_of(c[1]); m[4] = hi_of(c[3]); m[5] = hi_of(c[4]);
    };
    float a[8], b[8];                                  // the selected slots' matrix, the others'
    constexpr int CA = UNI ? CLS0 : CLS1;
    // an exchange or the identity has code of its own and no coefficients, except as one of two matrices to choose
    // between: both of those are applied as dense ones, whatever their class
    if constexpr ((!UNI && !CTRL) || (CA != QSV_M_XSWAP && CA != QSV_M_IDENT)) mat(C, a);
    if constexpr (!UNI && !CTRL) mat(C + 12, b);
#pragma unroll
    for (int r = 0; r < NV; r++) {
        const bool regsel = (r & CMREG) == CMREG;
        if (CTRL && !regsel) continue;
        float x0r, x0i, x1r, x1i;
        unpk(R[r], x0r, x1r);
        unpk(I[r], x0i, x1i);
        if constexpr (UNI) {
            pair_t<CA>(x0r, x0i, x1r, x1i, a);
        } else if constexpr (CTRL) {
            if (tok) pair_t<CA>(x0r, x0i, x1r, x1i, a);
        } else {
            if (regsel && tok) pair_t<QSV_M_DENSE>(x0r, x0i, x1r, x1i, a);
            else pair_t<QSV_M_DENSE>(x0r, x0i, x1r, x1i, b);
        }
        R[r] = pk(x0r, x1r);
        I[r] = pk(x0i, x1i);
    }
}

}  // namespace dev
}  // namespace qsv
