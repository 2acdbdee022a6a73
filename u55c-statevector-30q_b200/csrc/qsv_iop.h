// qsv_iop.h -- op records as packed FP32x2 code reads them (host and device).
#pragma once
#include <cstring>

#include "qsv_plan.h"

#ifdef __CUDACC__
#define QSV_HD __host__ __device__ __forceinline__
#else
#define QSV_HD inline
#endif

namespace qsv {
namespace dev {

typedef unsigned long long p2;      // two packed floats: low half = amplitude with tile bit 0 clear

// ---------------------------------------------------------------- expanded op records
// What the interpreter reads of an op: one 16-byte header with the code path already chosen, and the matrix
// as packed coefficients, so that an op costs a few 16-byte shared-memory loads and no moves to build them
// (splatting 12 coefficients took as many instructions as a fifth of a dense op's arithmetic).
//   matrix layout (register and lane targets): c0..c7 = m00 m01 m10 m11 as (re, im) for both halves, then
//     -m00.im, -m01.im, -m10.im, -m11.im
//   own layout (tile-bit-0 target: low half, high half): a.re a.im -a.im b.re b.im -b.im with y = a own +
//     b other, (a, b) = (m00, m01) on the low half and (m11, m10) on the high half
//   phase layout: a.re a.im -a.im for the selected amplitudes (path BASE_DIAG: then the same for amplitudes
//     with the target bit set; path PHASE_HI: the high halves alone count)
// A path is a group (path >> 2) and, for register-bit targets, the register bit (path & 3).
enum : int {
    QSV_G_DENSE_R0 = 0,       // every pair; m00 real (its imaginary part an exact zero, as in every U3)
    QSV_G_DENSE = 1,          // every pair
    QSV_G_PHASE = 2,          // slots whose index has every bit of rm, where tok
    QSV_G_SWAP = 3,           // pairs in sel, where tok
    QSV_G_DIAG = 4,           // a on the bit-0 slots (phase layout), b on the others
    QSV_G_CDENSE = 5,         // pairs in sel, where tok
    QSV_G_HALF = 6,           // high halves of the pairs in sel, where tok
    QSV_G_MUX = 7,            // matrix a on the pairs in sel where tok, b on the others
    QSV_P_LANE_DENSE = 32,    // every slot
    QSV_P_LANE_CDENSE = 33,   // slots in sel, kept where not tok
    QSV_P_LANE_SWAP = 34,
    QSV_P_LANE_HALF = 35,     // high halves of the slots in sel, where tok
    QSV_P_LANE_MUX = 36,
    QSV_P_COMP_DENSE = 40,    // every slot
    QSV_P_COMP_CDENSE = 41,   // slots in sel, where tok
    QSV_P_COMP_SWAP = 42,
    QSV_P_COMP_MUX = 43,
    QSV_P_BASE_DIAG = 44,     // every slot, by a bit of the thread base
    QSV_P_SKIP = 45,
    QSV_P_PHASE_HI = 46,      // high halves of the slots in sel, where tok: a phase under tile bit 0
};
struct alignas(16) QsvIOp {
    uint32_t cm_thr;          // thread-base bits that must be set (tok)
    uint32_t path;
    uint32_t sel;             // slots r (of a pair: with the target bit clear) whose register-bit controls hold
    uint32_t aux;             // PHASE: rm; LANE: the lane bit's mask (LANE_HALF: + 32 to exchange); HALF: 1 to
                              // exchange; BASE_DIAG: the target's bit of the thread base
    p2 a[12], b[12];
};
static_assert(sizeof(QsvIOp) == 208, "16-byte header and two packed matrices");

QSV_HD p2 pack2(float lo, float hi) {
#ifdef __CUDA_ARCH__
    return (p2)__float_as_uint(lo) | ((p2)__float_as_uint(hi) << 32);
#else
    uint32_t l, h;
    std::memcpy(&l, &lo, 4);
    std::memcpy(&h, &hi, 4);
    return (p2)l | ((p2)h << 32);
#endif
}
// a factor on the amplitudes with the target and every control set: diag(1, d), with or without controls
template <class Op>
QSV_HD bool iop_phase(const Op &op) {
    return op.variant == QSV_V_CTRL_DIAG1 || op.variant == QSV_V_CTRL_DIAG1_SEL ||
           (op.variant == QSV_V_MUX && op.kind == QSV_K_CTRL && op.cls1 == QSV_M_DIAG1) ||
           (op.variant == QSV_V_UNI_DIAG && op.cls == QSV_M_DIAG1);
}
// complex128: the same header and paths (no tile-bit-0 forms), the applied matrix and, for a choice of two, the other
struct alignas(16) QsvIOpD {
    uint32_t cm_thr, path, sel, aux;
    double a[8], b[8];
};
// the header of an expanded record; slots: 2^(register bits) of the layout the op was planned for
template <class Op, class IOp>
QSV_HD void iop_header(const Op &op, int slots, IOp &o) {
    const int slot = op.slot, v = op.variant;
    const bool lane = slot >= QSV_SLOT_LANE0, comp = slot == QSV_SLOT_COMP, base = slot == QSV_SLOT_BASE;
    const int rb = slot - QSV_SLOT_REG0;
    const bool reg = !lane && !comp && !base;
    const bool ctrl = op.kind == QSV_K_CTRL, mux = op.kind == QSV_K_MUX;
    const bool swap = v == QSV_V_UNI_SWAP || v == QSV_V_CTRL_SWAP || v == QSV_V_CTRL_SWAP_SEL;
    const bool half = v == QSV_V_MUX && ctrl;        // controlled, tile bit 0 among the controls
    const bool high = iop_phase(op) && (comp || half);       // ... or the target: only the high halves are touched
    int path = QSV_P_SKIP, flag = 0;
    uint32_t thr = op.cm_thr, tmask = 0;
    int rm = op.cm_reg;
    if (v == QSV_V_SKIP) {
        path = QSV_P_SKIP;
    } else if (iop_phase(op) || (comp && op.cls == QSV_M_DIAG && !mux)) {
        path = high ? QSV_P_PHASE_HI : QSV_G_PHASE << 2;
        if (reg) rm |= 1 << rb;
        else if (!comp) thr |= 1u << op.tbit;
    } else if (v == QSV_V_UNI_DIAG) {
        if (reg) path = (QSV_G_DIAG << 2) + rb;
        else { path = QSV_P_BASE_DIAG; tmask = 1u << op.tbit; }
    } else if (comp) {
        if (mux) path = QSV_P_COMP_MUX;
        else if (op.cls == QSV_M_XSWAP) path = QSV_P_COMP_SWAP;
        else path = ctrl ? QSV_P_COMP_CDENSE : QSV_P_COMP_DENSE;
    } else if (lane) {
        if (half) { path = QSV_P_LANE_HALF; flag = op.cls1 == QSV_M_XSWAP; }
        else if (mux) path = QSV_P_LANE_MUX;
        else path = swap ? QSV_P_LANE_SWAP : ctrl ? QSV_P_LANE_CDENSE : QSV_P_LANE_DENSE;
    } else {
        int g;
        if (half) { g = QSV_G_HALF; flag = op.cls1 == QSV_M_XSWAP; }
        else if (mux) g = QSV_G_MUX;
        else if (swap) g = QSV_G_SWAP;
        else if (ctrl) g = QSV_G_CDENSE;
        else g = op.r00 ? QSV_G_DENSE_R0 : QSV_G_DENSE;
        path = (g << 2) + rb;
    }
    uint32_t sel = 0;
    const int need = high ? rm : op.cm_reg;
    for (int r = 0; r < slots; r++)
        if ((r & need) == need) sel |= 1u << r;
    o.cm_thr = thr;
    o.path = (uint32_t)path;
    o.sel = sel;
    o.aux = path == QSV_P_BASE_DIAG ? tmask
            : path == QSV_G_PHASE << 2 ? (uint32_t)rm
            : lane ? (1u << (slot - QSV_SLOT_LANE0)) | (flag ? 32u : 0u) : (uint32_t)flag;
}
// coefficient e of an expanded record: 0..11 = a[e], 12..23 = b[e - 12]
QSV_HD p2 iop_coef(const QsvOp &op, int e) {
    const bool comp = op.slot == QSV_SLOT_COMP, second = e >= 12;
    const float *m0 = op.m0, *m1 = op.m1;
    const int k = second ? e - 12 : e;
    if (iop_phase(op) || op.variant == QSV_V_UNI_DIAG || (comp && op.kind != QSV_K_MUX && op.cls == QSV_M_DIAG)) {
        // phase layout
        const float *m = op.kind == QSV_K_UNI ? m0 : m1;
        const bool one = iop_phase(op) || k >= 3;        // which diagonal entry (not for a tile-bit-0 target)
        const int i = (k % 3) == 0 ? 0 : 1;
        float lo, hi;
        if (comp) { lo = m[i]; hi = m[6 + i]; }
        else lo = hi = m[(one ? 6 : 0) + i];
        return (k % 3) == 2 ? pack2(-lo, -hi) : pack2(lo, hi);
    }
    // the matrix of this half of the record: a = the one the op applies (M1 under controls), b = M0 (MUX)
    const float *hi_m = op.kind == QSV_K_UNI || second ? m0 : m1;
    const float *lo_m = op.kind == QSV_K_MUX && op.cm_c ? m0 : hi_m;
    if (comp) {
        if (k >= 6) return 0;
        const int i = k < 3 ? (k ? 1 : 0) : (k == 3 ? 2 : 3);       // m00 / m01 on the low half
        const float lo = hi_m[i], hi = hi_m[i ^ 6];                 // m11 / m10 on the high half
        return k == 2 || k == 5 ? pack2(-lo, -hi) : pack2(lo, hi);
    }
    if (k < 8) return pack2(lo_m[k], hi_m[k]);
    const int i = 2 * (k - 8) + 1;
    return pack2(-lo_m[i], -hi_m[i]);
}

// A phase's thread layout as the interpreters look it up: a thread's base is lane[lane] ^ warp[warp], the tile index in
// the low half and its shared-memory position (swizzled or not) in the high half; rbit: positions of the register
// bits. Spelled out from the phase record, a phase cost about a hundred instructions per tile and warp.
struct alignas(16) PhaseTab {
    uint32_t lane[32], warp[16], rbit[4];
};
// entry e (0..51) of a phase's table; pos(x): the position of tile index x (linear over XOR)
template <class PH, class POS>
QSV_HD uint32_t phase_entry(const PH &Q, int e, int rb, int wb, POS &&pos) {
    uint32_t x = 0;
    if (e < 32) {
        for (int l = 0; l < 3; l++)
            if ((e >> l) & 1) x |= 1u << Q.lane_lo[l];
        for (int l = 0; l < 2; l++)
            if ((e >> (3 + l)) & 1) x |= 1u << Q.lane_bits[l];
    } else if (e < 48) {
        for (int w = 0; w < wb; w++)
            if (((e - 32) >> w) & 1) x |= 1u << Q.warp_bits[w];
    } else {
        return e - 48 < rb ? pos(1u << Q.reg_bits[e - 48]) : 0u;
    }
    return x | (pos(x) << 16);
}

}  // namespace dev
}  // namespace qsv
