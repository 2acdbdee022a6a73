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
// 64-bit values, 17.6 ms as it is now; a 24-qubit one with Toffolis, depth 20 (81 sweeps, floor 3.3 ms): 11.1,
// 7.3, 6.4 ms. The arithmetic is the canonical chain of qsv_device.cuh for every variant (specialised variants
// only skip exact-zero terms and unselected pairs).
#pragma once
#include <cstring>

#include "qsv_device.cuh"
#include "qsv_ops.cuh"

namespace qsv {
namespace dev {

typedef unsigned long long p2;      // two packed floats: low half = amplitude with tile bit 0 clear

__device__ __forceinline__ p2 pk(float lo, float hi) {
    p2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ p2 splat(float a) { return pk(a, a); }
__device__ __forceinline__ void unpk(p2 a, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a)); }
__device__ __forceinline__ p2 flip(p2 a) {       // exchange the halves
    float lo, hi;
    unpk(a, lo, hi);
    return pk(hi, lo);
}
__device__ __forceinline__ p2 fma2(p2 a, p2 b, p2 c) {
    p2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ p2 mul2(p2 a, p2 b) {
    p2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// ---------------------------------------------------------------- expanded op records
// What the interpreter reads of an op: one 16-byte header with the code path already chosen, and the matrix
// as packed coefficients, so that an op costs a few 16-byte shared-memory loads and no moves to build them
// (splatting 12 coefficients took as many instructions as a fifth of a dense op's arithmetic).
//   matrix layout (register and lane targets): c0..c7 = m00 m01 m10 m11 as (re, im) for both halves, then
//     -m00.im, -m01.im, -m10.im, -m11.im
//   own layout (tile-bit-0 target: low half, high half): a.re a.im -a.im b.re b.im -b.im with y = a own +
//     b other, (a, b) = (m00, m01) on the low half and (m11, m10) on the high half
//   phase layout: a.re a.im -a.im for the selected amplitudes (path BASE_DIAG: then the same for amplitudes
//     with the target bit set)
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

__host__ __device__ __forceinline__ p2 pack2(float lo, float hi) {
#ifdef __CUDA_ARCH__
    return pk(lo, hi);
#else
    uint32_t l, h;
    memcpy(&l, &lo, 4);
    memcpy(&h, &hi, 4);
    return (p2)l | ((p2)h << 32);
#endif
}
// a factor on the amplitudes with the target and every control set: diag(1, d), with or without controls
__host__ __device__ __forceinline__ bool iop_phase(const QsvOp &op) {
    return op.variant == QSV_V_CTRL_DIAG1 || op.variant == QSV_V_CTRL_DIAG1_SEL ||
           (op.variant == QSV_V_MUX && op.kind == QSV_K_CTRL && op.cls1 == QSV_M_DIAG1) ||
           (op.variant == QSV_V_UNI_DIAG && op.cls == QSV_M_DIAG1);
}
// the header of an expanded record; slots: 2^(register bits) of the layout the op was planned for
__host__ __device__ __forceinline__ void iop_header(const QsvOp &op, int slots, QsvIOp &o) {
    const int slot = op.slot, v = op.variant;
    const bool lane = slot >= QSV_SLOT_LANE0, comp = slot == QSV_SLOT_COMP, base = slot == QSV_SLOT_BASE;
    const int rb = slot - QSV_SLOT_REG0;
    const bool reg = !lane && !comp && !base;
    const bool ctrl = op.kind == QSV_K_CTRL, mux = op.kind == QSV_K_MUX;
    const bool swap = v == QSV_V_UNI_SWAP || v == QSV_V_CTRL_SWAP || v == QSV_V_CTRL_SWAP_SEL;
    const bool half = v == QSV_V_MUX && ctrl;        // controlled, tile bit 0 among the controls
    int path = QSV_P_SKIP, flag = 0;
    uint32_t thr = op.cm_thr, tmask = 0;
    int rm = op.cm_reg;
    if (v == QSV_V_SKIP) {
        path = QSV_P_SKIP;
    } else if (iop_phase(op) || (comp && op.cls == QSV_M_DIAG && !mux)) {
        path = QSV_G_PHASE << 2;
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
    for (int r = 0; r < slots; r++)
        if ((r & op.cm_reg) == op.cm_reg) sel |= 1u << r;
    o.cm_thr = thr;
    o.path = (uint32_t)path;
    o.sel = sel;
    o.aux = path == QSV_P_BASE_DIAG ? tmask
            : path == QSV_G_PHASE << 2 ? (uint32_t)rm
            : lane ? (1u << (slot - QSV_SLOT_LANE0)) | (flag ? 32u : 0u) : (uint32_t)flag;
}
// coefficient e of an expanded record: 0..11 = a[e], 12..23 = b[e - 12]
__host__ __device__ __forceinline__ p2 iop_coef(const QsvOp &op, int e) {
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
        else { lo = hi = m[(one ? 6 : 0) + i]; if (op.kind == QSV_K_CTRL && op.cm_c) lo = i ? 0.f : 1.f; }
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

// A matrix for packed pairs.
struct MatP {
    p2 c[8], n1, n3, n5, n7;
};
__device__ __forceinline__ MatP load_mat(const p2 *m) {
    MatP M;
    const ulonglong2 *v = reinterpret_cast<const ulonglong2 *>(m);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const ulonglong2 x = v[e];
        M.c[2 * e] = x.x;
        M.c[2 * e + 1] = x.y;
    }
    const ulonglong2 x = v[4], y = v[5];
    M.n1 = x.x; M.n3 = x.y; M.n5 = y.x; M.n7 = y.y;
    return M;
}
struct OwnP {
    p2 ar, ai, na, br, bi, nb;
};
__device__ __forceinline__ OwnP load_own(const p2 *m) {
    const ulonglong2 *v = reinterpret_cast<const ulonglong2 *>(m);
    const ulonglong2 x = v[0], y = v[1], z = v[2];
    return OwnP{x.x, x.y, y.x, y.y, z.x, z.y};
}
// the lane's side of a matrix: y = a own + b other
__device__ __forceinline__ OwnP lane_own(const MatP &M, bool mine) {
    return OwnP{mine ? M.c[6] : M.c[0], mine ? M.c[7] : M.c[1], mine ? M.n7 : M.n1,
                mine ? M.c[4] : M.c[2], mine ? M.c[5] : M.c[3], mine ? M.n5 : M.n3};
}
__device__ __forceinline__ float hi_of(p2 a) {
    float lo, hi;
    unpk(a, lo, hi);
    return hi;
}

// ---------------------------------------------------------------- pair arithmetic
__device__ __forceinline__ void dense_p(p2 &x0r, p2 &x0i, p2 &x1r, p2 &x1i, const MatP &M) {
    const p2 p0r = fma2(M.n1, x0i, fma2(M.c[2], x1r, mul2(M.n3, x1i)));
    const p2 p0i = fma2(M.c[1], x0r, fma2(M.c[2], x1i, mul2(M.c[3], x1r)));
    const p2 p1r = fma2(M.n7, x1i, fma2(M.c[4], x0r, mul2(M.n5, x0i)));
    const p2 p1i = fma2(M.c[7], x1r, fma2(M.c[4], x0i, mul2(M.c[5], x0r)));
    x0r = fma2(M.c[0], x0r, p0r);
    x0i = fma2(M.c[0], x0i, p0i);
    x1r = fma2(M.c[6], x1r, p1r);
    x1i = fma2(M.c[6], x1i, p1i);
}
// m00 real (every U3): its two m00.im terms are exact zeros
__device__ __forceinline__ void dense_r0_p(p2 &x0r, p2 &x0i, p2 &x1r, p2 &x1i, const MatP &M) {
    const p2 p0r = fma2(M.c[2], x1r, mul2(M.n3, x1i));
    const p2 p0i = fma2(M.c[2], x1i, mul2(M.c[3], x1r));
    const p2 p1r = fma2(M.n7, x1i, fma2(M.c[4], x0r, mul2(M.n5, x0i)));
    const p2 p1i = fma2(M.c[7], x1r, fma2(M.c[4], x0i, mul2(M.c[5], x0r)));
    x0r = fma2(M.c[0], x0r, p0r);
    x0i = fma2(M.c[0], x0i, p0i);
    x1r = fma2(M.c[6], x1r, p1r);
    x1i = fma2(M.c[6], x1i, p1i);
}
// y = a x
__device__ __forceinline__ void cmul_p(p2 &r, p2 &i, p2 ar, p2 ai, p2 nai) {
    const p2 p = mul2(nai, i), q = mul2(ai, r);
    r = fma2(ar, r, p);
    i = fma2(ar, i, q);
}
// y = a own + b other
__device__ __forceinline__ void own_p(p2 &r, p2 &i, p2 orr, p2 oi, p2 ar, p2 ai, p2 nai, p2 br, p2 bi, p2 nbi) {
    const p2 p = fma2(nai, i, fma2(br, orr, mul2(nbi, oi)));
    const p2 q = fma2(ai, r, fma2(br, oi, mul2(bi, orr)));
    r = fma2(ar, r, p);
    i = fma2(ar, i, q);
}
__device__ __forceinline__ void xchg(p2 &a, p2 &b) { const p2 t = a; a = b; b = t; }
// the high halves of a slot (the amplitude with tile bit 0 set), for ops under a control on tile bit 0
struct HalvesP {
    float rl, rh, il, ih;
    __device__ __forceinline__ HalvesP(p2 r, p2 i) {
        unpk(r, rl, rh);
        unpk(i, il, ih);
    }
    __device__ __forceinline__ void put(p2 &r, p2 &i, float yr, float yi) const {
        r = pk(rl, yr);
        i = pk(il, yi);
    }
};
// exchange the high halves of a and b
__device__ __forceinline__ void xchg_hi(p2 &a, p2 &b) {
    float al, ah, bl, bh;
    unpk(a, al, ah);
    unpk(b, bl, bh);
    a = pk(al, bh);
    b = pk(bl, ah);
}

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
__device__ __forceinline__ p2 shfl_p(p2 a, int xm) {
    float lo, hi;
    unpk(a, lo, hi);
    lo = __shfl_xor_sync(0xffffffffu, lo, xm);
    hi = __shfl_xor_sync(0xffffffffu, hi, xm);
    return pk(lo, hi);
}
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

// One phase of a tile in shared memory: read the thread's 2^RB slots in the phase's layout, apply ops
// [op_begin, op_end), write them back. PH is any phase record with reg_bits / lane_lo / lane_bits /
// warp_bits; swz: the tile is stored swizzled. split_in / split_out: the slots hold (re0, re1, im0, im1),
// the in-tile order between two phases (the two registers as they are), instead of the state's interleaved
// order (first phase in, last phase out).
template <int NV, int RB, int WB, class PH>
__device__ __forceinline__ void run_phase(float2 *tile, const PH &Q, const QsvIOp *ops, int op_begin, int op_end,
                                          int lane, int warp, bool swz = false, bool split_in = false,
                                          bool split_out = false) {
    uint32_t tb = ((uint32_t)(lane & 1) << Q.lane_lo[0]) | ((uint32_t)((lane >> 1) & 1) << Q.lane_lo[1]) |
                  ((uint32_t)((lane >> 2) & 1) << Q.lane_lo[2]) | ((uint32_t)((lane >> 3) & 1) << Q.lane_bits[0]) |
                  ((uint32_t)((lane >> 4) & 1) << Q.lane_bits[1]);
#pragma unroll
    for (int w = 0; w < WB; w++) tb |= (uint32_t)((warp >> w) & 1) << Q.warp_bits[w];
    // shared-memory positions: base and register offsets swizzle separately (swz128 is linear over XOR)
    const uint32_t base = swz ? swz128(tb) : tb;
    uint32_t rbit[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) rbit[r] = swz ? swz128(1u << Q.reg_bits[r]) : 1u << Q.reg_bits[r];
    auto addr = [&](int r) -> uint32_t {
        uint32_t o = base;
#pragma unroll
        for (int q = 0; q < RB; q++)
            if ((r >> q) & 1) o ^= rbit[q];
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
        for (int r = 0; r < NV; r++) {
            const float4 v = *reinterpret_cast<const float4 *>(tile + addr(r));
            R[r] = pk(v.x, v.z);
            I[r] = pk(v.y, v.w);
        }
    }
    if (op_begin < op_end) {
        // zero, but not known to be the same in all lanes: the coefficients are read into ordinary registers
        // (read at a warp-uniform address they went through uniform registers, 24 moves per op)
        uint32_t vary;
        asm volatile("mov.u32 %0, %%laneid;" : "=r"(vary));
        vary >>= 5;
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
        for (int r = 0; r < NV; r++) {
            float4 v;
            unpk(R[r], v.x, v.z);
            unpk(I[r], v.y, v.w);
            *reinterpret_cast<float4 *>(tile + addr(r)) = v;
        }
    }
}

}  // namespace dev
}  // namespace qsv
