// qsv_sweep_d.cu -- complex128 sweeps: the pass engine on FP64 states with FP64 matrices (sm_100a).
//
// No reference counterpart (the FPGA engine is complex64 only); this is the on-GPU FP64 path of the
// precision study (a 32-qubit complex128 state is 64 GiB). Same sweep plans, addressing and staging
// pipeline as the complex64 engine (qsv_sweep_body.cuh), with one 16-byte amplitude per thread slot: tile
// bits 0-2 are lane bits 0-2 (with the swizzled layout any of bits 0-5 can be register bits), two chosen
// tile bits are lane bits 3-4, four are register bits and the rest warp bits (windows of at most 12 qubits:
// 3 x 64 KiB buffers).
// What bounds it: staging first. A window of short runs staged with one bulk copy per run (256 copies of
// 256 bytes per 64 KiB tile each way) moved 0.9 TB/s whatever its ops; with one tensor-map box per tile the
// same sweeps are bound by their ops. Those run in one tight loop per op variant and slot over all of a
// thread's pairs, coefficients in registers (a class test per pair cost as much as the arithmetic).
// A 27-qubit random-layer circuit with Toffolis, depth 8 (41 sweeps, HBM floor 27 ms): 189 ms before, 107 ms
// with the loops, 53 ms with the tensor maps and swizzled layouts as well.
// Every pair update is the canonical fused-multiply-add chain in double precision
//   y0.re = fma(m00.re, x0.re, fma(-m00.im, x0.im, fma(m01.re, x1.re, -(m01.im * x1.im))))  (etc.)
// which the CPU oracle's complex128 engine writes identically, so results agree value for value; the
// diagonal / swap / identity forms skip exact-zero terms only.
#include <cuda.h>
#include <cuda_runtime.h>

#include "qsv_device.cuh"
#include "qsv_launch.h"
#include "qsv_planner.h"
#include "qsv_sweep_body.cuh"

namespace qsv {
namespace dev {

__device__ __forceinline__ void lin_own_d(double &yr, double &yi, double ar, double ai, double br, double bi,
                                          double owr, double owi, double otr, double oti) {
    yr = fma(ar, owr, fma(-ai, owi, fma(br, otr, -__dmul_rn(bi, oti))));
    yi = fma(ar, owi, fma(ai, owr, fma(br, oti, __dmul_rn(bi, otr))));
}

// ---------------------------------------------------------------- ops by target slot
// One uniform dispatch per op selects a tight loop over the thread's pairs, coefficients in registers. Each
// loop computes the partial sums of all four outputs of a pair first and the final multiply-adds last, so
// that every final is the last use of the input it replaces and can be written over its registers.
struct MatD {
    double m[8];
};
__device__ __forceinline__ void dense_d(double2 &x0, double2 &x1, const MatD &M) {
    const double *m = M.m;
    const double p0r = fma(-m[1], x0.y, fma(m[2], x1.x, -__dmul_rn(m[3], x1.y)));
    const double p0i = fma(m[1], x0.x, fma(m[2], x1.y, __dmul_rn(m[3], x1.x)));
    const double p1r = fma(-m[7], x1.y, fma(m[4], x0.x, -__dmul_rn(m[5], x0.y)));
    const double p1i = fma(m[7], x1.x, fma(m[4], x0.y, __dmul_rn(m[5], x0.x)));
    x0.x = fma(m[0], x0.x, p0r);
    x0.y = fma(m[0], x0.y, p0i);
    x1.x = fma(m[6], x1.x, p1r);
    x1.y = fma(m[6], x1.y, p1i);
}
// dense with m00 real (every U3): its two m00.im terms are exact zeros and are skipped
__device__ __forceinline__ void dense_r0_d(double2 &x0, double2 &x1, const MatD &M) {
    const double *m = M.m;
    const double p0r = fma(m[2], x1.x, -__dmul_rn(m[3], x1.y));
    const double p0i = fma(m[2], x1.y, __dmul_rn(m[3], x1.x));
    const double p1r = fma(-m[7], x1.y, fma(m[4], x0.x, -__dmul_rn(m[5], x0.y)));
    const double p1i = fma(m[7], x1.x, fma(m[4], x0.y, __dmul_rn(m[5], x0.x)));
    x0.x = fma(m[0], x0.x, p0r);
    x0.y = fma(m[0], x0.y, p0i);
    x1.x = fma(m[6], x1.x, p1r);
    x1.y = fma(m[6], x1.y, p1i);
}
__device__ __forceinline__ void cmul_d(double2 &x, double ar, double ai) {
    const double p = -__dmul_rn(ai, x.y), q = __dmul_rn(ai, x.x);
    x.x = fma(ar, x.x, p);
    x.y = fma(ar, x.y, q);
}
__device__ __forceinline__ MatD load_mat(const double *m) {
    MatD M;
#pragma unroll
    for (int e = 0; e < 8; e++) M.m[e] = m[e];
    return M;
}

// Register-bit target RBIT: pairs (r, r | 2^RBIT). tok: the controls outside the register bits hold.
template <int NV, int RBIT>
__device__ __forceinline__ void reg_op_d(double2 (&A)[NV], const QsvOpD &op, bool tok) {
    constexpr int B = 1 << RBIT;
    const int cm = op.cm_reg;
#define QSV_FOR_PAIRS for (int r = 0; r < NV; r++) if (!(r & B))
    switch (op.variant) {
        case QSV_V_UNI_DENSE: {
            const MatD M = load_mat(op.m0);
            if (op.r00) {
#pragma unroll
                QSV_FOR_PAIRS dense_r0_d(A[r], A[r | B], M);
            } else {
#pragma unroll
                QSV_FOR_PAIRS dense_d(A[r], A[r | B], M);
            }
            break;
        }
        case QSV_V_UNI_SWAP:
        case QSV_V_CTRL_SWAP:
        case QSV_V_CTRL_SWAP_SEL:
            // lanes of a warp whose controls do not hold sit the exchange out
            if (tok) {
#pragma unroll
                QSV_FOR_PAIRS if ((r & cm) == cm) { const double2 t = A[r]; A[r] = A[r | B]; A[r | B] = t; }
            }
            break;
        case QSV_V_CTRL_DENSE:
        case QSV_V_CTRL_DENSE_SEL: {
            const MatD M = load_mat(op.m1);
            if (tok) {
#pragma unroll
                QSV_FOR_PAIRS if ((r & cm) == cm) dense_d(A[r], A[r | B], M);
            }
            break;
        }
        case QSV_V_MUX: {
            const double *m0 = op.m0, *m1 = op.m1;
#pragma unroll
            QSV_FOR_PAIRS {
                const bool s = tok && (r & cm) == cm;
                MatD M;
#pragma unroll
                for (int e = 0; e < 8; e++) M.m[e] = s ? m1[e] : m0[e];
                dense_d(A[r], A[r | B], M);
            }
            break;
        }
        default: break;
    }
#undef QSV_FOR_PAIRS
}

// Lane-bit target: each thread computes its own amplitudes as a*own + b*other, the other from the partner
// lane, with (a, b) = (m00, m01) on the bit-0 side and (m11, m10) on the bit-1 side. Controls on register
// bits are uniform (pairs outside them are left alone, no exchange); for controls elsewhere every lane
// takes part in the exchange and keeps its amplitude where they do not hold.
template <int NV>
__device__ __forceinline__ void lane_op_d(double2 (&A)[NV], const QsvOpD &op, bool tok, int lanebit, int lane) {
    const int xm = 1 << lanebit;
    const bool mine = (lane >> lanebit) & 1;
    const int cm = op.cm_reg;
    auto partner = [&](const double2 &x) {
        double2 o;
        o.x = __shfl_xor_sync(0xffffffffu, x.x, xm);
        o.y = __shfl_xor_sync(0xffffffffu, x.y, xm);
        return o;
    };
    switch (op.variant) {
        case QSV_V_UNI_SWAP:
        case QSV_V_CTRL_SWAP:
        case QSV_V_CTRL_SWAP_SEL:
#pragma unroll
            for (int r = 0; r < NV; r++)
                if ((r & cm) == cm) {
                    const double2 o = partner(A[r]);
                    if (tok) A[r] = o;
                }
            break;
        case QSV_V_UNI_DENSE:
        case QSV_V_CTRL_DENSE:
        case QSV_V_CTRL_DENSE_SEL: {
            const double *m = op.kind == QSV_K_UNI ? op.m0 : op.m1;
            const double ar = m[mine ? 6 : 0], ai = m[mine ? 7 : 1], br = m[mine ? 4 : 2], bi = m[mine ? 5 : 3];
#pragma unroll
            for (int r = 0; r < NV; r++)
                if ((r & cm) == cm) {
                    const double2 o = partner(A[r]);
                    double2 y;
                    lin_own_d(y.x, y.y, ar, ai, br, bi, A[r].x, A[r].y, o.x, o.y);
                    if (tok) A[r] = y;
                }
            break;
        }
        case QSV_V_MUX: {
#pragma unroll
            for (int r = 0; r < NV; r++) {
                const double *m = tok && (r & cm) == cm ? op.m1 : op.m0;
                const double2 o = partner(A[r]);
                double2 y;
                lin_own_d(y.x, y.y, m[mine ? 6 : 0], m[mine ? 7 : 1], m[mine ? 4 : 2], m[mine ? 5 : 3], A[r].x, A[r].y,
                          o.x, o.y);
                A[r] = y;
            }
            break;
        }
        default: break;
    }
}

// Diagonal ops act on each amplitude alone, so their target may sit anywhere. With the target in the thread
// (slots differ) or not (the thread's bit decides), diag(a, b) is a factor on the slots without and one on
// the slots with it; controlled ops are diag(1, d): a factor on the slots with target and controls set.
template <int NV, int RM>
__device__ __forceinline__ void phase_slots_d(double2 (&A)[NV], double ar, double ai) {
#pragma unroll
    for (int r = 0; r < NV; r++)
        if ((r & RM) == RM) cmul_d(A[r], ar, ai);
}
template <int NV, int RB>
__device__ __forceinline__ void diag_op_d(double2 (&A)[NV], const QsvOpD &op, uint32_t tb) {
    const int slot = op.slot;
    const bool reg = slot < QSV_SLOT_BASE, uni = op.kind == QSV_K_UNI;
    int rm = op.cm_reg;
    uint32_t thr = op.cm_thr;
    if (reg) rm |= 1 << (slot - QSV_SLOT_REG0);
    else thr |= 1u << op.tbit;
    const bool on = (tb & thr) == thr;
    const double *m = uni ? op.m0 : op.m1;
    if (uni && op.cls == QSV_M_DIAG && (reg || !on)) {       // the amplitudes with the target bit clear
        const double ar = m[0], ai = m[1];
        switch (reg ? rm : 0) {
            case 0: phase_slots_d<NV, 0>(A, ar, ai); break;
            case 1:
#pragma unroll
                for (int r = 0; r < NV; r++) if (!(r & 1)) cmul_d(A[r], ar, ai);
                break;
            case 2:
#pragma unroll
                for (int r = 0; r < NV; r++) if (!(r & 2)) cmul_d(A[r], ar, ai);
                break;
            case 4:
#pragma unroll
                for (int r = 0; r < NV; r++) if (!(r & 4)) cmul_d(A[r], ar, ai);
                break;
            default:
#pragma unroll
                for (int r = 0; r < NV; r++) if (!(r & 8)) cmul_d(A[r], ar, ai);
                break;
        }
    }
    if (!on) return;
    const double br = m[6], bi = m[7];
    switch (rm) {
        case 0: phase_slots_d<NV, 0>(A, br, bi); break;
        case 1: phase_slots_d<NV, 1>(A, br, bi); break;
        case 2: phase_slots_d<NV, 2>(A, br, bi); break;
        case 3: phase_slots_d<NV, 3>(A, br, bi); break;
        case 4: phase_slots_d<NV, 4>(A, br, bi); break;
        case 5: phase_slots_d<NV, 5>(A, br, bi); break;
        case 6: phase_slots_d<NV, 6>(A, br, bi); break;
        case 8: phase_slots_d<NV, 8>(A, br, bi); break;
        case 9: phase_slots_d<NV, 9>(A, br, bi); break;
        case 10: phase_slots_d<NV, 10>(A, br, bi); break;
        case 12: phase_slots_d<NV, 12>(A, br, bi); break;
        default:
#pragma unroll
            for (int r = 7; r < NV; r++)
                if ((r & rm) == rm) cmul_d(A[r], br, bi);
            break;
    }
}

template <int NV, int RB>
__device__ __forceinline__ void apply_op_d(const QsvOpD &op, double2 (&A)[NV], uint32_t tb, int lane) {
    const int slot = op.slot, v = op.variant;
    if (v == QSV_V_UNI_DIAG || v == QSV_V_CTRL_DIAG1 || v == QSV_V_CTRL_DIAG1_SEL) {
        diag_op_d<NV, RB>(A, op, tb);
        return;
    }
    const bool tok = (tb & op.cm_thr) == op.cm_thr;
    switch (slot) {
        case QSV_SLOT_REG0 + 0: reg_op_d<NV, 0>(A, op, tok); break;
        case QSV_SLOT_REG0 + 1: if constexpr (RB > 1) reg_op_d<NV, (RB > 1 ? 1 : 0)>(A, op, tok); break;
        case QSV_SLOT_REG0 + 2: if constexpr (RB > 2) reg_op_d<NV, (RB > 2 ? 2 : 0)>(A, op, tok); break;
        case QSV_SLOT_REG0 + 3: if constexpr (RB > 3) reg_op_d<NV, (RB > 3 ? 3 : 0)>(A, op, tok); break;
        default: lane_op_d<NV>(A, op, tok, slot - QSV_SLOT_LANE0, lane); break;
    }
}

// the complex128 interpreter body: per phase, each thread loads its 2^RB amplitudes, applies the phase's
// ops and stores them back
struct InterpBodyD {
    using Amp = double2;
    static constexpr int kHalfBits = 0;
    static constexpr bool kSmemOps = true;
    template <int NV, int RB, int WB>
    static __device__ __forceinline__ void tile(double2 *tile, const QsvSweepD &P, const QsvOpD *sops, int lane,
                                                int warp, int bar) {
        constexpr int NC = 1 << (5 + WB);
        for (int ph = 0; ph < P.nphases; ph++) {
            if (ph > 0) named_bar_sync(bar, NC);
            const QsvPhase &Q = P.phases[ph];
            uint32_t tb = ((uint32_t)(lane & 1) << Q.lane_lo[0]) | ((uint32_t)((lane >> 1) & 1) << Q.lane_lo[1]) |
                          ((uint32_t)((lane >> 2) & 1) << Q.lane_lo[2]) |
                          ((uint32_t)((lane >> 3) & 1) << Q.lane_bits[0]) |
                          ((uint32_t)((lane >> 4) & 1) << Q.lane_bits[1]);
#pragma unroll
            for (int w = 0; w < WB; w++) tb |= (uint32_t)((warp >> w) & 1) << Q.warp_bits[w];
            // slot r at tile index tb | bits of r, a swizzled tile holding amplitude x at x ^ ((x >> 3) & 7)
            // (16-byte chunks, rows of 8): linear over XOR, so base and register offsets swizzle separately
            const uint32_t sw = P.swz ? 7u : 0u;
            const uint32_t base = tb ^ ((tb >> 3) & sw);
            uint32_t rbit[RB];
#pragma unroll
            for (int q = 0; q < RB; q++) {
                const uint32_t x = 1u << Q.reg_bits[q];
                rbit[q] = x ^ ((x >> 3) & sw);
            }
            auto pos = [&](int r) -> uint32_t {
                uint32_t o = base;
#pragma unroll
                for (int q = 0; q < RB; q++)
                    if ((r >> q) & 1) o ^= rbit[q];
                return o;
            };
            double2 A[NV];
#pragma unroll
            for (int r = 0; r < NV; r++) A[r] = tile[pos(r)];
            for (int o = Q.op_begin; o < Q.op_end; o++) apply_op_d<NV, RB>(sops[o], A, tb, lane);
#pragma unroll
            for (int r = 0; r < NV; r++) tile[pos(r)] = A[r];
        }
    }
};

template <int KW, int RB, int WB, int S>
__global__ void __launch_bounds__((1 << (5 + WB)) + 32, 1)
    sweep_kernel_c128(double2 *__restrict__ state, const __grid_constant__ QsvSweepD P,
                      const __grid_constant__ CUtensorMap tmap, int *status) {
    sweep_pipeline<KW, RB, WB, S, 1, InterpBodyD, QsvSweepD>(state, P, &tmap, status);
}

cudaError_t make_tmap(CUtensorMap *map, double2 *state, const QsvSweepD &sw);

template <int KW, int RB, int WB, int S>
static cudaError_t launch_c128_t(double2 *state, const QsvSweepD &sw, int nsm, int *status, cudaStream_t stream) {
    constexpr int NT = (1 << (5 + WB)) + 32;
    const size_t smem = sweep_smem_bytes<KW, S, InterpBodyD, QsvSweepD>();
    static int configured_dev = -1;     // attribute set once per device (under the engine's launch lock)
    static int per_sm = 1;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (configured_dev != dev) {
        e = cudaFuncSetAttribute(sweep_kernel_c128<KW, RB, WB, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sweep_kernel_c128<KW, RB, WB, S>, NT, smem);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
        configured_dev = dev;
    }
    alignas(64) CUtensorMap map;
    e = make_tmap(&map, state, sw);
    if (e != cudaSuccess) return e;
    int64_t grid = (int64_t)nsm * per_sm;
    if (grid > sw.ntiles) grid = sw.ntiles;
    return launch_behind(sweep_kernel_c128<KW, RB, WB, S>, (unsigned)grid, NT, smem, stream, state, sw, map, status);
}

}  // namespace dev

cudaError_t status_word_ptr(int **out);

cudaError_t launch_sweep_c128(double2 *state, const QsvSweepD &sw, int nsm, cudaStream_t stream) {
    int *status = nullptr;
    cudaError_t e = status_word_ptr(&status);
    if (e != cudaSuccess) return e;
    switch (sw.kw) {
        case 12: return dev::launch_c128_t<12, 4, 3, 3>(state, sw, nsm, status, stream);
        case 11: return dev::launch_c128_t<11, 4, 2, 3>(state, sw, nsm, status, stream);
        case 10: return dev::launch_c128_t<10, 4, 1, 3>(state, sw, nsm, status, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace qsv
