// qsv_sweep_d.cu -- complex128 sweeps: the pass engine on FP64 states with FP64 matrices (sm_100a).
//
// No reference counterpart (the FPGA engine is complex64 only); this is the on-GPU FP64 path of the
// precision study (a 32-qubit complex128 state is 64 GiB). Same sweep plans, addressing and staging
// pipeline as the complex64 engine (qsv_sweep_body.cuh), with one 16-byte amplitude per thread slot: tile
// bits 0-2 are lane bits 0-2 (with the swizzled layout any of bits 0-5 can be register bits), two chosen
// tile bits are lane bits 3-4, three are register bits (8 amplitudes per thread) and the other kw - 8 are warp
// bits (windows of at most 12 qubits: 3 x 64 KiB buffers).
// What bounds it: staging first. A window of short runs staged with one bulk copy per run (256 copies of
// 256 bytes per 64 KiB tile each way) moved 0.9 TB/s whatever its ops; with one tensor-map box per tile the
// same sweeps are bound by their ops. Those run in one tight loop per op variant and slot over all of a
// thread's pairs, coefficients in registers (a class test per pair cost as much as the arithmetic).
// A 27-qubit random-layer circuit with Toffolis, depth 8 (41 sweeps, HBM floor 27 ms): 189 ms before, 107 ms
// with the loops, 53 ms with the tensor maps and swizzled layouts as well, 41 ms with expanded records and 16 warps.
// Every pair update is the canonical fused-multiply-add chain in double precision
//   y0.re = fma(m00.re, x0.re, fma(-m00.im, x0.im, fma(m01.re, x1.re, -(m01.im * x1.im))))  (etc.)
// which the CPU oracle's complex128 engine writes identically, so results agree value for value; the
// diagonal / swap / identity forms skip exact-zero terms only.
#include <cuda.h>
#include <cuda_runtime.h>

#include "qsv_device.cuh"
#include "qsv_iop.h"
#include "qsv_launch.h"
#include "qsv_packed.cuh"
#include "qsv_planner.h"
#include "qsv_sweep_body.cuh"

namespace qsv {
namespace dev {

__device__ __forceinline__ void lin_own_d(double &yr, double &yi, double ar, double ai, double br, double bi,
                                          double owr, double owi, double otr, double oti) {
    yr = fma(ar, owr, fma(-ai, owi, fma(br, otr, -__dmul_rn(bi, oti))));
    yi = fma(ar, owi, fma(ai, owr, fma(br, oti, __dmul_rn(bi, otr))));
}

// ---------------------------------------------------------------- ops by path (qsv_iop.h)
// One tight loop over the thread's pairs per path. Each loop computes the partial sums of all four outputs of a pair
// first and the final multiply-adds last, so that every final is the last use of the input it replaces and can be
// written over its registers.
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
__device__ __forceinline__ MatD load_mat_d(const double *m) {
    MatD M;
    const double2 *v = reinterpret_cast<const double2 *>(m);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const double2 x = v[e];
        M.m[2 * e] = x.x;
        M.m[2 * e + 1] = x.y;
    }
    return M;
}

#define QSV_PAIRS for (int r = 0; r < NV; r++) if (!(r & B))
#define QSV_SEL if ((sel >> r) & 1u)
template <int NV, int RBIT, bool R0>
__device__ __forceinline__ void dense_op_d(double2 (&A)[NV], const MatD &M) {
    constexpr int B = 1 << RBIT;
#pragma unroll
    QSV_PAIRS {
        if (R0) dense_r0_d(A[r], A[r | B], M);
        else dense_d(A[r], A[r | B], M);
    }
}
template <int NV, int RBIT>
__device__ __forceinline__ void diag_op_d(double2 (&A)[NV], const MatD &M) {
    constexpr int B = 1 << RBIT;
#pragma unroll
    QSV_PAIRS { cmul_d(A[r], M.m[0], M.m[1]); cmul_d(A[r | B], M.m[6], M.m[7]); }
}
template <int NV, int RBIT>
__device__ __forceinline__ void cdense_op_d(double2 (&A)[NV], const MatD &M, uint32_t sel, bool tok) {
    constexpr int B = 1 << RBIT;
    if (tok) {
#pragma unroll
        QSV_PAIRS QSV_SEL dense_d(A[r], A[r | B], M);
    }
}
template <int NV, int RBIT>
__device__ __forceinline__ void swap_op_d(double2 (&A)[NV], uint32_t sel, bool tok) {
    constexpr int B = 1 << RBIT;
    if (tok) {
#pragma unroll
        QSV_PAIRS QSV_SEL { const double2 t = A[r]; A[r] = A[r | B]; A[r | B] = t; }
    }
}
template <int NV, int RBIT>
__device__ __forceinline__ void mux_op_d(double2 (&A)[NV], const MatD &M, const double *other, uint32_t sel, bool tok) {
    constexpr int B = 1 << RBIT;
    cdense_op_d<NV, RBIT>(A, M, sel, tok);
    const MatD N = load_mat_d(other);
    if (!tok) sel = 0;
#pragma unroll
    QSV_PAIRS if (!((sel >> r) & 1u)) dense_d(A[r], A[r | B], N);
}
// a factor on the slots whose index has every bit of RM
template <int NV, int RM>
__device__ __forceinline__ void phase_slots_d(double2 (&A)[NV], double ar, double ai) {
#pragma unroll
    for (int r = 0; r < NV; r++)
        if ((r & RM) == RM) cmul_d(A[r], ar, ai);
}
template <int NV>
__device__ __forceinline__ void phase_op_d(double2 (&A)[NV], double ar, double ai, uint32_t rm) {
    static_assert(NV == 8, "one case per mask");
    if (rm == 0) phase_slots_d<NV, 0>(A, ar, ai);
    else if (rm == 1) phase_slots_d<NV, 1>(A, ar, ai);
    else if (rm == 2) phase_slots_d<NV, 2>(A, ar, ai);
    else if (rm == 3) phase_slots_d<NV, 3>(A, ar, ai);
    else if (rm == 4) phase_slots_d<NV, 4>(A, ar, ai);
    else if (rm == 5) phase_slots_d<NV, 5>(A, ar, ai);
    else if (rm == 6) phase_slots_d<NV, 6>(A, ar, ai);
    else phase_slots_d<NV, 7>(A, ar, ai);
}

// Lane-bit target: each thread computes its own amplitudes as a*own + b*other, the other from the partner lane, with
// (a, b) = (m00, m01) on the bit-0 side and (m11, m10) on the bit-1 side. Controls on register bits are uniform
// (slots outside them are left alone, no exchange); for controls elsewhere every lane takes part in the exchange
// and keeps its amplitude where they do not hold.
struct OwnD {
    double ar, ai, br, bi;
};
__device__ __forceinline__ OwnD lane_own_d(const MatD &M, bool mine) {
    return OwnD{mine ? M.m[6] : M.m[0], mine ? M.m[7] : M.m[1], mine ? M.m[4] : M.m[2], mine ? M.m[5] : M.m[3]};
}
__device__ __forceinline__ double2 shfl_d(const double2 &x, int xm) {
    double2 o;
    o.x = __shfl_xor_sync(0xffffffffu, x.x, xm);
    o.y = __shfl_xor_sync(0xffffffffu, x.y, xm);
    return o;
}
template <int NV>
__device__ __forceinline__ void lane_dense_d(double2 (&A)[NV], const OwnD &M, int xm, uint32_t sel, bool keep) {
#pragma unroll
    for (int r = 0; r < NV; r++)
        QSV_SEL {
            const double2 o = shfl_d(A[r], xm);
            double2 y;
            lin_own_d(y.x, y.y, M.ar, M.ai, M.br, M.bi, A[r].x, A[r].y, o.x, o.y);
            A[r].x = keep ? A[r].x : y.x;
            A[r].y = keep ? A[r].y : y.y;
        }
}
template <int NV>
__device__ __forceinline__ void lane_op_d(double2 (&A)[NV], uint32_t path, uint32_t sel, uint32_t aux, const MatD &M,
                                          const double *other, bool tok, int lane) {
    const int xm = (int)(aux & 31u);
    const bool mine = lane & xm;
    if (path == QSV_P_LANE_SWAP) {
#pragma unroll
        for (int r = 0; r < NV; r++)
            QSV_SEL {
                const double2 o = shfl_d(A[r], xm);
                A[r].x = tok ? o.x : A[r].x;
                A[r].y = tok ? o.y : A[r].y;
            }
        return;
    }
    const OwnD S = lane_own_d(M, mine);
    if (path == QSV_P_LANE_DENSE) {
        lane_dense_d<NV>(A, S, xm, 0xffffffffu, false);
    } else if (path == QSV_P_LANE_CDENSE) {
        lane_dense_d<NV>(A, S, xm, sel, !tok);
    } else {                                     // QSV_P_LANE_MUX
        const OwnD N = lane_own_d(load_mat_d(other), mine);
        const OwnD T = {tok ? S.ar : N.ar, tok ? S.ai : N.ai, tok ? S.br : N.br, tok ? S.bi : N.bi};
        lane_dense_d<NV>(A, T, xm, sel, false);
        lane_dense_d<NV>(A, N, xm, ~sel, false);
    }
}
#undef QSV_PAIRS
#undef QSV_SEL

// The applied matrix is loaded before the path's branches so that both latencies overlap; vary: 0, unknown to be the
// same in all lanes (lane_zero).
template <int NV>
__device__ __forceinline__ void apply_op_d(const uint4 &h, const QsvIOpD *op, double2 (&A)[NV], uint32_t tb, int lane,
                                           uint32_t vary) {
    const bool tok = (tb & h.x) == h.x;
    const uint32_t path = h.y, sel = h.z, aux = h.w;
    const MatD M = load_mat_d((op + vary)->a);
#define QSV_BY_RBIT(G, CALL)                                        \
    if (path == 4 * G) { constexpr int RBIT = 0; CALL; }            \
    else if (path == 4 * G + 1) { constexpr int RBIT = 1; CALL; }   \
    else { constexpr int RBIT = 2; CALL; }
    if (path < 4 * (QSV_G_DENSE_R0 + 1)) {
        QSV_BY_RBIT(QSV_G_DENSE_R0, (dense_op_d<NV, RBIT, true>(A, M)))
    } else if (path < 4 * (QSV_G_DENSE + 1)) {
        QSV_BY_RBIT(QSV_G_DENSE, (dense_op_d<NV, RBIT, false>(A, M)))
    } else if (path == 4 * QSV_G_PHASE) {
        if (tok) phase_op_d<NV>(A, M.m[6], M.m[7], aux);
    } else if (path < 4 * (QSV_G_SWAP + 1)) {
        QSV_BY_RBIT(QSV_G_SWAP, (swap_op_d<NV, RBIT>(A, sel, tok)))
    } else if (path >= QSV_P_LANE_DENSE) {
        if (path <= QSV_P_LANE_MUX) {
            lane_op_d<NV>(A, path, sel, aux, M, op->b, tok, lane);
        } else if (path == QSV_P_BASE_DIAG) {
            const bool one = tb & aux;
            phase_slots_d<NV, 0>(A, one ? M.m[6] : M.m[0], one ? M.m[7] : M.m[1]);
        }
    } else if (path < 4 * (QSV_G_DIAG + 1)) {
        QSV_BY_RBIT(QSV_G_DIAG, (diag_op_d<NV, RBIT>(A, M)))
    } else if (path < 4 * (QSV_G_CDENSE + 1)) {
        QSV_BY_RBIT(QSV_G_CDENSE, (cdense_op_d<NV, RBIT>(A, M, sel, tok)))
    } else {
        QSV_BY_RBIT(QSV_G_MUX, (mux_op_d<NV, RBIT>(A, M, op->b, sel, tok)))
    }
#undef QSV_BY_RBIT
}

// the complex128 interpreter body: per phase, each thread loads its 2^RB amplitudes, applies the phase's
// ops and stores them back
struct InterpBodyD {
    using Amp = double2;
    static constexpr int kHalfBits = 0;
    static constexpr bool kSmemOps = true;
    using IOp = QsvIOpD;
    // the expanded table follows the raw one (whose size keeps it on a 16-byte boundary)
    static_assert(sizeof(QsvOpD) * QSV_MAX_SWEEP_OPS % 16 == 0, "expanded records are read as 16-byte vectors");
    static __device__ __forceinline__ QsvIOpD *table(const QsvOpD *sops) {
        return reinterpret_cast<QsvIOpD *>(const_cast<QsvOpD *>(sops) + QSV_MAX_SWEEP_OPS);
    }
    // the phase tables take the raw ops' place
    static __device__ __forceinline__ PhaseTab *phase_table(const QsvOpD *sops) {
        static_assert(sizeof(PhaseTab) * QSV_MAX_PHASES <= sizeof(QsvOpD) * QSV_MAX_SWEEP_OPS, "phase tables fit");
        return reinterpret_cast<PhaseTab *>(const_cast<QsvOpD *>(sops));
    }
    template <int RB, int WB>
    static __device__ __forceinline__ void expand_phases(const QsvOpD *sops, const QsvSweepD &P, int tid, int nthreads) {
        // a swizzled tile holds amplitude x at x ^ ((x >> 3) & 7) (16-byte chunks, rows of 8)
        const uint32_t sw = P.swz ? 7u : 0u;
        PhaseTab *pt = phase_table(sops);
        for (int i = tid; i < P.nphases * 52; i += nthreads) {
            const int ph = i / 52, e = i - ph * 52;
            reinterpret_cast<uint32_t *>(pt + ph)[e] =
                phase_entry(P.phases[ph], e, RB, WB, [&](uint32_t x) { return x ^ ((x >> 3) & sw); });
        }
    }
    template <int NV>
    static __device__ __forceinline__ void expand(const QsvOpD *sops, int nops, int tid, int nthreads) {
        QsvIOpD *t = table(sops);
        for (int i = tid; i < nops * 17; i += nthreads) {        // 16 coefficients and the header of each op
            const int o = i / 17, e = i - o * 17;
            const QsvOpD &op = sops[o];
            if (e == 16) iop_header(op, NV, t[o]);
            else if (e < 8) t[o].a[e] = op.kind == QSV_K_UNI ? op.m0[e] : op.m1[e];
            else t[o].b[e - 8] = op.m0[e - 8];
        }
    }
    template <int NV, int RB, int WB>
    static __device__ __forceinline__ void tile(double2 *tile, const QsvSweepD &P, const QsvOpD *sops, int lane,
                                                int warp, int bar) {
        constexpr int NC = 1 << (5 + WB);
        const QsvIOpD *ops = table(sops);
        const PhaseTab *pt = phase_table(sops);
        const uint32_t vary = lane_zero();
        for (int ph = 0; ph < P.nphases; ph++) {
            if (ph > 0) named_bar_sync(bar, NC);
            const QsvPhase &Q = P.phases[ph];
            const uint32_t v = pt[ph].lane[lane] ^ pt[ph].warp[warp];
            const uint32_t tb = v & 0xffffu, base = v >> 16;
            const uint4 rv = *reinterpret_cast<const uint4 *>(pt[ph].rbit);
            const uint32_t rbit[4] = {rv.x, rv.y, rv.z, rv.w};
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
            const int ob = Q.op_begin, oe = Q.op_end;
            if (ob < oe) {
                uint4 next = *reinterpret_cast<const uint4 *>(ops + ob);     // the next op's header, read ahead
                for (int o = ob; o < oe; o++) {
                    const uint4 h = next;
                    if (o + 1 < oe) next = *reinterpret_cast<const uint4 *>(ops + o + 1);
                    apply_op_d<NV>(h, ops + o, A, tb, lane, vary);
                }
            }
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
        case 12: return dev::launch_c128_t<12, 3, 4, 3>(state, sw, nsm, status, stream);
        case 11: return dev::launch_c128_t<11, 3, 3, 3>(state, sw, nsm, status, stream);
        case 10: return dev::launch_c128_t<10, 3, 2, 3>(state, sw, nsm, status, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace qsv
