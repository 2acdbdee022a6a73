// qsv_aux.cu -- the remap (qubit permutation) kernel, |0..0> init, FP64 reductions and the Born sampler.
//
// remap: replaces the reference's exchange path -- sv_swap (kernels/sv/sv_swap.cpp:10-39) for
// bank<->local transpositions and the host permutes of host/sv/runtime.py:261-268 -- with one in-HBM
// sweep for an arbitrary bit permutation perm[new] = old (host/sv/model.py:74-78). Each CTA moves 32 KiB tiles
// that are contiguous in 512-byte runs on both sides: the tile holds the lowest source bits (coalesced reads) and
// the source bits that land on the lowest destination bits (coalesced writes), padded with the lowest remaining
// source bits; the transpose happens in shared memory.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>
#include <mutex>

#include "qsv_device.cuh"
#include "qsv_reduce.h"

namespace qsv {
namespace dev {

#define REMAP_TB 12                 // most tile bits
#define REMAP_BANK_BITS 5           // a warp's shared-memory accesses vary five tile bits
#define REMAP_THREADS 256

// Everything linear in an index is given bit by bit: the bits of an index select terms that are combined with OR
// (offsets) or XOR (shared-memory positions).
struct RemapParams {
    int nfree;
    uint64_t roff[REMAP_TB];        // source offset of source-ordered tile position bit i
    uint64_t woff[REMAP_TB];        // destination offset of destination-ordered tile position bit i
    uint32_t spin[REMAP_TB];        // shared-memory position of source-ordered bit i
    uint32_t spout[REMAP_TB];       // and of destination-ordered bit i
    uint8_t fx[32];                 // source position of tile number bit i (free source bits, ascending)
    uint8_t fy[32];                 // its destination position
};

// Bit permutation of the state, one HBM read and one write per amplitude. A tile is 2^TB amplitudes that share the
// free bits (the source bits outside the tile); it holds the lowest source bits, so that reads are contiguous in
// runs of 512 bytes, and the source bits that land on the lowest destination bits, so that writes are too (2 x 6 bits
// of complex64, 2 x 5 of complex128). Shared memory holds the tile as 32-bit planes (W = sizeof(A) / 4 words per
// amplitude) at a swizzled position: a warp's stores vary tile bits 0..4 and its loads vary the tile bits of
// destination bits 0..4; the swizzle (host-chosen, linear) moves each such bit above bit 4 onto a low bit the others
// leave free, so both sides hit 32 distinct banks. The loads of the next tile are issued before the stores of the
// current one. What bounds it: how much of HBM's rate scattered runs reach. With runs of 256 bytes (2^11-amplitude
// tiles) and every thread's offsets in registers, a random permutation of 29 qubits took 1.63 ms (0.81 of the
// measured copy rate), of 24 qubits 64 us; now 1.41 ms (0.93) and 48 us, complex128 at 28 qubits 1.70 -> 1.47 ms.
template <class A, int TB>
__global__ void __launch_bounds__(REMAP_THREADS, 3)
    remap_kernel(const A *__restrict__ src, A *__restrict__ dst, const __grid_constant__ RemapParams P) {
    constexpr int TS = 1 << TB;
    constexpr int EPT = TS / REMAP_THREADS;           // amplitudes per thread per tile: position bits 8..TB-1
    constexpr int W = sizeof(A) / 4;
    using Word = uint32_t;
    extern __shared__ Word plane[];                   // W * TS words
    const int t = threadIdx.x, lane = t & 31;
    uint64_t ro = 0, wo = 0;
    uint32_t si = 0, so = 0;
#pragma unroll
    for (int i = 0; i < 8; i++)
        if ((t >> i) & 1) {
            ro |= P.roff[i];
            wo |= P.woff[i];
            si ^= P.spin[i];
            so ^= P.spout[i];
        }
    // the part of an offset that belongs to the thread's e-th amplitude (the same in all threads)
    auto part64 = [](const uint64_t *off, int e) {
        uint64_t o = 0;
#pragma unroll
        for (int k = 0; k < TB - 8; k++)
            if ((e >> k) & 1) o |= off[8 + k];
        return o;
    };
    auto part32 = [](const uint32_t *off, int e) {
        uint32_t o = 0;
#pragma unroll
        for (int k = 0; k < TB - 8; k++)
            if ((e >> k) & 1) o ^= off[8 + k];
        return o;
    };
    // a tile's bases: lane i places bit i of the tile number
    const uint64_t bx = lane < P.nfree ? 1ull << P.fx[lane] : 0, by = lane < P.nfree ? 1ull << P.fy[lane] : 0;
    auto spread = [&](uint32_t T, uint64_t bit) {
        const uint64_t x = (T >> lane) & 1u ? bit : 0;
        return (uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)x) |
               ((uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(x >> 32)) << 32);
    };
    const uint32_t ntiles = 1u << P.nfree;
    uint32_t T = blockIdx.x;
    if (T >= ntiles) return;
    A v[EPT];
    const A *s = src + (spread(T, bx) | ro);
#pragma unroll
    for (int e = 0; e < EPT; e++) v[e] = s[part64(P.roff, e)];
    while (true) {
#pragma unroll
        for (int e = 0; e < EPT; e++) {
            const Word *w = reinterpret_cast<const Word *>(&v[e]);
            const uint32_t at = si ^ part32(P.spin, e);
#pragma unroll
            for (int p = 0; p < W; p++) plane[p * TS + at] = w[p];
        }
        __syncthreads();
        A *d = dst + (spread(T, by) | wo);
        const uint32_t Tn = T + gridDim.x;
        if (Tn < ntiles) {                      // next tile's loads in flight during this tile's stores
            s = src + (spread(Tn, bx) | ro);
#pragma unroll
            for (int e = 0; e < EPT; e++) v[e] = s[part64(P.roff, e)];
        }
#pragma unroll
        for (int e = 0; e < EPT; e++) {
            A a;
            Word *w = reinterpret_cast<Word *>(&a);
            const uint32_t at = so ^ part32(P.spout, e);
#pragma unroll
            for (int p = 0; p < W; p++) w[p] = plane[p * TS + at];
            d[part64(P.woff, e)] = a;
        }
        if (Tn >= ntiles) break;
        T = Tn;
        __syncthreads();                        // this tile's shared-memory reads are done
    }
}

// ---------------------------------------------------------------- HBM copy probe
// The achievable-bandwidth denominator (the B200 counterpart of the reference's FPGA HBM stream
// microbenchmark, kernels/hbm_stream/): a grid-stride 16-byte copy, every byte read once and written once.
__global__ void __launch_bounds__(512) copy_probe_kernel(const float4 *__restrict__ src, float4 *__restrict__ dst,
                                                         int64_t n16) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n16; i += 4 * stride) {
        const float4 a = __ldcs(src + i), b = __ldcs(src + i + stride), c = __ldcs(src + i + 2 * stride),
                     d = __ldcs(src + i + 3 * stride);
        __stcs(dst + i, a);
        __stcs(dst + i + stride, b);
        __stcs(dst + i + 2 * stride, c);
        __stcs(dst + i + 3 * stride, d);
    }
    for (; i < n16; i += stride) __stcs(dst + i, __ldcs(src + i));
}

// ---------------------------------------------------------------- |0...0>
__global__ void set_amp0_kernel(float2 *state) { state[0] = make_float2(1.0f, 0.0f); }
__global__ void set_amp0_kernel_d(double2 *state) { state[0] = make_double2(1.0, 0.0); }

// ---------------------------------------------------------------- FP64 reductions
// Sum |a|^2 and, for every index bit q, the sum over the indices with bit q set. A block takes chunks of 2^13
// amplitudes (256 threads, 16-byte loads, 16 in flight per thread: 16 float4 of two complex64 amplitudes each,
// or 2 x 16 double2). A chunk's index bits are: bits in the 16-byte vector (complex64), 8 thread bits, 4 (5)
// load bits, and the chunk number above. Per-bit sums of the load bits share one addition tree; a bit of the
// thread or the chunk number selects whole-thread sums. The order of the sums depends on the qubit count and the
// element type alone (reduce_grid), so results are equal bit for bit from run to run and on any number of SMs.
// What bounds it: HBM. One read of the state, about 4 FP64 operations and 2 conversions per amplitude. With
// the per-bit sums in a run-time-indexed array (local memory) a 30-qubit complex64 reduction took 2.61 ms,
// half the HBM rate; now 1.23 ms (7.0 TB/s, reads only).
#define RED_THREADS 256
#define RED_CHUNK_BITS kRedChunkBits
#define RED_HI 21                  // bits above a chunk: n <= 34

// sums of |a|^2 over 16 loads: total, and the four load bits' sums (added to acc)
__device__ __forceinline__ double tree16(const double (&u)[16], double (&bit)[4]) {
    double a[8], b[4], c[2];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = u[2 * k] + u[2 * k + 1];
#pragma unroll
    for (int k = 0; k < 4; k++) b[k] = a[2 * k] + a[2 * k + 1];
    c[0] = b[0] + b[1];
    c[1] = b[2] + b[3];
    bit[0] += ((u[1] + u[3]) + (u[5] + u[7])) + ((u[9] + u[11]) + (u[13] + u[15]));
    bit[1] += (a[1] + a[3]) + (a[5] + a[7]);
    bit[2] += b[1] + b[3];
    bit[3] += c[1];
    return c[0] + c[1];
}
__device__ __forceinline__ double prob(float x, float y) { return (double)x * x + (double)y * y; }

// 16 bytes of the state: two complex64 amplitudes or one complex128. AL: the state starts on a 16-byte boundary
// (a view of a larger tensor may start between two)
template <bool AL>
__device__ __forceinline__ float4 load16(const float2 *p, int64_t i) {
    if (AL) return reinterpret_cast<const float4 *>(p)[i];
    const float2 a = p[2 * i], b = p[2 * i + 1];
    return make_float4(a.x, a.y, b.x, b.y);
}
template <bool AL>
__device__ __forceinline__ double2 load16(const double2 *p, int64_t i) { return p[i]; }

struct RedAcc {
    double tot, vec;               // vec: bit 0 of complex64 (in the vector) / the fifth load bit of complex128
    double ld[4];
};
// one chunk of a thread: returns the thread's total over the chunk
template <bool AL>
__device__ __forceinline__ double red_chunk(const float2 *p, int t, RedAcc &r) {
    float4 x[16];
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = load16<AL>(p, t + 256 * k);
    double u[16], one = 0.0;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const double hi = prob(x[k].z, x[k].w);
        one += hi;
        u[k] = prob(x[k].x, x[k].y) + hi;
    }
    r.vec += one;
    return tree16(u, r.ld);
}
template <bool AL>
__device__ __forceinline__ double red_chunk(const double2 *p, int t, RedAcc &r) {
    double sum[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double2 x[16];
        double u[16];
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = p[t + 256 * (16 * h + k)];
#pragma unroll
        for (int k = 0; k < 16; k++) u[k] = x[k].x * x[k].x + x[k].y * x[k].y;
        sum[h] = tree16(u, r.ld);
    }
    r.vec += sum[1];
    return sum[0] + sum[1];
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block b takes chunks b, b + gridDim.x, ...; out: nout doubles per block, the total and the sums of index bits
// 0 .. nout - 2 (nout = 14: the bits of one chunk, or n + 1: all bits).
template <class A, bool AL>
__global__ void __launch_bounds__(RED_THREADS, 2)
    reduce_chunks_kernel(const A *__restrict__ state, int64_t nchunks, int nout, double *__restrict__ partials) {
    constexpr bool C64 = sizeof(A) == 8;
    __shared__ double part[RED_THREADS / 32][RED_CHUNK_BITS + 1 + RED_HI];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    RedAcc r = {0.0, 0.0, {0.0, 0.0, 0.0, 0.0}};
    double hi[RED_HI];
#pragma unroll
    for (int q = 0; q < RED_HI; q++) hi[q] = 0.0;
    for (int64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const double s = red_chunk<AL>(state + (c << RED_CHUNK_BITS), t, r);
        r.tot += s;
        if (nout > RED_CHUNK_BITS + 1) {
#pragma unroll
            for (int q = 0; q < RED_HI; q++)
                if ((c >> q) & 1) hi[q] += s;
        }
    }
    auto put = [&](int o, double v) {
        v = warp_sum(v);
        if (lane == 0) part[warp][o] = v;
    };
    constexpr int T0 = C64 ? 1 : 0;              // first thread bit
    put(0, r.tot);
    if (C64) put(1, r.vec);
#pragma unroll
    for (int q = 0; q < 8; q++) put(1 + T0 + q, (t >> q) & 1 ? r.tot : 0.0);
#pragma unroll
    for (int q = 0; q < 4; q++) put(1 + T0 + 8 + q, r.ld[q]);
    if (!C64) put(13, r.vec);
    if (nout > RED_CHUNK_BITS + 1) {
#pragma unroll
        for (int q = 0; q < RED_HI; q++)
            if (q < nout - 1 - RED_CHUNK_BITS) put(1 + RED_CHUNK_BITS + q, hi[q]);
    }
    __syncthreads();
    if (t < nout) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < RED_THREADS / 32; w++) s += part[w][t];
        partials[(int64_t)blockIdx.x * nout + t] = s;
    }
}

// states of fewer than 2^13 amplitudes: one block, a strided pass per output (nout = n + 1)
template <class A>
__global__ void __launch_bounds__(RED_THREADS)
    reduce_small_kernel(const A *__restrict__ state, int n, double *__restrict__ partials) {
    __shared__ double part[RED_THREADS / 32][RED_CHUNK_BITS + 1];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double s[RED_CHUNK_BITS + 1];
#pragma unroll
    for (int q = 0; q <= RED_CHUNK_BITS; q++) s[q] = 0.0;
    for (int i = t; i < (1 << n); i += RED_THREADS) {
        const A a = state[i];
        const double p = (double)a.x * a.x + (double)a.y * a.y;
        s[0] += p;
#pragma unroll
        for (int q = 0; q < RED_CHUNK_BITS; q++)
            if ((i >> q) & 1) s[1 + q] += p;
    }
#pragma unroll
    for (int q = 0; q <= RED_CHUNK_BITS; q++) {
        const double v = warp_sum(s[q]);
        if (lane == 0) part[warp][q] = v;
    }
    __syncthreads();
    if (t <= n) {
        double v = 0.0;
        for (int w = 0; w < RED_THREADS / 32; w++) v += part[w][t];
        partials[t] = v;
    }
}

// out[0] = total, out[1 + q] = total - 2 * (sum over i with bit q set). Block o reduces output o over the block
// partials (nout each); with one-chunk partials (nout = 14) a bit above a chunk is a bit of the block number.
__global__ void __launch_bounds__(128)
    reduce_final_kernel(const double *__restrict__ partials, int nblocks, int nout, double *__restrict__ out) {
    __shared__ double s_tot[4], s_bit[4];
    const int o = blockIdx.x, t = threadIdx.x;
    double tot = 0.0, s = 0.0;
    for (int b = t; b < nblocks; b += 128) {
        const double *p = partials + (int64_t)b * nout;
        const double x = p[0];
        tot += x;
        if (o >= 1) s += o < nout ? p[o] : ((b >> (o - nout)) & 1 ? x : 0.0);
    }
    tot = warp_sum(tot);
    s = warp_sum(s);
    if ((t & 31) == 0) { s_tot[t >> 5] = tot; s_bit[t >> 5] = s; }
    __syncthreads();
    if (t == 0) {
        tot = (s_tot[0] + s_tot[1]) + (s_tot[2] + s_tot[3]);
        s = (s_bit[0] + s_bit[1]) + (s_bit[2] + s_bit[3]);
        out[o] = o == 0 ? tot : tot - 2.0 * s;
    }
}

// ---------------------------------------------------------------- chunk probabilities
// What bounds it: the read of the state. Small chunks (256 amplitudes to 8 KiB) take a warp each, grid-strided; larger
// ones a block each, which the hardware deals out as blocks finish. A warp per chunk had been used up to 2^13 amplitudes,
// where the last turn of the grid-stride is a good part of the time and a few chunks leave the SMs idle. Device time,
// warp / block: chunks of 2^12 complex64 amplitudes (the default) 8.6 / 5.0 us at 18 qubits, 24.5 / 23.2 at 24, 322 / 290
// at 28; 2^11: 26.7 / 23.2 at 24; 2^10: 24.8 / 29.9; of 2^12 complex128 amplitudes 48.6 / 43.7 us at 24 qubits, 622 / 582
// at 28, 2^10: 43.8 / 41.6 at 24, 2^9: 43.9 / 62.0.
#define CHUNK_WARP_MIN 8           // 256 complex64 amplitudes: 4 loads per lane
#define CHUNK_WARP_BYTES 8192
// One warp per chunk of 2^cb amplitudes: 16-byte loads, eight in flight per lane, no block barriers.
__device__ __forceinline__ double prob16(const float4 &v) { return prob(v.x, v.y) + prob(v.z, v.w); }
__device__ __forceinline__ double prob16(const double2 &v) { return v.x * v.x + v.y * v.y; }
template <class A, bool AL>
__global__ void __launch_bounds__(RED_THREADS)
    chunk_probs_warp_kernel(const A *__restrict__ state, int cb, int64_t nchunks, double *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * (RED_THREADS / 32);
    const int len = (int)(((size_t)sizeof(A) << cb) / 16);       // a multiple of 128
    for (int64_t c = (int64_t)blockIdx.x * (RED_THREADS / 32) + (threadIdx.x >> 5); c < nchunks; c += nw) {
        const A *p = state + (c << cb);
        double acc = 0.0;
        int i = lane;
        for (; i + 224 < len; i += 256) {
            decltype(load16<AL>(p, 0)) v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = load16<AL>(p, i + 32 * k);
#pragma unroll
            for (int k = 0; k < 8; k++) acc += prob16(v[k]);
        }
        for (; i < len; i += 32) acc += prob16(load16<AL>(p, i));
        acc = warp_sum(acc);
        if (lane == 0) out[c] = acc;
    }
}

// One block per chunk (any other chunk size), eight loads in flight per thread. (One at a time with 64-bit indices, a
// whole 24-qubit complex128 state in one chunk took 12.3 ms, with 32-bit ones 9.3.)
template <class A>
__global__ void __launch_bounds__(RED_THREADS)
    chunk_probs_kernel(const A *__restrict__ state, int cb, double *__restrict__ out) {
    __shared__ double s[RED_THREADS];
    const A *p = state + ((int64_t)blockIdx.x << cb);
    const int64_t len = 1ll << cb;
    double acc = 0.0;
    auto add = [&](const A &a) { acc += (double)a.x * a.x + (double)a.y * a.y; };
    int64_t i = threadIdx.x;
    for (; i + 7 * RED_THREADS < len; i += 8 * RED_THREADS) {
        A a[8];
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = p[i + k * RED_THREADS];
#pragma unroll
        for (int k = 0; k < 8; k++) add(a[k]);
    }
    for (; i < len; i += RED_THREADS) add(p[i]);
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = s[0];
}

// ---------------------------------------------------------------- Born sampler
// Chunk probabilities are scanned in groups of 2^SCAN_BITS (one block each, in place), and the groups' totals by
// every sampling block for itself: the cumulative sum up to chunk c is the total of the groups before c's plus
// the scanned value. One warp per shot then finds the chunk (binary searches), the 1/32 of the chunk and the
// amplitude, each the first whose running FP64 sum exceeds what is left of the draw.
// What bounds it: the read of the state for the chunk probabilities. A scan of 2^16 values in one block and one
// thread per shot adding up to 4096 amplitudes one after the other took 1.20 ms for 1024 shots of 28 qubits
// (HBM floor 0.33 ms); now 0.34 ms, and 38 instead of 440-530 us at 12-20 qubits.
#define SCAN_BITS 12
#define SCAN_THREADS 1024
__device__ __forceinline__ double warp_scan(double v, int lane) {       // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
    }
    return v;
}
__global__ void __launch_bounds__(SCAN_THREADS) scan_kernel(double *__restrict__ v, int64_t nc) {
    __shared__ double wsum[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int64_t i = ((int64_t)blockIdx.x << SCAN_BITS) + 4 * t;
    double x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = i + k < nc ? v[i + k] : 0.0;
    x[1] += x[0]; x[2] += x[1]; x[3] += x[2];
    const double incl = warp_scan(x[3], lane);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) wsum[lane] = warp_scan(wsum[lane], lane);
    __syncthreads();
    double before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = 0.0;
    if (warp > 0) before += wsum[warp - 1];
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (i + k < nc) v[i + k] = before + x[k];
}

#define SAMPLE_WARPS 8
#define SAMPLE_GROUPS 1024         // groups of chunks: 2^(34 - 12 - SCAN_BITS)
template <class A>
__global__ void __launch_bounds__(32 * SAMPLE_WARPS)
    sample_kernel(const A *__restrict__ state, int cb, const double *__restrict__ cdf, int64_t nc,
                  const double *__restrict__ uni, int shots, int64_t *__restrict__ out) {
    __shared__ double gcdf[SAMPLE_GROUPS];       // inclusive sums of the group totals
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int ng = (int)((nc + (1 << SCAN_BITS) - 1) >> SCAN_BITS);
    for (int g = t; g < ng; g += 32 * SAMPLE_WARPS) {
        const int64_t last = ((int64_t)(g + 1) << SCAN_BITS) - 1;
        gcdf[g] = cdf[last < nc ? last : nc - 1];
    }
    __syncthreads();
    if (warp == 0) {
        double run = 0.0;
        for (int g0 = 0; g0 < ng; g0 += 32) {
            const double v = warp_scan(g0 + lane < ng ? gcdf[g0 + lane] : 0.0, lane) + run;
            run = __shfl_sync(0xffffffffu, v, 31);
            if (g0 + lane < ng) gcdf[g0 + lane] = v;
        }
    }
    __syncthreads();
    const int s = blockIdx.x * SAMPLE_WARPS + warp;
    if (s >= shots) return;
    const double x = uni[s] * gcdf[ng - 1];
    int lo = 0, hi = ng;                         // first group whose cumulative sum exceeds x
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (gcdf[mid] > x) hi = mid;
        else lo = mid + 1;
    }
    const int g = lo < ng ? lo : ng - 1;
    double rem = x - (g > 0 ? gcdf[g - 1] : 0.0);
    const int64_t first = (int64_t)g << SCAN_BITS;
    const int cnt = (int)(nc - first < (1 << SCAN_BITS) ? nc - first : 1 << SCAN_BITS);
    lo = 0; hi = cnt;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cdf[first + mid] > rem) hi = mid;
        else lo = mid + 1;
    }
    const int cc = lo < cnt ? lo : cnt - 1;
    if (cc > 0) rem -= cdf[first + cc - 1];
    const int64_t base = (first + cc) << cb;
    const A *p = state + base;
    // the lane sums of 32 consecutive runs of `per` amplitudes; picks the first run whose cumulative sum exceeds
    // rem (-1: none) and leaves in rem what remains inside it
    auto pick = [&](double v) -> int {
        double run = 0.0;
        for (int k = 0; k < 32; k++) {
            const double y = __shfl_sync(0xffffffffu, v, k);
            if (run + y > rem) {
                rem -= run;
                return k;
            }
            run += y;
        }
        return -1;
    };
    auto prob_at = [&](int i) -> double {
        const A a = p[i];
        return (double)a.x * a.x + (double)a.y * a.y;
    };
    int at = 0, len = 1 << cb;                   // the run the draw lies in: [at, at + len), len >= 1024 / 32
    while (len > 32) {
        const int per = len >> 5;
        double v = 0.0;
#pragma unroll 8
        for (int i = 0; i < per; i++) v += prob_at(at + lane * per + i);
        const int k = pick(v);
        if (k < 0) break;                        // rounding left the draw beyond the run's sum: its last amplitude
        at += k * per;
        len = per;
    }
    if (len <= 32) {
        const double v = lane < len ? prob_at(at + lane) : 0.0;
        const int k = pick(v);
        const unsigned some = __ballot_sync(0xffffffffu, v > 0.0);
        if (k >= 0) at += k;
        else at += some ? 31 - __clz((int)some) : len - 1;
    } else {
        at += len - 1;
    }
    if (lane == 0) out[s] = base + at;
}

}  // namespace dev

// ---------------------------------------------------------------- host launchers
// dtype: 0 = complex64 (float2 amplitudes), 1 = complex128 (double2)
template <class A, int TB>
static cudaError_t launch_remap_t(const void *src, void *dst, const dev::RemapParams &P, int nsm, cudaStream_t stream) {
    constexpr int smem = (int)(sizeof(A) << TB);
    static_assert(smem <= 48 * 1024, "no opt-in needed");
    const int64_t ntiles = 1ll << P.nfree;
    int64_t grid = (int64_t)nsm * 3;
    if (grid > ntiles) grid = ntiles;
    dev::remap_kernel<A, TB><<<(unsigned)grid, REMAP_THREADS, smem, stream>>>((const A *)src, (A *)dst, P);
    return cudaGetLastError();
}

cudaError_t launch_remap(const void *src, void *dst, int n, const int32_t *perm, int dtype, int nsm,
                         cudaStream_t stream) {
    dev::RemapParams P;
    memset(&P, 0, sizeof(P));
    const int run = dtype ? 5 : 6;                         // 512-byte runs on both sides
    const int most = 2 * run < REMAP_TB ? 11 : REMAP_TB;   // 32 KiB tiles
    const int tbits = n < most ? n : most;
    int inv[64];
    for (int j = 0; j < n; j++) inv[perm[j]] = j;          // source bit perm[j] -> destination bit j
    bool in_tile[64] = {false};
    int cnt = 0;
    // the lowest source and destination bits by turns (a small state's tile may not hold all of them)
    for (int b = 0; b < run; b++) {
        if (cnt < tbits && !in_tile[b]) { in_tile[b] = true; cnt++; }
        if (cnt < tbits && !in_tile[perm[b]]) { in_tile[perm[b]] = true; cnt++; }
    }
    for (int b = 0; b < n && cnt < tbits; b++)
        if (!in_tile[b]) { in_tile[b] = true; cnt++; }
    int ubits[REMAP_TB], nu = 0, nf = 0;                   // tile position bit i <-> source bit ubits[i], ascending
    for (int b = 0; b < n; b++) {
        if (in_tile[b]) {
            ubits[nu++] = b;
        } else {
            P.fx[nf] = (uint8_t)b;
            P.fy[nf] = (uint8_t)inv[b];
            nf++;
        }
    }
    P.nfree = nf;
    // destination order: bit q walks the tile bit with the q-th smallest destination position
    int order[REMAP_TB];
    bool used[REMAP_TB] = {false};
    for (int q = 0; q < nu; q++) {
        int best = -1;
        for (int i = 0; i < nu; i++)
            if (!used[i] && (best < 0 || inv[ubits[i]] < inv[ubits[best]])) best = i;
        used[best] = true;
        order[q] = best;
    }
    // swizzle: the tile bits that destination-order bits 0..4 walk vary across a warp's shared-memory loads; each of
    // them above bit 4 is XORed onto a low bit (0..4) that none of the others occupies
    int swz[REMAP_TB];
    for (int b = 0; b < REMAP_TB; b++) swz[b] = -1;
    bool low_used[REMAP_BANK_BITS] = {false};
    for (int q = 0; q < REMAP_BANK_BITS; q++)
        if (order[q] < REMAP_BANK_BITS) low_used[order[q]] = true;
    for (int q = 0, slot = 0; q < REMAP_BANK_BITS; q++) {
        if (order[q] < REMAP_BANK_BITS) continue;
        while (low_used[slot]) slot++;
        swz[order[q]] = slot;
        low_used[slot] = true;
    }
    auto place = [&](int b) { return (1u << b) ^ (swz[b] >= 0 ? 1u << swz[b] : 0u); };
    for (int i = 0; i < nu; i++) {
        P.roff[i] = 1ull << ubits[i];
        P.woff[i] = 1ull << inv[ubits[order[i]]];
        P.spin[i] = place(i);
        P.spout[i] = place(order[i]);
    }
    if (dtype) {
        if (tbits == 11) return launch_remap_t<double2, 11>(src, dst, P, nsm, stream);
        return launch_remap_t<double2, 10>(src, dst, P, nsm, stream);
    }
    if (tbits == 12) return launch_remap_t<float2, 12>(src, dst, P, nsm, stream);
    if (tbits == 11) return launch_remap_t<float2, 11>(src, dst, P, nsm, stream);
    return launch_remap_t<float2, 10>(src, dst, P, nsm, stream);
}

cudaError_t launch_copy_probe(void *dst, const void *src, size_t bytes, int nsm, cudaStream_t stream) {
    const int64_t n16 = (int64_t)(bytes / 16);
    int64_t grid = (int64_t)nsm * 4;
    if (grid > (n16 + 511) / 512) grid = (n16 + 511) / 512;
    if (grid < 1) grid = 1;
    dev::copy_probe_kernel<<<(unsigned)grid, 512, 0, stream>>>((const float4 *)src, (float4 *)dst, n16);
    return cudaGetLastError();
}

cudaError_t launch_set_amp0(void *state, int dtype, cudaStream_t stream) {
    if (dtype) dev::set_amp0_kernel_d<<<1, 1, 0, stream>>>((double2 *)state);
    else dev::set_amp0_kernel<<<1, 1, 0, stream>>>((float2 *)state);
    return cudaGetLastError();
}

int reduce_bits(int n) { return reduce_bits_of(n); }

size_t reduce_scratch_bytes(int n, int chunk_bits) {
    const int B = reduce_bits(n);
    const size_t red = ((size_t)1 << (n - B)) * (B + 1) * sizeof(double);
    const size_t smp = ((size_t)1 << (n - chunk_bits)) * sizeof(double);
    return red > smp ? red : smp;
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <class A>
static cudaError_t launch_reduce_t(const A *state, int n, double *out, double *partials, cudaStream_t stream) {
    const auto [blocks, nout] = reduce_grid(n);
    if (n < RED_CHUNK_BITS) dev::reduce_small_kernel<A><<<1, RED_THREADS, 0, stream>>>(state, n, partials);
    else if (aligned16(state))
        dev::reduce_chunks_kernel<A, true><<<(unsigned)blocks, RED_THREADS, 0, stream>>>(
            state, 1ll << (n - RED_CHUNK_BITS), nout, partials);
    else
        dev::reduce_chunks_kernel<A, false><<<(unsigned)blocks, RED_THREADS, 0, stream>>>(
            state, 1ll << (n - RED_CHUNK_BITS), nout, partials);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    dev::reduce_final_kernel<<<(unsigned)(n + 1), 128, 0, stream>>>(partials, (int)blocks, nout, out);
    return cudaGetLastError();
}

cudaError_t launch_reduce(const void *state, int n, int dtype, double *out, void *scratch, cudaStream_t stream) {
    if (dtype) return launch_reduce_t((const double2 *)state, n, out, (double *)scratch, stream);
    return launch_reduce_t((const float2 *)state, n, out, (double *)scratch, stream);
}

// ---------------------------------------------------------------- reduction without caller scratch
// Fixed-size scratch for reduce_f64_noalloc: a 2^n state needs 2^(n-B) * (B+1) doubles of block partials
// (B = reduce_bits(n)); the largest supported state (n = 34, B = 24) needs 1024 * 25 = 25600. The array
// holds 32768 doubles (256 KiB). It is part of the module image, so every GPU that loads the library keeps
// it until the process exits. The partial count does not depend on the amplitude type.
#define QSV_NOALLOC_REDUCE_DOUBLES 32768
#define QSV_NOALLOC_N_MIN 10
#define QSV_NOALLOC_N_MAX 34
static __device__ __align__(256) double g_noalloc_reduce_scratch[QSV_NOALLOC_REDUCE_DOUBLES];

constexpr bool noalloc_fits_every_n() {
    for (int n = QSV_NOALLOC_N_MIN; n <= QSV_NOALLOC_N_MAX; n++)
        if (reduce_room(n) > QSV_NOALLOC_REDUCE_DOUBLES) return false;
    return true;
}
static_assert(noalloc_fits_every_n(), "the fixed reduction scratch must hold the partials of every supported n");

size_t noalloc_reduce_capacity() { return QSV_NOALLOC_REDUCE_DOUBLES * sizeof(double); }

// Device address of the fixed scratch for the current device. Looked up once per device (the host-side
// name of the array is only a stand-in for it, never a device address) and cached for the life of the
// process: the cache assumes the device's primary context is not reset (cudaDeviceReset) while the library
// is loaded, since a reset unloads the module and the cached address would then be stale.
static cudaError_t noalloc_scratch_ptr(double **out) {
    static std::mutex mu;
    static double *ptr[64] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(mu);
    if (!ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_reduce_scratch);
        if (e != cudaSuccess) return e;
        ptr[dev] = static_cast<double *>(p);
    }
    *out = ptr[dev];
    return cudaSuccess;
}

cudaError_t launch_reduce_noalloc(const void *state, int n, int dtype, double *out, cudaStream_t stream, size_t *need) {
    const size_t doubles = (size_t)reduce_room(n);
    *need = doubles * sizeof(double);
    if (doubles > QSV_NOALLOC_REDUCE_DOUBLES) return cudaErrorInvalidValue;
    double *scratch = nullptr;
    cudaError_t e = noalloc_scratch_ptr(&scratch);
    if (e != cudaSuccess) return e;
    return launch_reduce(state, n, dtype, out, scratch, stream);
}

template <class A>
static cudaError_t launch_chunk_probs_t(const A *state, int n, int cb, double *out, int nsm, cudaStream_t stream) {
    const int64_t nc = 1ll << (n - cb);
    if (cb >= CHUNK_WARP_MIN && sizeof(A) << cb <= CHUNK_WARP_BYTES) {
        int64_t grid = (nc + RED_THREADS / 32 - 1) / (RED_THREADS / 32);
        if (grid > (int64_t)nsm * 8) grid = (int64_t)nsm * 8;
        if (aligned16(state))
            dev::chunk_probs_warp_kernel<A, true><<<(unsigned)grid, RED_THREADS, 0, stream>>>(state, cb, nc, out);
        else
            dev::chunk_probs_warp_kernel<A, false><<<(unsigned)grid, RED_THREADS, 0, stream>>>(state, cb, nc, out);
    } else {
        dev::chunk_probs_kernel<A><<<(unsigned)nc, RED_THREADS, 0, stream>>>(state, cb, out);
    }
    return cudaGetLastError();
}

cudaError_t launch_chunk_probs(const void *state, int n, int dtype, int cb, double *out, int nsm, cudaStream_t stream) {
    if (dtype) return launch_chunk_probs_t((const double2 *)state, n, cb, out, nsm, stream);
    return launch_chunk_probs_t((const float2 *)state, n, cb, out, nsm, stream);
}

cudaError_t launch_sample(const void *state, int n, int dtype, int cb, const double *uni, int shots, int64_t *out,
                          void *scratch, int nsm, cudaStream_t stream) {
    double *cdf = (double *)scratch;
    const int64_t nc = 1ll << (n - cb);
    cudaError_t e = launch_chunk_probs(state, n, dtype, cb, cdf, nsm, stream);
    if (e != cudaSuccess) return e;
    dev::scan_kernel<<<(unsigned)((nc + (1 << SCAN_BITS) - 1) >> SCAN_BITS), SCAN_THREADS, 0, stream>>>(cdf, nc);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (shots > 0) {
        const unsigned grid = (unsigned)((shots + SAMPLE_WARPS - 1) / SAMPLE_WARPS);
        if (dtype)
            dev::sample_kernel<double2><<<grid, 32 * SAMPLE_WARPS, 0, stream>>>((const double2 *)state, cb, cdf, nc, uni,
                                                                                shots, out);
        else
            dev::sample_kernel<float2><<<grid, 32 * SAMPLE_WARPS, 0, stream>>>((const float2 *)state, cb, cdf, nc, uni,
                                                                               shots, out);
    }
    return cudaGetLastError();
}

}  // namespace qsv
