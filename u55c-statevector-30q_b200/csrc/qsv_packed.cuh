// qsv_packed.cuh -- packed FP32x2 arithmetic on 64-bit registers (sm_100a), shared by the interpreter
// (qsv_interp.cuh) and kernels specialised at run time (qsv_jit_ops.cuh).
//
// A consumer thread holds its slots as R = (re, re) and I = (im, im) of the two amplitudes of tile bit 0, each one
// 64-bit value from load to store: the packed instructions take aligned register pairs, and values that are
// 64 bits wide throughout never have to be moved into one. The arithmetic is the canonical
// fused-multiply-add chain of qsv_device.cuh.
#pragma once
#include "qsv_device.cuh"

namespace qsv {
namespace dev {

typedef unsigned long long p2;      // two packed floats: low half = amplitude with tile bit 0 clear

__device__ __forceinline__ p2 pk(float lo, float hi) {
    p2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpk(p2 a, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a)); }
__device__ __forceinline__ p2 flip(p2 a) {       // exchange the halves
    float lo, hi;
    unpk(a, lo, hi);
    return pk(hi, lo);
}
// zero, but not known to be the same in all lanes: data read through it goes to ordinary registers (read at a
// warp-uniform address it would go through uniform ones, and packed operands have to be moved out of those)
__device__ __forceinline__ uint32_t lane_zero() {
    uint32_t z;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(z));
    return z >> 5;
}
// A slot between the state's order (re0, im0, re1, im1) and the packed registers (re0, re1), (im0, im1): the middle
// words change places. As plain moves they are issued to the multiply-add pipe, which the ops need; combined with
// z, a zero that is not known at compile time, they are logic, off that pipe.
__device__ __forceinline__ void swap_mid(uint4 &v, uint32_t z) {
    const uint32_t t = v.y ^ z;
    v.y = v.z ^ z;
    v.z = t ^ z;
}
__device__ __forceinline__ p2 pku(uint32_t lo, uint32_t hi) {
    p2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpku(p2 a, uint32_t &lo, uint32_t &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(a));
}
__device__ __forceinline__ void load_slot(const float2 *p, p2 &R, p2 &I, uint32_t z) {
    uint4 v = *reinterpret_cast<const uint4 *>(p);
    swap_mid(v, z);
    R = pku(v.x, v.y);
    I = pku(v.z, v.w);
}
__device__ __forceinline__ void store_slot(float2 *p, p2 R, p2 I, uint32_t z) {
    uint4 v;
    unpku(R, v.x, v.y);
    unpku(I, v.z, v.w);
    swap_mid(v, z);
    *reinterpret_cast<uint4 *>(p) = v;
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

__device__ __forceinline__ p2 shfl_p(p2 a, int xm) {
    float lo, hi;
    unpk(a, lo, hi);
    lo = __shfl_xor_sync(0xffffffffu, lo, xm);
    hi = __shfl_xor_sync(0xffffffffu, hi, xm);
    return pk(lo, hi);
}
}  // namespace dev
}  // namespace qsv
