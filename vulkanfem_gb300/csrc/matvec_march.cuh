// matvec_march.cuh -- the element-by-element product's building blocks shared by
// its translation units: the Walsh-basis and dense element products, the output
// stage and the march up a z range (kernels.cu: FP32, FP64 and double-float
// kernels; matvec_fx.cu: the fixed-point FP64 product, which hands blocks it
// cannot represent to the FP64 march).  Everything here has
// internal linkage (one copy per translation unit).
#pragma once

#include <type_traits>

#include "double_float.cuh"
#include "kernels.h"
#include "reduce.cuh"

namespace vfem {
namespace {

constexpr int MV_TX = 32, MV_TY = 8, MV_ZC = 32;  // z layers per product block (32: 5% faster than 16)

// One name for FP32, FP64 and double-float multiply-adds in the templates below.
__device__ __forceinline__ float fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma(double a, double b, double c) { return ::fma(a, b, c); }

// Conversions between a storage type T and a compute type TC of the matvec.
template <typename T, typename TC>
struct Cvt {
    static __device__ __forceinline__ TC in(T v) { return TC(v); }
    static __device__ __forceinline__ T out(TC v) { return T(v); }
};
template <>
struct Cvt<double, df> {
    static __device__ __forceinline__ df in(double v) {
        const float h = __double2float_rn(v);
        return df(h, __double2float_rn(v - (double)h));
    }
    static __device__ __forceinline__ double out(df v) { return (double)v.hi + (double)v.lo; }
};
__device__ __forceinline__ float toF(float v) { return v; }
__device__ __forceinline__ float toF(double v) { return (float)v; }
__device__ __forceinline__ float toF(df v) { return v.hi; }  // hi is v rounded to FP32

template <>
struct DotAcc<df> {
    df s = df(0.f, 0.f);
    __device__ __forceinline__ void add(df v) { s = s + v; }
    __device__ __forceinline__ double get() const { return (double)s.hi + (double)s.lo; }
};

template <typename T>
struct Ks {
    T v[45];
};
// The same for a cube, whose axes are interchangeable: one constant per kind of
// entry (cubeConstants): a - b and b of the normal strains, the shears, the
// mode-7 terms, a and b of the bending pairs, a - b and b of the (1,1,1) triple.
template <typename T>
struct Kc {
    T v[8];
};
template <typename T>
struct Kd {
    T v[576];
};

// y = Khat u on the 45-entry pattern (modes 1..7; mode 0, the rigid translation,
// has no energy).  u and y hold 3 m + c for mode m and component c.
template <typename T>
__device__ __forceinline__ void applyKhat(const T (&u)[24], T (&y)[24], const Ks<T>& k) {
#pragma unroll
    for (int i = 0; i < 24; ++i) y[i] = T(0);
#define KS_(n, r, c) y[r] = fma(k.v[n], u[c], y[r]);
    KS_(0, 3, 3) KS_(1, 3, 7) KS_(2, 3, 14) KS_(3, 7, 3) KS_(4, 7, 7) KS_(5, 7, 14) KS_(6, 14, 3) KS_(7, 14, 7)
    KS_(8, 14, 14)
    KS_(9, 6, 6) KS_(10, 6, 4) KS_(11, 4, 6) KS_(12, 4, 4) KS_(13, 23, 23)
    KS_(14, 12, 12) KS_(15, 12, 5) KS_(16, 5, 12) KS_(17, 5, 5) KS_(18, 22, 22)
    KS_(19, 13, 13) KS_(20, 13, 8) KS_(21, 8, 13) KS_(22, 8, 8) KS_(23, 21, 21)
    KS_(24, 10, 10) KS_(25, 10, 17) KS_(26, 17, 10) KS_(27, 17, 17)
    KS_(28, 9, 9) KS_(29, 9, 20) KS_(30, 20, 9) KS_(31, 20, 20)
    KS_(32, 15, 15) KS_(33, 15, 19) KS_(34, 19, 15) KS_(35, 19, 19)
    KS_(36, 18, 18) KS_(37, 18, 16) KS_(38, 18, 11) KS_(39, 16, 18) KS_(40, 16, 16) KS_(41, 16, 11)
    KS_(42, 11, 18) KS_(43, 11, 16) KS_(44, 11, 11)
#undef KS_
}

// y = e Khat u in the modes 1..7.
template <typename T>
__device__ __forceinline__ void scaledKhat(T (&u)[24], T (&y)[24], const Ks<T>& k, T e);
// The cube's: 8 scaled constants and 33 operations instead of 21 and 45.
template <typename T>
__device__ __forceinline__ void scaledKhat(T (&u)[24], T (&y)[24], const Kc<T>& k, T e) {
    T c[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = e * k.v[i];
    y[0] = y[1] = y[2] = T(0);
    const T n = c[1] * (u[3] + u[7] + u[14]), t = c[7] * (u[18] + u[16] + u[11]);
    y[3] = fma(c[0], u[3], n);
    y[7] = fma(c[0], u[7], n);
    y[14] = fma(c[0], u[14], n);
    y[6] = y[4] = c[2] * (u[6] + u[4]);
    y[12] = y[5] = c[2] * (u[12] + u[5]);
    y[13] = y[8] = c[2] * (u[13] + u[8]);
    y[23] = c[3] * u[23];
    y[22] = c[3] * u[22];
    y[21] = c[3] * u[21];
    y[10] = fma(c[4], u[10], c[5] * u[17]);
    y[17] = fma(c[4], u[17], c[5] * u[10]);
    y[9] = fma(c[4], u[9], c[5] * u[20]);
    y[20] = fma(c[4], u[20], c[5] * u[9]);
    y[15] = fma(c[4], u[15], c[5] * u[19]);
    y[19] = fma(c[4], u[19], c[5] * u[15]);
    y[18] = fma(c[6], u[18], t);
    y[16] = fma(c[6], u[16], t);
    y[11] = fma(c[6], u[11], t);
}

// y = e * Ke u, general symmetric Ke.
template <typename T>
__device__ __forceinline__ void elemDense(const T (&u)[24], T (&y)[24], const Kd<T>& k, T e) {
#pragma unroll
    for (int r = 0; r < 24; ++r) {
        T s = T(0);
#pragma unroll
        for (int c = 0; c < 24; ++c) s = fma(k.v[r * 24 + c], u[c], s);
        y[r] = s * e;
    }
}

// Shared-memory node slots are padded to 4 values (x, y, z, unused) so that a
// node moves with one 16-byte (float) or two 16-byte (double) accesses.
constexpr int kSuElems = 2 * (MV_TY + 1) * (MV_TX + 1) * 4;
constexpr int kSyElems = MV_TY * MV_TX * 6 * 4;

template <typename T>
__device__ __forceinline__ void stSlot(T* p, T a, T b, T c);
template <>
__device__ __forceinline__ void stSlot<float>(float* p, float a, float b, float c) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, 0.f);
}
template <>
__device__ __forceinline__ void stSlot<double>(double* p, double a, double b, double c) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
    reinterpret_cast<double2*>(p)[1] = make_double2(c, 0.0);
}
template <>
__device__ __forceinline__ void stSlot<df>(df* p, df a, df b, df c) {
    reinterpret_cast<float4*>(p)[0] = make_float4(a.hi, a.lo, b.hi, b.lo);
    reinterpret_cast<float4*>(p)[1] = make_float4(c.hi, c.lo, 0.f, 0.f);
}
template <typename T>
__device__ __forceinline__ void ldSlot(const T* p, T& a, T& b, T& c);
template <>
__device__ __forceinline__ void ldSlot<df>(const df* p, df& a, df& b, df& c) {
    const float4 v0 = reinterpret_cast<const float4*>(p)[0], v1 = reinterpret_cast<const float4*>(p)[1];
    a = df(v0.x, v0.y);
    b = df(v0.z, v0.w);
    c = df(v1.x, v1.y);
}
template <>
__device__ __forceinline__ void ldSlot<float>(const float* p, float& a, float& b, float& c) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = v.x;
    b = v.y;
    c = v.z;
}
template <>
__device__ __forceinline__ void ldSlot<double>(const double* p, double& a, double& b, double& c) {
    const double2 v0 = reinterpret_cast<const double2*>(p)[0], v1 = reinterpret_cast<const double2*>(p)[1];
    a = v0.x;
    b = v0.y;
    c = v1.x;
}

// Output stage of the matvec kernels for one owned node s: sum = (K x)_s before
// the fixed-row mask; writes y (and y32) by mode and accumulates the dots.  fl:
// the node's flags.  The x.(Kx) term skips unused and fixed nodes, where Kx is
// 0, so that whatever x holds there (the caller's buffer may carry NaN at nodes
// no element touches) cannot reach the dot.
template <typename T, typename TC>
__device__ __forceinline__ void mvOutput(const MatvecArgs<T>& a, int64_t s, const TC (&sum)[3], uint8_t fl,
                                         const TC (&xo)[3], DotAcc<TC>& d0, DotAcc<TC>& d1) {
    typedef Cvt<T, TC> C;
    const bool fixed = (fl & FLAG_FIXED) != 0;
    const bool live = (fl & FLAG_USED) && !fixed;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const TC ax = fixed ? TC(0) : sum[c];
        TC out;
        TC fv = TC(0);
        if (a.mode != MV_AX) fv = C::in(a.f[3 * s + c]);
        const TC xv = xo[c];
        switch (a.mode) {
            case MV_AX: out = ax; break;
            case MV_RESID: out = fv - ax; break;
            case MV_RESID0: out = fixed ? TC(0) : fv - ax; break;
            default: out = fixed ? TC(0) : xv + TC(a.omega) * C::in(a.dinv[3 * s + c]) * (fv - ax); break;
        }
        if (std::is_same<T, float>::value || a.y) a.y[3 * s + c] = C::out(out);
        if (a.y32) a.y32[3 * s + c] = toF(out);
        if (a.dot0 == DOT_X_OUT) d0.add(live ? xv * out : TC(0));
        else if (a.dot0 == DOT_OUT_OUT) d0.add(out * out);
        else if (a.dot0 == DOT_F_OUT) d0.add(fv * out);
        if (a.dot1) d1.add(out * C::in(a.aux[3 * s + c]));
    }
}

// Element-by-element product with a general (dense 24 x 24) Ke, for element
// matrices without the isotropic-cube symmetry (for example the reference's
// Ke0.dat in its own node order); structured Ke use kMatvecH below.
// A 2.5-D tile: a block of 32 x 8 threads marches
// up a z-range; at each element layer thread (tx,ty) computes the element whose
// lower corner is node (x0+tx-1, y0+ty-1) and owns node (x0+tx, y0+ty), which is
// the (1,1) corner of its own element and a corner of the three neighbouring
// threads' elements.  Element outputs pass through shared memory once; each
// owned node sums its four in-layer contributions for the bottom face (node
// layer k) and the top face (node layer k+1), so no atomics are needed.
// The march is software-pipelined: while layer k is computed, the node values
// of layer k+2, the modulus of element layer k+1 and the owned node's flags
// are already in flight to registers.  The 33 x 9 node tile of a layer is
// loaded without integer division: every thread loads its own slot, row 8
// comes from the ty == 0 threads and column 32 from nine threads of row 1.
//
// T is the storage type of the vectors, TC the arithmetic type (T, or df for the
// true residual of the mixed-precision solve: FP64 vectors, df arithmetic).
// One block's march: fills d0 and d1 (this thread's dots).
template <typename T, typename TC>
__device__ __forceinline__ void denseMarch(const MatvecArgs<T>& a, const Kd<TC>& kp, unsigned char* smemRaw,
                                           DotAcc<TC>& d0, DotAcc<TC>& d1, [[maybe_unused]] int layers = MV_ZC) {
    typedef Cvt<T, TC> C;
    TC* su = reinterpret_cast<TC*>(smemRaw);
    TC* sy = su + kSuElems;
    const Grid g = a.g;
    const int zc = std::is_same<TC, double>::value ? layers : MV_ZC;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * (MV_TX - 1), y0 = blockIdx.y * (MV_TY - 1), z0 = blockIdx.z * zc;
    const int zend = min(z0 + zc, g.nz);
    const int64_t plane = (int64_t)g.nx * g.ny;
    const int ecx = x0 + tx - 1, ecy = y0 + ty - 1;
    const int onx = x0 + tx, ony = y0 + ty;
    const bool owner = (tx < MV_TX - 1) && (ty < MV_TY - 1) && onx < g.nx && ony < g.ny;
    const bool ecxy = ecx >= 0 && ecx < g.ex && ecy >= 0 && ecy < g.ey;
    const int eCol = ecy * g.nx + ecx;   // in-plane offsets fit in 32 bits for every accepted grid
    const int oCol = ony * g.nx + onx;
    const TC sc = TC(a.scale);
    // Extra tile slots: row MV_TY (ty == 0 threads), column MV_TX (row-1 threads tx <= MV_TY).
    const bool hasR = ty == 0, hasC = (ty == 1) && (tx <= MV_TY);
    const int rX = x0 - 1 + tx, rY = y0 - 1 + MV_TY;
    const int cX = x0 - 1 + MV_TX, cY = y0 - 1 + tx;
    const bool ok0 = ecx >= 0 && ecx < g.nx && ecy >= 0 && ecy < g.ny;
    const bool okR = hasR && rX >= 0 && rX < g.nx && rY >= 0 && rY < g.ny;
    const bool okC = hasC && cX >= 0 && cX < g.nx && cY >= 0 && cY < g.ny;
#define SU(b, iy, ix) (su + (((((b) * (MV_TY + 1)) + (iy)) * (MV_TX + 1) + (ix)) << 2))
#define SY(k, iy, ix) (sy + (((((k) * MV_TY) + (iy)) * MV_TX + (ix)) << 2))
    T pf[9];
    auto gload = [&](int zl) {
        const bool zok = zl >= 0 && zl < g.nz;
        const int64_t zoff = (int64_t)zl * plane;
#pragma unroll
        for (int i = 0; i < 9; ++i) pf[i] = T(0);
        if (ok0 && zok) {
            const T* p = a.x + 3 * ((int64_t)eCol + zoff);
            pf[0] = p[0]; pf[1] = p[1]; pf[2] = p[2];
        }
        if (okR && zok) {
            const T* p = a.x + 3 * ((int64_t)(rY * g.nx + rX) + zoff);
            pf[3] = p[0]; pf[4] = p[1]; pf[5] = p[2];
        }
        if (okC && zok) {
            const T* p = a.x + 3 * ((int64_t)(cY * g.nx + cX) + zoff);
            pf[6] = p[0]; pf[7] = p[1]; pf[8] = p[2];
        }
    };
    auto sstore = [&](int zl) {
        const int b = zl & 1;
        stSlot<TC>(SU(b, ty, tx), C::in(pf[0]), C::in(pf[1]), C::in(pf[2]));
        if (hasR) stSlot<TC>(SU(b, MV_TY, tx), C::in(pf[3]), C::in(pf[4]), C::in(pf[5]));
        if (hasC) stSlot<TC>(SU(b, tx, MV_TX), C::in(pf[6]), C::in(pf[7]), C::in(pf[8]));
    };
    auto eload = [&](int k) -> float {
        return (ecxy && k >= 0 && k < g.ez) ? a.E[(int64_t)eCol + (int64_t)k * plane] : 0.f;
    };
    auto fload = [&](int k) -> uint8_t {
        return (owner && k >= z0 && k < zend) ? a.flags[(int64_t)oCol + (int64_t)k * plane] : (uint8_t)0;
    };
    TC acc[3] = {TC(0), TC(0), TC(0)};
    gload(z0 - 1);
    sstore(z0 - 1);
    gload(z0);
    float Enext = eload(z0 - 1);
    uint8_t flNext = fload(z0 - 1);
    for (int k = z0 - 1; k < zend; ++k) {
        sstore(k + 1);
        const float Ee = Enext;
        const uint8_t fl = flNext;
        __syncthreads();
        gload(k + 2);           // consumed by the next iteration
        Enext = eload(k + 1);
        flNext = fload(k + 1);
        // x at the owned node of layer k, read now: the next iteration's store
        // overwrites this layer's buffer without waiting for the output phase.
        TC xo[3];
        ldSlot<TC>(SU(k & 1, ty + 1, tx + 1), xo[0], xo[1], xo[2]);
        TC ye[24];
        if (Ee != 0.f) {
            TC u[24];
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int dx = n & 1, dy = (n >> 1) & 1, dz = n >> 2;
                ldSlot<TC>(SU((k + dz) & 1, ty + dy, tx + dx), u[3 * n], u[3 * n + 1], u[3 * n + 2]);
            }
            elemDense<TC>(u, ye, kp, sc * TC(Ee));
        } else {
#pragma unroll
            for (int i = 0; i < 24; ++i) ye[i] = TC(0);
        }
        stSlot<TC>(SY(0, ty, tx), ye[0], ye[1], ye[2]);     // a = 0
        stSlot<TC>(SY(1, ty, tx), ye[3], ye[4], ye[5]);     // a = 1
        stSlot<TC>(SY(2, ty, tx), ye[6], ye[7], ye[8]);     // a = 2
        stSlot<TC>(SY(3, ty, tx), ye[12], ye[13], ye[14]);  // a = 4
        stSlot<TC>(SY(4, ty, tx), ye[15], ye[16], ye[17]);  // a = 5
        stSlot<TC>(SY(5, ty, tx), ye[18], ye[19], ye[20]);  // a = 6
        __syncthreads();
        if (owner) {
            TC lo[3], hi[3], q[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                lo[c] = ye[9 + c];
                hi[c] = ye[21 + c];
            }
            ldSlot<TC>(SY(2, ty, tx + 1), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) lo[c] += q[c];
            ldSlot<TC>(SY(1, ty + 1, tx), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) lo[c] += q[c];
            ldSlot<TC>(SY(0, ty + 1, tx + 1), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) lo[c] += q[c];
            ldSlot<TC>(SY(5, ty, tx + 1), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) hi[c] += q[c];
            ldSlot<TC>(SY(4, ty + 1, tx), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) hi[c] += q[c];
            ldSlot<TC>(SY(3, ty + 1, tx + 1), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) hi[c] += q[c];
            if (k >= z0) {
                TC sum[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) sum[c] = acc[c] + lo[c];
                mvOutput<T, TC>(a, (int64_t)oCol + (int64_t)k * plane, sum, fl, xo, d0, d1);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c] = hi[c];
        }
    }
#undef SU
#undef SY
}

// 4-point Walsh-Hadamard transform of a node quad (corner q = dx + 2 dy), per
// component: v[3m+c] = sum_q (-1)^popcount(m&q) u[3q+c].
template <typename T>
__device__ __forceinline__ void fwht4x3(T (&v)[12]) {
#pragma unroll
    for (int s = 1; s < 4; s <<= 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q & s) continue;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T p = v[3 * q + c], r = v[3 * (q + s) + c];
                v[3 * q + c] = p + r;
                v[3 * (q + s) + c] = p - r;
            }
        }
    }
}

// FP32: the x and y components of a node move as one register pair through
// the packed FP32x2 instructions (same IEEE results; p - r as fma(r, -1, p) is
// exact before its rounding), the z component alone: 2/3 of the instructions.
__device__ __forceinline__ float2 pr2(const float* v) { return make_float2(v[0], v[1]); }
__device__ __forceinline__ void st2(float* v, float2 a) {
    v[0] = a.x;
    v[1] = a.y;
}
__device__ __forceinline__ float2 sub2(float2 p, float2 r) { return __ffma2_rn(r, make_float2(-1.f, -1.f), p); }
__device__ __forceinline__ void bfly3(float* a, float* b) {
    const float2 p = pr2(a), r = pr2(b);
    st2(a, __fadd2_rn(p, r));
    st2(b, sub2(p, r));
    const float pz = a[2], rz = b[2];
    a[2] = pz + rz;
    b[2] = pz - rz;
}
template <>
__device__ __forceinline__ void fwht4x3<float>(float (&v)[12]) {
    bfly3(v, v + 3);
    bfly3(v + 6, v + 9);
    bfly3(v, v + 6);
    bfly3(v + 3, v + 9);
}

// uh = (qb + qt, qb - qt) (24 values).
template <typename T>
__device__ __forceinline__ void sumDiff12(const T (&a)[12], const T (&b)[12], T (&u)[24]) {
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        u[i] = a[i] + b[i];
        u[12 + i] = a[i] - b[i];
    }
}
template <>
__device__ __forceinline__ void sumDiff12<float>(const float (&a)[12], const float (&b)[12], float (&u)[24]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 p = pr2(a + 3 * q), r = pr2(b + 3 * q);
        st2(u + 3 * q, __fadd2_rn(p, r));
        st2(u + 12 + 3 * q, sub2(p, r));
        u[3 * q + 2] = a[3 * q + 2] + b[3 * q + 2];
        u[12 + 3 * q + 2] = a[3 * q + 2] - b[3 * q + 2];
    }
}
// u[i] *= e for the modes 1..7 (i >= 3).
template <typename T>
__device__ __forceinline__ void scaleModes(T (&u)[24], T e) {
#pragma unroll
    for (int i = 3; i < 24; ++i) u[i] *= e;
}
template <>
__device__ __forceinline__ void scaleModes<float>(float (&u)[24], float e) {
#pragma unroll
    for (int m = 1; m < 8; ++m) {
        st2(u + 3 * m, __fmul2_rn(pr2(u + 3 * m), make_float2(e, e)));
        u[3 * m + 2] *= e;
    }
}
template <typename T>
__device__ __forceinline__ void scaledKhat(T (&u)[24], T (&y)[24], const Ks<T>& k, T e) {
    scaleModes<T>(u, e);
    applyKhat<T>(u, y, k);
}
// nb = carry + (y_bottom + y_top); carry = y_bottom - y_top.
template <typename T>
__device__ __forceinline__ void foldCarry(const T (&y)[24], T (&carry)[12], T (&nb)[12]) {
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        nb[i] = carry[i] + (y[i] + y[12 + i]);
        carry[i] = y[i] - y[12 + i];
    }
}
template <>
__device__ __forceinline__ void foldCarry<float>(const float (&y)[24], float (&carry)[12], float (&nb)[12]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 yb = pr2(y + 3 * q), yt = pr2(y + 12 + 3 * q), cr = pr2(carry + 3 * q);
        st2(nb + 3 * q, __fadd2_rn(cr, __fadd2_rn(yb, yt)));
        st2(carry + 3 * q, sub2(yb, yt));
        const float zb = y[3 * q + 2], zt = y[12 + 3 * q + 2];
        nb[3 * q + 2] = carry[3 * q + 2] + (zb + zt);
        carry[3 * q + 2] = zb - zt;
    }
}

// The structured (isotropic cube) product with the Walsh-Hadamard factors
// shared along z.  With corner a = (q, dz) and mode m = (mq, mz), the 8-point
// transform splits into the 4-point transforms Q_0, Q_1 of the element's bottom
// and top node quads: uh[(mq,0)] = Q_0 + Q_1, uh[(mq,1)] = Q_0 - Q_1.  The top
// quad's transform of element layer k is the bottom one of layer k+1, so each
// quad is transformed once.  On the way back the top-face output of layer k-1
// and the bottom-face output of layer k land on the same node quad and are
// added in the Walsh domain before one inverse 4-point transform.  Per element
// this halves the shared-memory node reads (4 instead of 8), the exported
// contributions (3 instead of 6) and the quad transforms, against kMatvec.
// Same tile, pipelining and output stage as kMatvec.  The two Walsh-domain
// carries stay in registers across the z march.  Launch bounds, measured on
// the 256^3 workload: FP32 3 blocks per SM (80 registers, no spills; 4 blocks
// spill and run 33% slower); FP64 and df 2 blocks per SM (128 registers, a few
// spilled values; 20% faster than 1 block without spills).
//
// OUT selects the output stage at compile time (runtime mode switches in the
// owner stage cost ~20% of this issue-bound kernel):
//   OUT_ANY   mvOutput with the runtime mode and dots;
//   OUT_CG    the CG product: y = Kx (fixed rows 0), dot x.(Kx); a thread adds its nodes'
//             sums of three plainly, up to 47 layers in FP32 (productLayers): a chain of
//             50 roundings, where a term at a time had 96 in marches of 32;
//   OUT_TRUE  the true residual: r = f - Kx, its FP32 rounding to y32, y (FP64)
//             only when given, dot r.r;
//   OUT_CG_PX the CG product with the mixed solve's direction update fused into
//             the input stage: every staged node value is p = z + beta p_old
//             (halo copies computed the same way by every block that stages
//             them), and the thread that stages an owned node writes the new p
//             to the other p buffer and adds the deferred alpha p_old to the
//             FP32 solution correction.  The p buffers alternate (Scalars::pSel,
//             flipped by the last block), because neighbouring blocks still read
//             p_old as their halo.
enum MvOut : int { OUT_ANY = 0, OUT_CG = 1, OUT_TRUE = 2, OUT_CG_PX = 3 };

// The march of one block of 32 x 8 threads over its `layers` node layers: fills d0 and d1
// (this thread's dots) and returns the p buffer read (OUT_CG_PX).
template <typename T, typename TC, int OUT, typename KP>
__device__ __forceinline__ int walshMarch(const MatvecArgs<T>& a, const KP& kp, Scalars* S,
                                           unsigned char* smemRaw, DotAcc<TC>& d0, DotAcc<TC>& d1,
                                          [[maybe_unused]] int layers = MV_ZC) {
    typedef Cvt<T, TC> C;
    TC* su = reinterpret_cast<TC*>(smemRaw);
    TC* sy = su + kSuElems;
    const Grid g = a.g;
    const int zc = layers;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * (MV_TX - 1), y0 = blockIdx.y * (MV_TY - 1), z0 = blockIdx.z * zc;
    const int zend = min(z0 + zc, g.nz);
    const int64_t plane = (int64_t)g.nx * g.ny;
    const int ecx = x0 + tx - 1, ecy = y0 + ty - 1;
    const int onx = x0 + tx, ony = y0 + ty;
    const bool owner = (tx < MV_TX - 1) && (ty < MV_TY - 1) && onx < g.nx && ony < g.ny;
    const bool ecxy = ecx >= 0 && ecx < g.ex && ecy >= 0 && ecy < g.ey;
    const int eCol = ecy * g.nx + ecx;
    const int oCol = ony * g.nx + onx;
    const TC sc = TC(a.scale);
    const bool hasR = ty == 0, hasC = (ty == 1) && (tx <= MV_TY);
    const int rX = x0 - 1 + tx, rY = y0 - 1 + MV_TY;
    const int cX = x0 - 1 + MV_TX, cY = y0 - 1 + tx;
    const bool ok0 = ecx >= 0 && ecx < g.nx && ecy >= 0 && ecy < g.ny;
    const bool okR = hasR && rX >= 0 && rX < g.nx && rY >= 0 && rY < g.ny;
    const bool okC = hasC && cX >= 0 && cX < g.nx && cY >= 0 && cY < g.ny;
#define SU(b, iy, ix) (su + (((((b) * (MV_TY + 1)) + (iy)) * (MV_TX + 1) + (ix)) << 2))
#define SY(k, iy, ix) (sy + (((((k) * MV_TY) + (iy)) * MV_TX + (ix)) << 2))
    // Input source; OUT_CG_PX: p_old, the buffer for the new p, beta and the
    // deferred alpha (0 when a flush has folded it).  Every block reads the
    // scalars here, before it reaches the grid reduction after which the last
    // block flips pSel and advances matvecs.
    const T* src = a.x;
    T* pNew = nullptr;
    T beta = T(0), ax = T(0);
    int sel = 0;
    if constexpr (OUT == OUT_CG_PX) {
        sel = S->pSel;
        src = sel ? a.pAlt : a.x;
        pNew = sel ? const_cast<T*>(a.x) : a.pAlt;
        beta = T(S->beta);
        ax = S->foldStamp == S->matvecs ? T(0) : T(S->alpha);
        if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tx == 0 && ty == 0)
            S->pxStamp = S->matvecs;  // read only by kFlushX
    }
    // The thread that stages node (ecx, ecy) is the one after its owner in x and y.
    // OUT_CG_PX keeps the raw z, p_old (and, for an owned node, x) values of the
    // prefetched layer in registers and forms p = z + beta p_old when the layer
    // is staged to shared memory, so the prefetch stays in flight across the
    // element computation as in the plain product.
    const bool stagesOwned = OUT == OUT_CG_PX && tx >= 1 && ty >= 1;
    T pf[9];
    [[maybe_unused]] T pq[OUT == OUT_CG_PX ? 9 : 1], xq[OUT == OUT_CG_PX ? 3 : 1];
    auto ld3 = [&](int64_t i, int o) {
        pf[o] = src[i];
        pf[o + 1] = src[i + 1];
        pf[o + 2] = src[i + 2];
        if constexpr (OUT == OUT_CG_PX) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                pq[o + c] = pf[o + c];
                pf[o + c] = a.zin[i + c];
            }
        }
    };
    auto ownsLayer = [&](int zl) { return stagesOwned && ok0 && zl >= z0 && zl < zend; };
    auto gload = [&](int zl) {
        const bool zok = zl >= 0 && zl < g.nz;
        const int64_t zoff = (int64_t)zl * plane;
#pragma unroll
        for (int i = 0; i < 9; ++i) pf[i] = T(0);
        if constexpr (OUT == OUT_CG_PX) {
#pragma unroll
            for (int i = 0; i < 9; ++i) pq[i] = T(0);
        }
        if (ok0 && zok) {
            ld3(3 * ((int64_t)eCol + zoff), 0);
            if constexpr (OUT == OUT_CG_PX) {
                if (ax != T(0) && ownsLayer(zl)) {
                    const int64_t i = 3 * ((int64_t)eCol + zoff);
                    xq[0] = a.xacc[i];
                    xq[1] = a.xacc[i + 1];
                    xq[2] = a.xacc[i + 2];
                }
            }
        }
        if (okR && zok) ld3(3 * ((int64_t)(rY * g.nx + rX) + zoff), 3);
        if (okC && zok) ld3(3 * ((int64_t)(cY * g.nx + cX) + zoff), 6);
    };
    auto sstore = [&](int zl) {
        const int b = zl & 1;
        if constexpr (OUT == OUT_CG_PX) {
            if (beta != T(0)) {
#pragma unroll
                for (int i = 0; i < 9; ++i) pf[i] = fma(beta, pq[i], pf[i]);
            }
            if (ownsLayer(zl)) {
                const int64_t i = 3 * ((int64_t)eCol + (int64_t)zl * plane);
#pragma unroll
                for (int c = 0; c < 3; ++c) pNew[i + c] = pf[c];
                if (ax != T(0)) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) a.xacc[i + c] = fma(ax, pq[c], xq[c]);
                }
            }
        }
        stSlot<TC>(SU(b, ty, tx), C::in(pf[0]), C::in(pf[1]), C::in(pf[2]));
        if (hasR) stSlot<TC>(SU(b, MV_TY, tx), C::in(pf[3]), C::in(pf[4]), C::in(pf[5]));
        if (hasC) stSlot<TC>(SU(b, tx, MV_TX), C::in(pf[6]), C::in(pf[7]), C::in(pf[8]));
    };
    auto eload = [&](int k) -> float {
        return (ecxy && k >= 0 && k < g.ez) ? a.E[(int64_t)eCol + (int64_t)k * plane] : 0.f;
    };
    auto fload = [&](int k) -> uint8_t {
        return (owner && k >= z0 && k < zend) ? a.flags[(int64_t)oCol + (int64_t)k * plane] : (uint8_t)0;
    };
    // Walsh-domain quad of the current bottom node layer, and the top-face
    // output of the previous element layer (Walsh domain).
    TC qb[12], carry[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) carry[i] = TC(0);
    TC dAx = TC(0);  // OUT_CG: x.(Kx) of this thread
    gload(z0 - 1);
    sstore(z0 - 1);
    gload(z0);
    float Enext = eload(z0 - 1);
    uint8_t flNext = fload(z0 - 1);
    for (int k = z0 - 1; k < zend; ++k) {
        sstore(k + 1);
        const float Ee = Enext;
        const uint8_t fl = flNext;
        __syncthreads();
        gload(k + 2);
        Enext = eload(k + 1);
        flNext = fload(k + 1);
        TC xo[3];
        ldSlot<TC>(SU(k & 1, ty + 1, tx + 1), xo[0], xo[1], xo[2]);
        if (k == z0 - 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                ldSlot<TC>(SU(k & 1, ty + (q >> 1), tx + (q & 1)), qb[3 * q], qb[3 * q + 1], qb[3 * q + 2]);
            fwht4x3<TC>(qb);
        }
        TC qt[12];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            ldSlot<TC>(SU((k + 1) & 1, ty + (q >> 1), tx + (q & 1)), qt[3 * q], qt[3 * q + 1], qt[3 * q + 2]);
        fwht4x3<TC>(qt);
        TC nb[12];  // node layer k: Walsh-domain contributions at the element's bottom quad
        if (Ee != 0.f) {
            TC uh[24], yh[24];
            const TC e = sc * TC(Ee);
            sumDiff12<TC>(qb, qt, uh);
            scaledKhat<TC>(uh, yh, kp, e);
            foldCarry<TC>(yh, carry, nb);
        } else {
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                nb[i] = carry[i];
                carry[i] = TC(0);
            }
        }
#pragma unroll
        for (int i = 0; i < 12; ++i) qb[i] = qt[i];
        fwht4x3<TC>(nb);
        stSlot<TC>(SY(0, ty, tx), nb[0], nb[1], nb[2]);  // corner (0,0)
        stSlot<TC>(SY(1, ty, tx), nb[3], nb[4], nb[5]);  // corner (1,0)
        stSlot<TC>(SY(2, ty, tx), nb[6], nb[7], nb[8]);  // corner (0,1)
        __syncthreads();
        if (owner && k >= z0) {
            TC sum[3] = {nb[9], nb[10], nb[11]}, q[3];  // own corner (1,1)
            ldSlot<TC>(SY(2, ty, tx + 1), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) sum[c] += q[c];
            ldSlot<TC>(SY(1, ty + 1, tx), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) sum[c] += q[c];
            ldSlot<TC>(SY(0, ty + 1, tx + 1), q[0], q[1], q[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) sum[c] += q[c];
            const int64_t s = (int64_t)oCol + (int64_t)k * plane;
            if constexpr (OUT == OUT_CG || OUT == OUT_CG_PX) {
                const bool fixed = (fl & FLAG_FIXED) != 0;
                // FP64: x is the caller's (vfem_apply_operator_device_noalloc) and may hold anything
                // at unused nodes; the FP32 solver's own vectors hold 0 there and at fixed nodes
                const bool live = std::is_same<T, float>::value || ((fl & FLAG_USED) && !fixed);
                TC node = TC(0);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const TC out = fixed ? TC(0) : sum[c];
                    a.y[3 * s + c] = C::out(out);
                    node = c == 0 ? xo[c] * out : fma(xo[c], out, node);
                }
                if (live) dAx += node;
            } else if constexpr (OUT == OUT_TRUE) {
                const bool fixed = (fl & FLAG_FIXED) != 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const TC out = C::in(a.f[3 * s + c]) - (fixed ? TC(0) : sum[c]);
                    if (a.y) a.y[3 * s + c] = C::out(out);
                    a.y32[3 * s + c] = toF(out);
                    d0.add(out * out);
                }
            } else {
                mvOutput<T, TC>(a, s, sum, fl, xo, d0, d1);
            }
        }
    }
#undef SU
#undef SY
    if constexpr (OUT == OUT_CG || OUT == OUT_CG_PX) d0.add(dAx);
    return sel;
}

}  // namespace
}  // namespace vfem
