// matvec_fx.cu -- the FP64 product in block fixed point.
//
// Two forms: the cube's 8 constants in the Walsh basis, and the dense 24 x 24 matrix
// for a Ke in another corner order (which matrices: fxPrepare).
//
// GB300 issues FP64 at 1/64 of its FP32 rate: measured 1.7 FP64 operations per
// clock and SM against 58 64-bit integer additions and 29 multiply-adds 32 x 32
// -> 64.  The FP64 marches (walshMarch and denseMarch, matvec_march.cuh) are
// bound by their ~190 and ~600 FP64 operations per element.  This kernel does
// the same element products in 64-bit integers and leaves three conversions and
// the dot of a node to the FP64 pipe.
//
// Measured: 191^3 with voids and log-normal moduli 3.72 -> 0.49 ms; 33 x 17 x 17
// nodes 262 -> 20 us (shorter marches by marchLayers among it); a Ke in another
// corner order, as the dense 24 x 24 product, 96 x 80 x 72 half full, 1.56 ->
// 0.26 ms.  Bound now: instruction issue (1,100 warp instructions per element
// row, 59% of the issue slots, ALU 56%, wide multiply-adds 54% of their pipe)
// with two 8-warp blocks per SM for their registers; the dense form by its 1,728
// wide multiply-adds an element.  Cube tiles of 12 rows in one block per SM (168
// registers) or of 6 rows in two measured 14% slower; the dense form with two
// blocks per SM (128 registers, 240 bytes spilled) the same as with one.
//
// Numbers.  A node's three components are staged as 58-bit integers under the
// node's largest exponent.  An element reads its 24 values on a grid S with
// S - 3 <= (exponent of its largest value) <= S (dense: S) and 2^-57 of 2^S as the
// unit; the Walsh transforms are then exact.  The largest of the 20 combinations that
// Khat scales is shifted up to 2^61..2^62 (lz), multiplied by 62-bit constants
// in two 32-bit digits, and by the modulus' 24-bit significand, with rounding;
// what leaves the element has the unit 2^(O + 9 - f), O = S + exponent(E) - lz,
// at most 2^-56 of C E times that largest combination (C, f: fxPrepare).
// Outputs with different O are aligned to the larger one where they meet.
// Against 113-bit arithmetic the result's relative error is 3e-16 to 6e-16
// (random, smooth, graded and point vectors, moduli 1, log-normal or spread
// over e^20), where the FP64 march has 5e-16 to 4e-15; the dense form's, for the
// matrices it takes, 5e-17 to 8e-16, where the FP64 one has 1e-16 to 2.5e-15.
//
// The common grid cuts off what components have below 2^-57 of the largest value.  FP64
// rounds its Walsh sums there as well (x = 1e6 + random beside random y and z: 2e-12
// relative, FP64 1.2e-11), unless that component sums without rounding, as a rigid
// translation does (x = 1e6: 2e-12 against 1e-16).  A block with an element whose largest
// combination is below 2^43 units (2^-18 of the grid's top) therefore looks at its elements
// again (fxRepeat) and repeats in FP64 for such components; otherwise the cut-offs, up to 48
// units, stay below 2^-37 of the largest combination, typically 2^-41.  191^3 492 us and
// a 64^3 FP64 solve 117.9 ms, as without; FP64 solves of slender beams (512 x 16 x 16) 2% slower,
// 5% with 2^-16; with 2^-14 the 64^3 solve 3%.  The march is at its 128 registers: noted in
// another form the same test spilled there (191^3 532 us).
//
// No sum overflows.  Staged values are below 2^58 (S = the largest exponent), modes below
// 2^61, sums of two below 2^62, of three below 3 x 2^61; where lz > 0 all are below 2^62.  A
// component's corner value is then at most C 2^f (3 x 2^61) / 2^64 / 2 <= 3 x 2^58 per element,
// a node's 8 of them 3 x 2^61; sums in between are taken modulo 2^64.  A middle digit
// sum has one product with k0 (at most 2^30 2^31) and one with k1 (with its start in
// kb at most 2^32 |k1|, |k1| <= 2^30); the threes' has two of each, fxPrepare checks
// their constants; the dense form's 24, hence its coarser k0.  Values the grid cannot take
// (non-finite ones or exponents beyond 2^+-575 next to a filled voxel, subnormal
// moduli) make the block repeat its march in FP64, so that results for those
// are what the FP64 march gives.
#include <cmath>
#include <cstring>

#include "matvec_march.cuh"

namespace vfem {

namespace {

constexpr int FX_EMIN = 448, FX_EMAX = 1600;  // biased exponents the integer march takes
constexpr int FX_BAD = 4000;                  // a node outside of them
constexpr int FX_NONE = -(1 << 20);           // exponent of a zero contribution
constexpr int FX_SLACK = 3;
constexpr int FX_FAR = 18;                    // combinations below 2^-18 of the grid: fxRepeat looks closer

// Constants times 2^f = k1 2^32 + k0, signed digits.  kb: start of a middle digit
// sum, 2^31 (rounding) + 2^31 k1.
struct FxArgs {        // the cube's 8 constants (cubeConstants)
    long long kb[8];
    int k1[8], k0[8];
    int scaleExp;      // log2 of the level's operator scale
    int outExp;        // exponent-field offset of an output at O
};
struct FxDenseArgs {   // Ke, row-major; k0 in units of 2^3, so that 24 of its products fit their sum
    long long kb[24];
    int k1[576], k0[576];
    int scaleExp, outExp;
};

struct FxNode {
    long long v[3];
    int e;
};

// Three FP64 components on their common grid.
__device__ __forceinline__ FxNode fxNode(double x, double y, double z) {
    const double d[3] = {x, y, z};
    FxNode n;
    int e = 0, ec[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        ec[c] = (__double2hiint(d[c]) >> 20) & 0x7ff;
        e = max(e, ec[c]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int hi = __double2hiint(d[c]);
        const unsigned long long m =
            (((unsigned long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(d[c])) << 5;
        // a zero or subnormal component (field 0) is shifted out: e >= FX_EMIN below
        const unsigned long long q = m >> min(e - ec[c], 63);
        const long long s = (long long)(hi >> 31);
        n.v[c] = ((long long)q ^ s) - s;
    }
    if ((unsigned)(e - FX_EMIN) > (unsigned)(FX_EMAX - FX_EMIN)) {
        const bool zero = (((__double2hiint(x) | __double2hiint(y) | __double2hiint(z)) & 0x7fffffff) |
                           __double2loint(x) | __double2loint(y) | __double2loint(z)) == 0;
        n.v[0] = n.v[1] = n.v[2] = 0;
        e = zero ? 0 : FX_BAD;
    }
    n.e = e;
    return n;
}

__device__ __forceinline__ long long fxShr(long long v, int by) { return v >> (int)min((unsigned)by, 63u); }

__device__ __forceinline__ void fwht4x3i(long long (&v)[12]) {
#pragma unroll
    for (int s = 1; s < 4; s <<= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q & s) continue;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long p = v[3 * q + c], r = v[3 * (q + s) + c];
                v[3 * q + c] = p + r;
                v[3 * (q + s) + c] = p - r;
            }
        }
}

template <int TY>
constexpr size_t fxSmemBytes() {
    // staged nodes (two layers) and exported corners (three), 32 bytes each; the
    // FP64 march of a block that falls back uses the same memory
    constexpr size_t fx = 32 * (2 * (size_t)(TY + 1) * (MV_TX + 1) + 3 * (size_t)TY * MV_TX);
    constexpr size_t fp = (size_t)(kSuElems + kSyElems) * sizeof(double);
    return fx > fp ? fx : fp;
}

// One block's march, the counterpart of walshMarch<double, double, OUT> (KA =
// FxArgs) and denseMarch<double, double> (FxDenseArgs) with the same tile, halo
// and pipelining.  Returns true when a value did not fit, so that the outputs and dots are to be
// recomputed, or an element's strains were small against its grid: fxAgain finds out.  The
// dense form has the 24 values themselves in place of the Walsh combinations and reads both
// quads every layer, to keep their digits in registers.
template <int OUT, int TY, typename KA>
__device__ __forceinline__ bool fxMarch(const MatvecArgs<double>& a, const KA& K, int zc, unsigned char* smem,
                                        DotAcc<double>& d0, DotAcc<double>& d1) {
    constexpr bool DENSE = std::is_same<KA, FxDenseArgs>::value;
    // 16-byte halves of the 32-byte slots in arrays of their own: conflict-free
    longlong2* suA = reinterpret_cast<longlong2*>(smem);           // {v0, v1}
    longlong2* suB = suA + 2 * (TY + 1) * (MV_TX + 1);             // {v2, exponent}
    longlong2* syA = suB + 2 * (TY + 1) * (MV_TX + 1);
    longlong2* syB = syA + 3 * TY * MV_TX;
    const Grid g = a.g;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * (MV_TX - 1), y0 = blockIdx.y * (TY - 1), z0 = blockIdx.z * zc;
    const int zend = min(z0 + zc, g.nz);
    const int64_t plane = (int64_t)g.nx * g.ny;
    const int ecx = x0 + tx - 1, ecy = y0 + ty - 1;
    const int onx = x0 + tx, ony = y0 + ty;
    const bool owner = (tx < MV_TX - 1) && (ty < TY - 1) && onx < g.nx && ony < g.ny;
    const bool ecxy = ecx >= 0 && ecx < g.ex && ecy >= 0 && ecy < g.ey;
    const int eCol = ecy * g.nx + ecx, oCol = ony * g.nx + onx;
    // the tile's extra row (ty == 0 threads) and column (row-1 threads): at most one extra node a thread
    const bool hasR = ty == 0, hasC = (ty == 1) && (tx <= TY);
    const int exX = hasR ? x0 - 1 + tx : x0 - 1 + MV_TX, exY = hasR ? y0 - 1 + TY : y0 - 1 + tx;
    const int exSlot = hasR ? TY * (MV_TX + 1) + tx : tx * (MV_TX + 1) + MV_TX;
    const bool hasX = hasR || hasC;
    const bool ok0 = ecx >= 0 && ecx < g.nx && ecy >= 0 && ecy < g.ny;
    const bool okX = hasX && exX >= 0 && exX < g.nx && exY >= 0 && exY < g.ny;
    const int exCol = exY * g.nx + exX;
#define SLOT(b, iy, ix) (((b) * (TY + 1) + (iy)) * (MV_TX + 1) + (ix))
#define YSLOT(k, iy, ix) (((k) * TY + (iy)) * MV_TX + (ix))
    double pf[6];
    auto gload = [&](int zl) {
        const bool zok = zl >= 0 && zl < g.nz;
        const int64_t zoff = (int64_t)zl * plane;
#pragma unroll
        for (int i = 0; i < 6; ++i) pf[i] = 0.0;
        if (ok0 && zok) {
            const double* p = a.x + 3 * ((int64_t)eCol + zoff);
            pf[0] = p[0]; pf[1] = p[1]; pf[2] = p[2];
        }
        if (okX && zok) {
            const double* p = a.x + 3 * ((int64_t)exCol + zoff);
            pf[3] = p[0]; pf[4] = p[1]; pf[5] = p[2];
        }
    };
    auto put = [&](int slot, const FxNode& n) {
        suA[slot] = make_longlong2(n.v[0], n.v[1]);
        suB[slot] = make_longlong2(n.v[2], n.e);
    };
    auto sstore = [&](int zl) {
        const int b = zl & 1;
        put(SLOT(b, ty, tx), fxNode(pf[0], pf[1], pf[2]));
        if (hasX) put(SLOT(b, 0, 0) + exSlot, fxNode(pf[3], pf[4], pf[5]));
    };
    auto eload = [&](int k) -> float {
        return (ecxy && k >= 0 && k < g.ez) ? a.E[(int64_t)eCol + (int64_t)k * plane] : 0.f;
    };
    auto fload = [&](int k) -> uint8_t {
        return (owner && k >= z0 && k < zend) ? a.flags[(int64_t)oCol + (int64_t)k * plane] : (uint8_t)0;
    };
    // A staged node layer's quad: the second halves of its slots, the largest exponent ...
    auto quadB = [&](int b, longlong2 (&vb)[4]) {
        int e = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            vb[q] = suB[SLOT(b, ty + (q >> 1), tx + (q & 1))];
            e = max(e, (int)vb[q].y);
        }
        return e;
    };
    // ... and its Walsh transform on the grid S.
    auto quad = [&](int b, int S, const longlong2 (&vb)[4], long long (&v)[12]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const longlong2 va = suA[SLOT(b, ty + (q >> 1), tx + (q & 1))];
            const int by = S - (int)vb[q].y;
            v[3 * q] = fxShr(va.x, by);
            v[3 * q + 1] = fxShr(va.y, by);
            v[3 * q + 2] = fxShr(vb[q].x, by);
        }
        if constexpr (!DENSE) fwht4x3i(v);
    };
    long long qb[12], carry[12];  // bottom quad and the previous element's top-face output (Walsh domain)
#pragma unroll
    for (int i = 0; i < 12; ++i) qb[i] = carry[i] = 0;
    int S = 0, qS = -1, eb = 0, cO = FX_NONE;  // grid, the grid qb is on (-1: none), exponent of qb, of the carry
    bool bad = false;
    double dAx = 0.0;
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
        if (k == z0 - 1) {
            longlong2 vb[4];
            eb = quadB(k & 1, vb);
        }
        longlong2 vt[4];
        const int et = quadB((k + 1) & 1, vt), el = max(eb, et);
        const int eBits = __float_as_int(Ee);
        bool act = Ee != 0.f && el != 0;
        if (act && (el > FX_EMAX || (eBits >> 23) == 0)) {
            bad = true;
            act = false;
        }
        long long nb[12];
        int nO = cO;
        if (__any_sync(0xffffffffu, act)) {
            if constexpr (DENSE) {
                if (act) S = el;  // no quad is carried, so the finest grid each time
            } else if (act && (el > S || S > el + FX_SLACK || qS != S)) {
                longlong2 vb[4];
                quadB(k & 1, vb);
                S = el + 1;
                quad(k & 1, S, vb, qb);
            }
            long long qt[12], y[24];
            quad((k + 1) & 1, S, vt, qt);
            qS = et <= S ? S : -1;
            const unsigned m = act ? (unsigned)((eBits & 0x7fffff) | 0x800000) << 7 : 0u;
            // times the modulus, rounded
            auto scaled = [&](long long A, long long B) {
                const long long y1 = A + (B >> 32);
                const unsigned long long lo = (unsigned long long)(unsigned)y1 * m + 0x80000000ull;
                return (long long)(int)(y1 >> 32) * (int)m + (long long)(lo >> 32);
            };
            auto spread = [](long long w) {
                const int h = (int)(w >> 32);
                return (unsigned)(h ^ (h >> 31));
            };
            // w 2^lz = w1 2^32 + w0 + 2^31
            auto digits = [](long long w, int lz, int& w1, int& w0) {
                w1 = (int)__funnelshift_l((unsigned)w, (unsigned)(w >> 32), lz);
                w0 = (int)(((unsigned)w << lz) ^ 0x80000000u);
            };
            if constexpr (DENSE) {
                longlong2 vb[4];
                quadB(k & 1, vb);
                quad(k & 1, S, vb, qb);
                unsigned mag = 0;
#pragma unroll
                for (int i = 0; i < 12; ++i) mag |= spread(qb[i]) | spread(qt[i]);
                const int lz = max(__clz((int)mag) - 2, 0);
                cO = act ? S + (eBits >> 23) + K.scaleExp - lz : FX_NONE;
                int u1[24], u0[24];
#pragma unroll
                for (int i = 0; i < 12; ++i) {
                    digits(qb[i], lz, u1[i], u0[i]);
                    digits(qt[i], lz, u1[12 + i], u0[12 + i]);
                }
#pragma unroll
                for (int r = 0; r < 24; ++r) {
                    long long A = 0, B = K.kb[r], B3 = 0;
#pragma unroll
                    for (int c = 0; c < 24; ++c) {
                        A += (long long)u1[c] * K.k1[24 * r + c];
                        B += (long long)u0[c] * K.k1[24 * r + c];
                        B3 += (long long)u1[c] * K.k0[24 * r + c];
                    }
                    y[r] = scaled(A + (B3 >> 29), B);
                }
            } else {
                // The 20 combinations of the modes 1..7 that the cube's Khat scales (FxArgs).
                long long v[20];
                {
                    long long u[24];
#pragma unroll
                    for (int i = 0; i < 12; ++i) {
                        u[i] = qb[i] + qt[i];
                        u[12 + i] = qb[i] - qt[i];
                        qb[i] = qt[i];
                    }
                    v[0] = u[3]; v[1] = u[7]; v[2] = u[14]; v[3] = u[3] + u[7] + u[14];
                    v[4] = u[6] + u[4]; v[5] = u[12] + u[5]; v[6] = u[13] + u[8];
                    v[7] = u[23]; v[8] = u[22]; v[9] = u[21];
                    v[10] = u[10] + u[17]; v[11] = u[10] - u[17];
                    v[12] = u[9] + u[20]; v[13] = u[9] - u[20];
                    v[14] = u[15] + u[19]; v[15] = u[15] - u[19];
                    v[16] = u[18]; v[17] = u[16]; v[18] = u[11]; v[19] = u[18] + u[16] + u[11];
                }
                unsigned mag = 0;
#pragma unroll
                for (int i = 0; i < 20; ++i) mag |= spread(v[i]);
                if (mag < (1u << (29 - FX_FAR))) bad = bad || act;  // (in this form: no spills)
                const int lz = max(__clz((int)mag) - 2, 0);
                cO = act ? S + (eBits >> 23) + K.scaleExp - lz : FX_NONE;
                // k_j v 2^lz in 2^64 units as a leading (A) and a middle digit sum (B)
                auto mul = [&](long long w, int j, long long& A, long long& B) {
                    int v1, v0;
                    digits(w, lz, v1, v0);
                    A += (long long)v1 * K.k1[j];
                    B += (long long)v1 * K.k0[j] + (long long)v0 * K.k1[j];
                };
                auto one = [&](long long w, int j) {
                    long long A = 0, B = K.kb[j];
                    mul(w, j, A, B);
                    return scaled(A, B);
                };
                y[0] = y[1] = y[2] = 0;
                // a common part of three outputs plus each one's own
                auto three = [&](int at, int j, long long& ya, long long& yb, long long& yc) {
                    long long As = 0, Bs = K.kb[j] + K.kb[j + 1] - 0x80000000ll;
                    mul(v[at + 3], j + 1, As, Bs);
                    long long A = As, B = Bs;
                    mul(v[at], j, A, B);
                    ya = scaled(A, B);
                    A = As, B = Bs;
                    mul(v[at + 1], j, A, B);
                    yb = scaled(A, B);
                    mul(v[at + 2], j, As, Bs);
                    yc = scaled(As, Bs);
                };
                three(0, 0, y[3], y[7], y[14]);
                y[6] = y[4] = one(v[4], 2);
                y[12] = y[5] = one(v[5], 2);
                y[13] = y[8] = one(v[6], 2);
                y[23] = one(v[7], 3);
                y[22] = one(v[8], 3);
                y[21] = one(v[9], 3);
                auto two = [&](int at, long long& ya, long long& yb) {
                    const long long sum = one(v[at], 4), dif = one(v[at + 1], 5);
                    ya = sum + dif;
                    yb = sum - dif;
                };
                two(10, y[10], y[17]);
                two(12, y[9], y[20]);
                two(14, y[15], y[19]);
                three(16, 6, y[18], y[16], y[11]);
            }
            // fold with the carry on the coarser of the two units
            const int mO = max(nO, cO), sc = mO - nO, sy = mO - cO;
            nO = mO;
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                nb[i] = fxShr(carry[i], sc) + fxShr(DENSE ? y[i] : y[i] + y[12 + i], sy);
                carry[i] = DENSE ? y[12 + i] : y[i] - y[12 + i];
            }
        } else {
            qS = -1;
            cO = FX_NONE;
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                nb[i] = carry[i];
                carry[i] = 0;
            }
        }
        eb = et;
        // x or f at the owned node, in flight across the transform and the barrier
        double xo[3] = {0.0, 0.0, 0.0}, fo[3] = {0.0, 0.0, 0.0};
        if (owner && k >= z0) {
            const int64_t i = 3 * ((int64_t)oCol + (int64_t)k * plane);
            if (OUT == OUT_TRUE) {
                const double* p = a.f + i;
                fo[0] = p[0]; fo[1] = p[1]; fo[2] = p[2];
            } else if (OUT == OUT_CG || a.mode == MV_SMOOTH || a.dot0 == DOT_X_OUT) {
                const double* p = a.x + i;
                xo[0] = p[0]; xo[1] = p[1]; xo[2] = p[2];
            }
        }
        if constexpr (!DENSE) fwht4x3i(nb);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            syA[YSLOT(q, ty, tx)] = make_longlong2(nb[3 * q], nb[3 * q + 1]);
            syB[YSLOT(q, ty, tx)] = make_longlong2(nb[3 * q + 2], nO);
        }
        __syncthreads();
        if (owner && k >= z0) {
            const int64_t s = (int64_t)oCol + (int64_t)k * plane;
            const longlong2 a1 = syA[YSLOT(2, ty, tx + 1)], b1 = syB[YSLOT(2, ty, tx + 1)];
            const longlong2 a2 = syA[YSLOT(1, ty + 1, tx)], b2 = syB[YSLOT(1, ty + 1, tx)];
            const longlong2 a3 = syA[YSLOT(0, ty + 1, tx + 1)], b3 = syB[YSLOT(0, ty + 1, tx + 1)];
            const int o1 = (int)b1.y, o2 = (int)b2.y, o3 = (int)b3.y;
            const int o = max(max(nO, o1), max(o2, o3));
            const long long t[3] = {
                fxShr(nb[9], o - nO) + fxShr(a1.x, o - o1) + fxShr(a2.x, o - o2) + fxShr(a3.x, o - o3),
                fxShr(nb[10], o - nO) + fxShr(a1.y, o - o1) + fxShr(a2.y, o - o2) + fxShr(a3.y, o - o3),
                fxShr(nb[11], o - nO) + fxShr(b1.x, o - o1) + fxShr(b2.x, o - o2) + fxShr(b3.x, o - o3)};
            double sum[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double r = __ll2double_rn(t[c]);
                sum[c] = t[c] == 0 ? 0.0
                                   : __hiloint2double(__double2hiint(r) + ((o + K.outExp) << 20), __double2loint(r));
            }
            if constexpr (OUT == OUT_CG) {
                // (x at unused nodes may be anything: it must not reach the dot)
                const bool fixed = (fl & FLAG_FIXED) != 0, live = (fl & FLAG_USED) && !fixed;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double out = fixed ? 0.0 : sum[c];
                    a.y[3 * s + c] = out;
                    if (live) dAx = fma(xo[c], out, dAx);
                }
            } else if constexpr (OUT == OUT_TRUE) {
                const bool fixed = (fl & FLAG_FIXED) != 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double out = fo[c] - (fixed ? 0.0 : sum[c]);
                    if (a.y) a.y[3 * s + c] = out;
                    a.y32[3 * s + c] = (float)out;
                    d0.add(out * out);
                }
            } else {
                mvOutput<double, double>(a, s, sum, fl, xo, d0, d1);
            }
        }
    }
#undef SLOT
#undef YSLOT
    if constexpr (OUT == OUT_CG) d0.add(dAx);
    return bad;
}

// The block's march in FP64, out of line: its registers must not weigh on the integer march.
template <int OUT>
__device__ __noinline__ void fp64March(const MatvecArgs<double>* a, const Ks<double>* kp, int zc, Scalars* S,
                                       unsigned char* smem, DotAcc<double>* d) {
    d[0] = d[1] = DotAcc<double>();
    walshMarch<double, double, OUT, Ks<double>>(*a, *kp, S, smem, d[0], d[1], zc);
}
template <int OUT>
__device__ __noinline__ void fp64March(const MatvecArgs<double>* a, const Kd<double>* kp, int zc, Scalars*,
                                       unsigned char* smem, DotAcc<double>* d) {
    d[0] = d[1] = DotAcc<double>();
    denseMarch<double, double>(*a, *kp, smem, d[0], d[1], zc);
}

// Whether the block is to repeat its march in FP64 for one of this thread's elements: a value
// or modulus that the grid cannot take, or digits that FP64 keeps and the grid cuts off: a
// component whose FP64 sums are exact (the same value at all corners, or values of few bits) is
// large, and another has digits below the grid's unit.  Components that FP64 rounds at the
// same place (the usual case) are no reason.
__device__ __noinline__ bool fxRepeat(const MatvecArgs<double>* a, int zc) {
    const Grid g = a->g;
    const int ex = (int)blockIdx.x * (MV_TX - 1) + (int)threadIdx.x - 1;
    const int ey = (int)blockIdx.y * (MV_TY - 1) + (int)threadIdx.y - 1;
    const int z0 = blockIdx.z * zc;
    if (ex < 0 || ex >= g.ex || ey < 0 || ey >= g.ey) return false;
    for (int k = max(z0 - 1, 0); k < min(z0 + zc, g.ez); ++k) {
        const float E = a->E[g.store(ex, ey, k)];
        if (E == 0.f) continue;
        long long first[3];
        bool equal[3] = {true, true, true};
        int e[3] = {0, 0, 0}, lo[3] = {1 << 20, 1 << 20, 1 << 20};  // exponents: largest value, lowest digit
        bool zero = true;
        for (int q = 0; q < 8; ++q) {
            int node = 0;
            bool any = false;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long v =
                    __double_as_longlong(a->x[3 * g.store(ex + (q & 1), ey + ((q >> 1) & 1), k + (q >> 2)) + c]);
                if (q == 0) first[c] = v;
                equal[c] = equal[c] && v == first[c];
                if ((v << 1) == 0) continue;
                any = true;
                const int ev = (int)(v >> 52) & 0x7ff;
                node = max(node, ev);
                e[c] = max(e[c], ev);
                lo[c] = min(lo[c], ev - 53 + __ffsll((v & 0xfffffffffffffll) | 0x10000000000000ll));
            }
            if (any && (node < FX_EMIN || node > FX_EMAX)) return true;
            zero = zero && !any;
        }
        if (!zero && (__float_as_int(E) >> 23) == 0) return true;
        int top = 0, rounded = 0, low = 1 << 20;  // largest, largest that FP64 rounds, lowest digit
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            top = max(top, e[c]);
            if (equal[c]) continue;
            low = min(low, lo[c]);
            if (lo[c] < e[c] - 49) rounded = max(rounded, e[c]);  // sums of 8 take more than 53 bits
        }
        if (low < top + FX_SLACK - 57 && rounded + 6 < top) return true;
    }
    return false;
}

template <int OUT, typename KP>
__device__ __noinline__ void fxAgain(const MatvecArgs<double>* a, const KP* kp, int zc, Scalars* S,
                                     unsigned char* smem, DotAcc<double>* d) {
    if (__syncthreads_or(fxRepeat(a, zc))) fp64March<OUT>(a, kp, zc, S, smem, d);
}

constexpr int FX_TY = MV_TY;

template <int OUT, typename KA, typename KP>
__global__ void __launch_bounds__(MV_TX* FX_TY, std::is_same<KA, FxArgs>::value ? 2 : 1)
    kMatvecFx(const __grid_constant__ MatvecArgs<double> a, const __grid_constant__ KA K,
              const __grid_constant__ KP kp, int zc, Scalars* S, RedBuf rb) {
    if (a.checkDone && S->done) return;
    if (a.condTrue && !trueResidualDue(S)) return;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    DotAcc<double> d[2];
    if (__syncthreads_or(fxMarch<OUT, FX_TY>(a, K, zc, smemRaw, d[0], d[1])))
        fxAgain<OUT, KP>(&a, &kp, zc, S, smemRaw, d);
    if (a.epi != EPI_NONE) {
        double v[2] = {d[0].get(), d[1].get()}, t[2];
        if (gridReduce<MV_TX * FX_TY, 2>(v, rb, t)) applyEpi(a.epi, S, t[0], t[1]);
    }
}

}  // namespace

namespace {
// Digits and f of k[0..n), k0 in units of 2^low.  C: a bound of the sum of |k|
// over what one node component collects from an element.
bool fxDigits(const double* k, int n, double C, int low, int32_t* k1, int32_t* k0, int& outExp) {
    if (!(C > 0.0) || !std::isfinite(C)) return false;
    int e = 0;
    std::frexp(C, &e);  // C <= 2^e
    if (std::abs(e) > 150) return false;
    const int f = 62 - e;
    for (int i = 0; i < n; ++i) {
        const long long v = std::llrint(std::ldexp(k[i], f));
        const int32_t rest = (int32_t)(uint32_t)(v & 0xffffffffll);
        k1[i] = (int32_t)((v - rest) >> 32);
        k0[i] = low ? (int32_t)std::lrint(std::ldexp((double)rest, -low)) : rest;
    }
    // field of 2^(S' + E' + 9 - f) with S' and E' the unbiased exponents of S and E
    outExp = 9 - f - 1023 - 127;
    return true;
}

// The middle digit sum of `three` for constants j and j + 1: the common product with j + 1
// of up to 3 x 2^61 beside an own one of 2^61, or both of 2^62 (digits of 2^32).
bool threeFits(const FxOperand& op, int j) {
    const double own = std::fabs((double)op.k0[j]), sum = std::fabs((double)op.k0[j + 1]);
    const double lead = std::fabs((double)op.k1[j]) + std::fabs((double)op.k1[j + 1]);
    const double w = 0x1p30 + 1.0;
    return std::fmax(1.5 * w * sum + 0.5 * w * own, w * (sum + own)) + 0x1p32 * lead + 0x1p31 < 0x1p63;
}
}  // namespace

// Khat of a cube, whose axes are interchangeable, has one constant per kind of
// entry (a: diagonal, b: off-diagonal): normal strains (a, b), in-plane shears
// (a = b: a rotation has no energy), bending pairs (a, b), the mode-7 terms and
// the (1,1,1)-class triples (a, b).  Rows then need 20 products instead of 45:
// a u_i + b (u_j + u_k) = (a - b) u_i + b (u_i + u_j + u_k), and a pair's sum and
// difference scale by a + b and a - b, halved when they are recombined.
bool cubeConstants(const KeData& ke, double (&k)[8], double& C) {
    if (!ke.structured) return false;
    static const int kind[45] = {0, 1, 1, 1, 0, 1, 1, 1, 0, 2, 2, 2, 2, 3, 2, 2, 2, 2, 3, 2, 2, 2, 2,
                                 3, 4, 5, 5, 4, 4, 5, 5, 4, 4, 5, 5, 4, 6, 7, 7, 7, 6, 7, 7, 7, 6};
    double c[8] = {}, cnt[8] = {}, top = 0.0;
    for (int n = 0; n < 45; ++n) {
        c[kind[n]] += ke.ks[n];
        cnt[kind[n]] += 1.0;
        top = std::fmax(top, std::fabs(ke.ks[n]));
    }
    for (int i = 0; i < 8; ++i) c[i] /= cnt[i];
    for (int n = 0; n < 45; ++n)  // equal up to the rounding of Khat itself
        if (!(std::fabs(ke.ks[n] - c[kind[n]]) <= 1e-15 * top)) return false;
    const double v[8] = {c[0] - c[1], c[1], c[2], c[3], 0.5 * (c[4] + c[5]), 0.5 * (c[4] - c[5]), c[6] - c[7], c[7]};
    for (int i = 0; i < 8; ++i) k[i] = v[i];
    // a component's rows: one normal strain, two shears, one mode-7 term, two of pairs, one of a triple
    C = std::fabs(k[0]) + std::fabs(k[1]) + 2 * std::fabs(k[2]) + std::fabs(k[3]) +
        2 * (std::fabs(k[4]) + std::fabs(k[5])) + std::fabs(k[6]) + std::fabs(k[7]);
    return true;
}

// The integer forms round every constant to one unit and every value of an element to
// one grid.  For a cube that is what the FP64 march's Walsh transforms do as well, and
// the constants themselves are sums rounded at 2^-53 of the largest entry.  The dense
// FP64 march keeps each product Ke_rc u_c to its own 53 bits, so the dense integers take
// only a Ke whose rows can't tell: every value reaches every row (no entry below the
// largest row sum / 256).  An error of 2^-56 of C max|u| is then within 2^-48 of any
// row's own sum |Ke_rc u_c|, the bound of the 26 roundings of an FP64 row.  Measured on
// random, graded and point vectors with one value 1e9 times the others, largest error
// over that sum, dense integers / FP64: ratio 126 2^-49.4 / 2^-49.4, 236 2^-48.6 /
// 2^-49.6, 2,396 2^-45.2 / 2^-49.4.  Rows of another scale, uncoupled components or
// corners and single zeros (the cube's at nu = 1/4) go to the FP64 marches, as does a Ke
// with the 45-entry pattern that is not a cube's.
bool fxPrepare(const KeData& ke, FxOperand& op) {
    double k[8], C = 0.0;
    op.cube = cubeConstants(ke, k, C);
    if (op.cube)
        return op.ready = fxDigits(k, 8, C, 0, op.k1, op.k0, op.outExp) && threeFits(op, 0) && threeFits(op, 6);
    if (ke.structured) return op.ready = false;
    double least = std::fabs(ke.Ke[0]);
    for (int r = 0; r < 24; ++r) {
        double row = 0.0;
        for (int c = 0; c < 24; ++c) {
            row += std::fabs(ke.Ke[24 * r + c]);
            least = std::fmin(least, std::fabs(ke.Ke[24 * r + c]));
        }
        C = std::fmax(C, row);
    }
    return op.ready = C <= 256.0 * least && fxDigits(ke.Ke, 576, C, 3, op.k1, op.k0, op.outExp);
}

cudaError_t fxSetAttributes() {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto kern) {
        if (!e) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fxSmemBytes<FX_TY>());
    };
    set(kMatvecFx<OUT_CG, FxArgs, Ks<double>>);
    set(kMatvecFx<OUT_ANY, FxArgs, Ks<double>>);
    set(kMatvecFx<OUT_TRUE, FxArgs, Ks<double>>);
    set(kMatvecFx<OUT_CG, FxDenseArgs, Kd<double>>);
    set(kMatvecFx<OUT_ANY, FxDenseArgs, Kd<double>>);
    return e;
}

// The operator scale of a level is a power of two (planLevels); other scales stay with the FP64 march.
bool fxEligible(const FxOperand& op, double scale) {
    int e = 0;
    return op.ready && scale > 0.0 && std::frexp(scale, &e) == 0.5 && std::abs(e) <= 64;
}

void launchMatvecFx(cudaStream_t stream, const MatvecArgs<double>& a, const FxOperand& op, const double* opconst,
                    Scalars* S, const RedBuf& rb) {
    const int zc = marchLayers(a.g, op.cube ? 2 : 1);
    const Grid& g = a.g;
    const dim3 block(MV_TX, FX_TY),
        grid((g.nx + MV_TX - 2) / (MV_TX - 1), (g.ny + FX_TY - 2) / (FX_TY - 1), (g.nz + zc - 1) / zc);
    const bool cg = a.mode == MV_AX && a.dot0 == DOT_X_OUT && !a.dot1 && !a.y32;
    const bool tr = a.mode == MV_RESID && a.dot0 == DOT_OUT_OUT && !a.dot1 && a.y32;
    auto go = [&](auto K, int rows, int cols, auto k, const double* src, auto kern) {
        for (int i = 0; i < rows * cols; ++i) {
            K.k1[i] = op.k1[i];
            K.k0[i] = op.k0[i];
        }
        for (int r = 0; r < rows; ++r) {
            K.kb[r] = 1ll << 31;
            for (int c = 0; c < cols; ++c) K.kb[r] += (long long)op.k1[r * cols + c] * (1ll << 31);
        }
        int e = 0;
        std::frexp(a.scale, &e);
        K.scaleExp = e - 1;
        K.outExp = op.outExp;
        std::memcpy(k.v, src, sizeof(k.v));
        kern<<<grid, block, fxSmemBytes<FX_TY>(), stream>>>(a, K, k, zc, S, rb);
    };
    if (op.cube)
        go(FxArgs(), 8, 1, Ks<double>(), opconst,
           cg ? kMatvecFx<OUT_CG, FxArgs, Ks<double>>
              : tr ? kMatvecFx<OUT_TRUE, FxArgs, Ks<double>> : kMatvecFx<OUT_ANY, FxArgs, Ks<double>>);
    else
        go(FxDenseArgs(), 24, 24, Kd<double>(), opconst + 45,
           cg ? kMatvecFx<OUT_CG, FxDenseArgs, Kd<double>> : kMatvecFx<OUT_ANY, FxDenseArgs, Kd<double>>);
}

}  // namespace vfem
