// kernels.cu -- sm_103a kernels of the voxel MG-PCG solve.
//
// Kernel map (reference shader / routine it replaces, paths relative to the
// reference project root):
//   kMatvecH, kMatvec  MatxVec.comp + FixedNodes.comp + VecDotVec.comp
//                    (MatrixFreeSparse.hpp:197-214): atomic-free element-by-element
//                    product on a 2.5-D tile (kMatvecH: Walsh-factorised isotropic
//                    cube Ke; kMatvec: general Ke; FP64 in matvec_fx.cu where the Ke allows
//                    it), fixed rows zeroed, dots fused.
//   kRestrict2, kRestrict64, kRestrictSmall, kRestrict  CWiseMult.comp + Restrict.comp (MultigridPreconditioner.hpp:67-108):
//                    full weighting on the dense grid (kRestrict2<T, true> also
//                    performs the mixed solve's residual update, ConjugateGradient_1.comp).
//   kProlongFlat, kProlong64, kProlongSmall, kProlongSmooth2, kProlongSmooth
//                    Interpolate.comp + PreSmoothAndAXPY.comp +
//                    Smooth.comp (MultigridPreconditioner.hpp:110-155,176-181),
//                    fixed mask and r.z fused.
//   kCoarseSmall, kCoarseGather/kSymRuns/kSymRunsReduce, kGemv64  the coarsest SimplicialLDLT solve
//                    (MultigridPreconditioner.hpp:174-175) as a dense symmetric
//                    inverse: FP16 packed half tiles (mixed) or the full FP64 matrix.
//   kUpdateXR, kUpdateR  ConjugateGradient_1.comp + VecDotVec.comp (r.r).
//   kUpdateP, kUpdatePX  ConjugateGradient_2.comp (kUpdatePX: with the mixed solve's
//                    deferred x update).
// Reductions are deterministic: block partials in a fixed grid, summed in a
// fixed order by the last block to finish (no floating-point atomics).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "matvec_march.cuh"
#include "reduce.cuh"

namespace vfem {

namespace {

constexpr int NT = 256;
constexpr int PZ = 8;  // z nodes per thread in the per-node kernels

// Element-by-element product with a general Ke: denseMarch (matvec_march.cuh)
// and the grid reduction of its dots.
template <typename T, typename TC = T>
__global__ void __launch_bounds__(MV_TX* MV_TY, 1)
    kMatvec(MatvecArgs<T> a, const Kd<TC> kp, int layers, Scalars* S, RedBuf rb) {
    if (a.checkDone && S->done) return;
    if (a.condTrue && !trueResidualDue(S)) return;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    DotAcc<TC> d0, d1;
    denseMarch<T, TC>(a, kp, smemRaw, d0, d1, layers);
    if (a.epi != EPI_NONE) {
        double v[2] = {d0.get(), d1.get()}, t[2];
        if (gridReduce<MV_TX * MV_TY, 2>(v, rb, t)) applyEpi(a.epi, S, t[0], t[1]);
    }
}

// The structured (isotropic cube) product: walshMarch (matvec_march.cuh) and the
// grid reduction of its dots.
// KP: Ks<TC>, or the cube's Kc<TC>.
template <typename T, typename TC, int OUT = OUT_ANY, typename KP = Ks<TC>>
__global__ void __launch_bounds__(MV_TX* MV_TY, sizeof(TC) == 4 ? 3 : 2)
    kMatvecH(MatvecArgs<T> a, const KP kp, int layers, Scalars* S, RedBuf rb) {
    if (a.checkDone && S->done) return;
    if (a.condTrue && !trueResidualDue(S)) return;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    DotAcc<TC> d0, d1;
    [[maybe_unused]] const int sel = walshMarch<T, TC, OUT, KP>(a, kp, S, smemRaw, d0, d1, layers);
    if (a.epi != EPI_NONE) {
        double v[2] = {d0.get(), d1.get()}, t[2];
        if (gridReduce<MV_TX * MV_TY, 2>(v, rb, t)) {
            applyEpi(a.epi, S, t[0], t[1]);
            if constexpr (OUT == OUT_CG_PX) S->pSel = sel ^ 1;
        }
    }
}

// Full weighting (the transpose of trilinear prolongation) on the dense grid:
// rc[C] = sum_{|d| < DIV} prod_i (DIV - |d_i|)/DIV * rf[DIV*C + d].  Equal to
// the reference's W-weighted per-element restriction (see setup.cpp).
template <typename T, int DIV>
__global__ void __launch_bounds__(256) kRestrict(Grid gf, Grid gc, const T* __restrict__ rf, T* __restrict__ rc,
                                                 const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    const int cx = blockIdx.x * 32 + threadIdx.x, cy = blockIdx.y * 8 + threadIdx.y;
    if (cx >= gc.nx || cy >= gc.ny) return;
    constexpr int R = DIV - 1;
    const T inv = T(1) / T(DIV);
    for (int cz = blockIdx.z * PZ; cz < min(gc.nz, (int)(blockIdx.z + 1) * PZ); ++cz) {
        T a0 = T(0), a1 = T(0), a2 = T(0);
        for (int dz = -R; dz <= R; ++dz) {
            const int fz = cz * DIV + dz;
            if (fz < 0 || fz >= gf.nz) continue;
            const T wz = T(DIV - abs(dz)) * inv;
            for (int dy = -R; dy <= R; ++dy) {
                const int fy = cy * DIV + dy;
                if (fy < 0 || fy >= gf.ny) continue;
                const T wy = T(DIV - abs(dy)) * inv;
                T s0 = T(0), s1 = T(0), s2 = T(0);
#pragma unroll
                for (int dx = -R; dx <= R; ++dx) {
                    const int fx = cx * DIV + dx;
                    if (fx < 0 || fx >= gf.nx) continue;
                    const T wx = T(DIV - abs(dx)) * inv;
                    const T* p = rf + 3 * gf.store(fx, fy, fz);
                    s0 = fma(wx, p[0], s0);
                    s1 = fma(wx, p[1], s1);
                    s2 = fma(wx, p[2], s2);
                }
                const T w = wz * wy;
                a0 = fma(w, s0, a0);
                a1 = fma(w, s1, a1);
                a2 = fma(w, s2, a2);
            }
        }
        T* q = rc + 3 * gc.store(cx, cy, cz);
        q[0] = a0;
        q[1] = a1;
        q[2] = a2;
    }
}

// Trilinear prolongation of coarse node values to fine node (fx,fy,fz).
// The same full weighting for the 2x coarsening, separably and with reuse:
// a thread owns coarse column (cx, cy) and marches PZC coarse layers up z.
// rc(cz) = P(2cz-1)/2 + P(2cz) + P(2cz+1)/2 with the fine-plane sums
// P(fz) = sum_dy w_dy (r(2cx-1)/2 + r(2cx) + r(2cx+1)/2) at row 2cy+dy; P(2cz+1)
// is kept for the next layer, and r(2cx-1) of a lane is r(2cx+1) of the lane
// below (a warp shuffle), so each fine value is loaded about 1.5 times.
constexpr int PZR = 4;
// UPD (mixed-precision CG): the residual update r -= alpha Ap of the finest
// level fused in.  rf is the old residual and Ap the product; each thread
// writes the updated values of the fine nodes its coarse cell owns (fine x, y,
// z in {2c, 2c + 1}) to rOut (a different vector: neighbouring cells read
// the old values of their halos) and sums their squares for r.r; halo values
// (row 2cy-1, the block's first plane, the left x neighbour of lane 0) are
// recomputed from rf and Ap.  checkDone = 2: run only in an iteration that
// replaced the residual by the true one (restricting the replacement).
// PZ: coarse layers a thread marches (1 on small grids: more blocks, shorter chains).
template <typename T, bool UPD, int PZ = PZR>
__global__ void __launch_bounds__(256) kRestrict2(Grid gf, Grid gc, const T* __restrict__ rf, const T* __restrict__ Ap,
                                                  T* __restrict__ rOut, T* __restrict__ rc, Scalars* S, RedBuf rb,
                                                  int checkDone) {
    if (checkDone && S->done) return;
    if (checkDone == 2 && S->replStamp != S->matvecs) return;
    const int lane = threadIdx.x;
    const int cx = blockIdx.x * 32 + lane, cy = blockIdx.y * 8 + threadIdx.y;
    const bool valid = cx < gc.nx && cy < gc.ny;
    const T half = T(0.5);
    const T av = UPD ? (T)S->alpha : T(0);
    const int fx0 = 2 * cx;
    DotAcc<T> acc;
    // Weighted plane sum at fine layer fz: the three rows 2cy-1 .. 2cy+1, each
    // r(2cx-1)/2 + r(2cx) + r(2cx+1)/2.  All loads of the plane are issued first,
    // then the shuffles; all lanes take part, out-of-grid fine nodes count 0.
    auto planeSum = [&](int fz, bool ownPlane, T (&P)[3]) {
        T c0[3][3], c1[3][3], cl[3][3];
        int64_t bases[3];
        bool ok0s[3], ok1s[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int fy = 2 * cy - 1 + r;
            const bool rowOk = fy >= 0 && fy < gf.ny && fz >= 0 && fz < gf.nz;
            const int64_t base = rowOk ? gf.store(0, fy, fz) : 0;
            const bool ok0 = rowOk && fx0 < gf.nx, ok1 = rowOk && fx0 + 1 < gf.nx;
            const bool okl = lane == 0 && rowOk && fx0 - 1 >= 0 && fx0 - 1 < gf.nx;
            bases[r] = base;
            ok0s[r] = ok0;
            ok1s[r] = ok1;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                c0[r][c] = ok0 ? rf[3 * (base + fx0) + c] : T(0);
                c1[r][c] = ok1 ? rf[3 * (base + fx0 + 1) + c] : T(0);
                cl[r][c] = okl ? rf[3 * (base + fx0 - 1) + c] : T(0);
                if (UPD) {
                    const T a0 = ok0 ? Ap[3 * (base + fx0) + c] : T(0);
                    const T a1 = ok1 ? Ap[3 * (base + fx0 + 1) + c] : T(0);
                    const T al = okl ? Ap[3 * (base + fx0 - 1) + c] : T(0);
                    c0[r][c] = fma(-av, a0, c0[r][c]);
                    c1[r][c] = fma(-av, a1, c1[r][c]);
                    cl[r][c] = fma(-av, al, cl[r][c]);
                }
            }
        }
        if (UPD && ownPlane && valid) {
#pragma unroll
            for (int r = 1; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    if (ok0s[r]) {
                        rOut[3 * (bases[r] + fx0) + c] = c0[r][c];
                        acc.add(c0[r][c] * c0[r][c]);
                    }
                    if (ok1s[r]) {
                        rOut[3 * (bases[r] + fx0 + 1) + c] = c1[r][c];
                        acc.add(c1[r][c] * c1[r][c]);
                    }
                }
        }
        T row[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                T cm = __shfl_up_sync(0xffffffffu, c1[r][c], 1);
                if (lane == 0) cm = cl[r][c];
                row[r][c] = c0[r][c] + half * (cm + c1[r][c]);
            }
#pragma unroll
        for (int c = 0; c < 3; ++c) P[c] = row[1][c] + half * (row[0][c] + row[2][c]);
    };
    const int cz0 = blockIdx.z * PZ, cz1 = min(gc.nz, cz0 + PZ);
    T Pm[3];
    planeSum(2 * cz0 - 1, false, Pm);
    for (int cz = cz0; cz < cz1; ++cz) {
        T P0[3], Pp[3];
        planeSum(2 * cz, true, P0);
        planeSum(2 * cz + 1, true, Pp);
        if (valid) {
            T* q = rc + 3 * gc.store(cx, cy, cz);
#pragma unroll
            for (int c = 0; c < 3; ++c) q[c] = P0[c] + half * (Pm[c] + Pp[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) Pm[c] = Pp[c];
    }
    if (UPD) {
        double v[1] = {acc.get()}, t[1];
        if (gridReduce<256, 1>(v, rb, t)) applyEpi(EPI_CONV, S, t[0], 0.0);
    }
}

// The same restriction for FP64, whose operations bound it: y, then z, then x
// (42 operations a coarse node instead of 54, and three shuffles a layer instead
// of eighteen a plane).  A warp's first lane only supplies its right column to
// the next one, so a warp restricts 31 coarse columns.
__global__ void __launch_bounds__(256) kRestrict64(Grid gf, Grid gc, const double* __restrict__ rf,
                                                   double* __restrict__ rc, const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    const int lane = threadIdx.x, cx = (int)blockIdx.x * 31 + lane - 1, cy = blockIdx.y * 8 + threadIdx.y;
    const bool out = lane > 0 && cx < gc.nx && cy < gc.ny;
    const int fx0 = 2 * cx;
    const bool ok0 = fx0 >= 0 && fx0 < gf.nx, ok1 = fx0 + 1 >= 0 && fx0 + 1 < gf.nx;
    // y-weighted columns 2cx and 2cx + 1 of fine layer fz
    auto plane = [&](int fz, double (&Y)[6]) {
        double v[3][6];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int fy = 2 * cy - 1 + r;
            const bool row = fy >= 0 && fy < gf.ny && fz >= 0 && fz < gf.nz;
            const double* p = rf + 3 * (row ? gf.store(0, fy, fz) : 0) + 3 * fx0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v[r][c] = row && ok0 ? p[c] : 0.0;
                v[r][3 + c] = row && ok1 ? p[3 + c] : 0.0;
            }
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) Y[c] = fma(0.5, v[0][c] + v[2][c], v[1][c]);
    };
    const int cz0 = blockIdx.z * PZR, cz1 = min(gc.nz, cz0 + PZR);
    double Ym[6];
    plane(2 * cz0 - 1, Ym);
    for (int cz = cz0; cz < cz1; ++cz) {
        double Y0[6], Yp[6], Z[6];
        plane(2 * cz, Y0);
        plane(2 * cz + 1, Yp);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            Z[c] = fma(0.5, Ym[c] + Yp[c], Y0[c]);
            Ym[c] = Yp[c];
        }
        double q[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) q[c] = fma(0.5, __shfl_up_sync(0xffffffffu, Z[3 + c], 1) + Z[3 + c], Z[c]);
        if (out) {
            double* o = rc + 3 * gc.store(cx, cy, cz);
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] = q[c];
        }
    }
}

template <typename T, int DIV>
__device__ __forceinline__ void prolongAt(const Grid& gf, const Grid& gc, const T* zc, int fx, int fy, int fz,
                                          T (&acc)[3]) {
    const int px = fx / DIV, py = fy / DIV, pz = fz / DIV;
    const int rx = fx - px * DIV, ry = fy - py * DIV, rz = fz - pz * DIV;
    const T inv = T(1) / T(DIV);
    acc[0] = acc[1] = acc[2] = T(0);
#pragma unroll
    for (int iz = 0; iz < 2; ++iz) {
        if (iz && rz == 0) continue;
        const T wz = iz ? T(rz) * inv : T(DIV - rz) * inv;
#pragma unroll
        for (int iy = 0; iy < 2; ++iy) {
            if (iy && ry == 0) continue;
            const T wy = iy ? T(ry) * inv : T(DIV - ry) * inv;
#pragma unroll
            for (int ix = 0; ix < 2; ++ix) {
                if (ix && rx == 0) continue;
                const T wx = ix ? T(rx) * inv : T(DIV - rx) * inv;
                const T w = wz * wy * wx;
                const T* p = zc + 3 * gc.store(px + ix, py + iy, pz + iz);
                acc[0] = fma(w, p[0], acc[0]);
                acc[1] = fma(w, p[1], acc[1]);
                acc[2] = fma(w, p[2], acc[2]);
            }
        }
    }
}

// Reference-mode up-leg of the V-cycle: zf = P zc + coef * dinv o rf on used
// nodes (coef = 2: the down-leg and up-leg Jacobi steps of the reference, which
// never update r), 0 elsewhere; fixed nodes zeroed on the finest level.
template <typename T, int DIV>
__global__ void __launch_bounds__(256)
    kProlongSmooth(Grid gf, Grid gc, const T* __restrict__ zc, const T* __restrict__ rf, const T* __restrict__ dinv,
                   const uint8_t* __restrict__ flags, T* __restrict__ zf, double coef, int maskFixed,
                   const T* __restrict__ aux, int epi, Scalars* S, RedBuf rb, int checkDone) {
    if (checkDone && S->done) return;
    const int fx = blockIdx.x * 32 + threadIdx.x, fy = blockIdx.y * 8 + threadIdx.y;
    const bool valid = fx < gf.nx && fy < gf.ny;
    DotAcc<T> d0, d1;
    if (valid) {
        for (int fz = blockIdx.z * PZ; fz < min(gf.nz, (int)(blockIdx.z + 1) * PZ); ++fz) {
            const int64_t s = gf.store(fx, fy, fz);
            const uint8_t fl = flags[s];
            T out[3] = {T(0), T(0), T(0)};
            T r[3] = {T(0), T(0), T(0)};
            if (fl & FLAG_USED) {
                T acc[3];
                prolongAt<T, DIV>(gf, gc, zc, fx, fy, fz, acc);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    r[c] = rf[3 * s + c];
                    out[c] = acc[c] + (T)coef * dinv[3 * s + c] * r[c];
                }
                if (maskFixed && (fl & FLAG_FIXED)) out[0] = out[1] = out[2] = T(0);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) zf[3 * s + c] = out[c];
            if (epi != EPI_NONE) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    d0.add(r[c] * out[c]);
                    if (aux) d1.add(out[c] * aux[3 * s + c]);
                }
            }
        }
    }
    if (epi != EPI_NONE) {
        double v[2] = {d0.get(), d1.get()}, t[2];
        if (gridReduce<256, 2>(v, rb, t)) applyEpi(epi, S, t[0], t[1]);
    }
}

// The same up-leg for the 2x coarsening, one thread per coarse cell column: a
// thread marches PZC coarse layers up z and writes the up-to-8 fine nodes
// (2cx+{0,1}, 2cy+{0,1}, 2cz+{0,1}) of each cell.  The coarse corners are read
// once per layer (the top corners become the next layer's bottom ones) and the
// trilinear weights are applied separably (z, then y, then x), so the kernel
// issues ~1.5 coarse loads per fine node instead of ~10.
constexpr int PZC = 4;
template <typename T>
__global__ void __launch_bounds__(256)
    kProlongSmooth2(Grid gf, Grid gc, const T* __restrict__ zc, const T* __restrict__ rf, const T* __restrict__ dinv,
                    const uint8_t* __restrict__ flags, T* __restrict__ zf, double coef, int maskFixed,
                    const T* __restrict__ aux, int epi, Scalars* S, RedBuf rb, int checkDone) {
    if (checkDone && S->done) return;
    const int cx = blockIdx.x * 32 + threadIdx.x, cy = blockIdx.y * 8 + threadIdx.y;
    // even fine x / y of the cell exist (the last coarse column has no fine node
    // when the fine element count is odd), and the odd ones
    const bool valid = cx < gc.nx && cy < gc.ny && 2 * cx < gf.nx && 2 * cy < gf.ny;
    const bool hx = valid && cx + 1 < gc.nx && 2 * cx + 1 < gf.nx;
    const bool hy = valid && cy + 1 < gc.ny && 2 * cy + 1 < gf.ny;
    const T half = T(0.5), cf = (T)coef;
    DotAcc<T> d0, d1;
    // Corner values of a coarse layer: [iy][ix][c], 0 where the corner does not exist.
    auto loadLayer = [&](int cz, T (&v)[2][2][3]) {
#pragma unroll
        for (int iy = 0; iy < 2; ++iy)
#pragma unroll
            for (int ix = 0; ix < 2; ++ix) {
                const bool ok = valid && cz < gc.nz && (ix == 0 || hx) && (iy == 0 || hy);
                v[iy][ix][0] = v[iy][ix][1] = v[iy][ix][2] = T(0);
                if (ok) {
                    const T* p = zc + 3 * gc.store(cx + ix, cy + iy, cz);
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[iy][ix][c] = p[c];
                }
            }
    };
    // Fine layer fz from the plane values P at the cell's coarse corners.
    // All loads of a fine layer are issued before any is used (the flag does not
    // guard them: vectors hold 0 at unused nodes), so they overlap in flight.
    auto emit = [&](int fz, const T (&P)[2][2][3]) {
        T rr[2][2][3], dd[2][2][3];
        uint8_t ff[2][2];
#pragma unroll
        for (int jy = 0; jy < 2; ++jy)
#pragma unroll
            for (int jx = 0; jx < 2; ++jx) {
                const bool ex = (jx == 0 || hx) && (jy == 0 || hy);
                const int64_t s = ex ? gf.store(2 * cx + jx, 2 * cy + jy, fz) : 0;
                ff[jy][jx] = ex ? flags[s] : (uint8_t)0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    rr[jy][jx][c] = ex ? rf[3 * s + c] : T(0);
                    dd[jy][jx][c] = ex ? dinv[3 * s + c] : T(0);
                }
            }
#pragma unroll
        for (int jy = 0; jy < 2; ++jy) {
            if (jy && !hy) continue;
#pragma unroll
            for (int jx = 0; jx < 2; ++jx) {
                if (jx && !hx) continue;
                const int64_t s = gf.store(2 * cx + jx, 2 * cy + jy, fz);
                const uint8_t fl = ff[jy][jx];
                const bool used = (fl & FLAG_USED) != 0;
                const bool zero = !used || (maskFixed && (fl & FLAG_FIXED));
                T out[3], r[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const T a0 = jx ? half * (P[0][0][c] + P[0][1][c]) : P[0][0][c];
                    const T a1 = jx ? half * (P[1][0][c] + P[1][1][c]) : P[1][0][c];
                    const T pv = jy ? half * (a0 + a1) : a0;
                    r[c] = used ? rr[jy][jx][c] : T(0);
                    out[c] = zero ? T(0) : pv + cf * dd[jy][jx][c] * r[c];
                    zf[3 * s + c] = out[c];
                }
                if (epi != EPI_NONE) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        d0.add(r[c] * out[c]);
                        if (aux) d1.add(out[c] * aux[3 * s + c]);
                    }
                }
            }
        }
    };
    if (valid) {
        const int cz0 = blockIdx.z * PZC, cz1 = min(gc.nz, cz0 + PZC);
        T B[2][2][3], Tp[2][2][3], M[2][2][3];
        loadLayer(cz0, B);
        for (int cz = cz0; cz < cz1; ++cz) {
            if (2 * cz >= gf.nz) break;
            const bool hz = cz + 1 < gc.nz && 2 * cz + 1 < gf.nz;
            emit(2 * cz, B);
            if (hz) {
                loadLayer(cz + 1, Tp);
#pragma unroll
                for (int iy = 0; iy < 2; ++iy)
#pragma unroll
                    for (int ix = 0; ix < 2; ++ix)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            M[iy][ix][c] = half * (B[iy][ix][c] + Tp[iy][ix][c]);
                            B[iy][ix][c] = Tp[iy][ix][c];
                        }
                emit(2 * cz + 1, M);
            }
        }
    }
    if (epi != EPI_NONE) {
        double v[2] = {d0.get(), d1.get()}, t[2];
        if (gridReduce<256, 2>(v, rb, t)) applyEpi(epi, S, t[0], t[1]);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) kJacobiZero(int64_t nnode, const T* __restrict__ r, const T* __restrict__ dinv,
                                                   const uint8_t* __restrict__ flags, T* __restrict__ z, double omega,
                                                   const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    for (int64_t s = blockIdx.x * (int64_t)NT + threadIdx.x; s < nnode; s += (int64_t)gridDim.x * NT) {
        const uint8_t fl = flags[s];
        const bool act = (fl & FLAG_USED) && !(fl & FLAG_FIXED);
#pragma unroll
        for (int c = 0; c < 3; ++c) z[3 * s + c] = act ? (T)omega * dinv[3 * s + c] * r[3 * s + c] : T(0);
    }
}

template <typename T, int DIV>
__global__ void __launch_bounds__(256) kProlongAdd(Grid gf, Grid gc, const T* __restrict__ zc,
                                                   const uint8_t* __restrict__ flags, T* __restrict__ zf,
                                                   const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    const int fx = blockIdx.x * 32 + threadIdx.x, fy = blockIdx.y * 8 + threadIdx.y;
    if (fx >= gf.nx || fy >= gf.ny) return;
    for (int fz = blockIdx.z * PZ; fz < min(gf.nz, (int)(blockIdx.z + 1) * PZ); ++fz) {
        const int64_t s = gf.store(fx, fy, fz);
        const uint8_t fl = flags[s];
        if (!(fl & FLAG_USED) || (fl & FLAG_FIXED)) continue;
        T acc[3];
        prolongAt<T, DIV>(gf, gc, zc, fx, fy, fz, acc);
#pragma unroll
        for (int c = 0; c < 3; ++c) zf[3 * s + c] += acc[c];
    }
}

template <typename T>
__global__ void kCoarseGather(int64_t n, const int32_t* __restrict__ freeDof, const T* __restrict__ rc,
                              T* __restrict__ b, const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = rc[freeDof[i]];
}

// 4-wide vector loads/stores of the flat vector kernels (float4; two double2).
template <typename T>
struct V4;
template <>
struct V4<float> {
    static __device__ __forceinline__ void ld(const float* p, float (&v)[4]) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    static __device__ __forceinline__ void st(float* p, const float (&v)[4]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <>
struct V4<double> {
    static __device__ __forceinline__ void ld(const double* p, double (&v)[4]) {
        const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
    static __device__ __forceinline__ void st(double* p, const double (&v)[4]) {
        reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
    }
};

// The 2x up-leg in flat form (same values as kProlongSmooth2): a block owns
// the fine rows [fy0, fy0 + PR) of fine layer fz, which are one contiguous
// range of every fine vector, and a thread takes 4 consecutive nodes at a time
// (12 values: three 16-byte loads of r and of dinv, three 16-byte stores of z,
// one 4-byte load of the flags).  The coarse rows the block interpolates from
// (PR/2 + 1 of them, averaged over the two coarse layers when fz is odd) are
// copied to shared memory with asynchronous copies while the first chunk
// loads, so a fine node costs 3-12 shared loads.  Only the first and last
// chunk of a block, which the neighbouring blocks share, take the scalar path
// (and every chunk when a vector is not 16-byte aligned).  Measured on GB300:
// 16 rows per block beat 32 (a partial last wave of blocks) and a persistent
// grid taking units from a counter (its per-unit barriers and counter round
// trips cost more than the wave tail).
// 160 threads in 6 blocks an SM against 256 in 4, us, FP32 up-leg to 65^3 nodes 12.7 / 14.4,
// 97^3 18.5 / 22.2, 161^2 x 145 42.3 / 46.4, 193^3 65.8 / 70.9, 257^3 124.6 / 130.5 (bytes
// alone 82); 128 threads in 8 63.5 to 193^3 but 144 to 257^3; 10 blocks spill registers.
constexpr int PR = 16, kProlongThreads = 160;
constexpr int kProlongCoarseRows = PR / 2 + 1;
constexpr size_t kProlongFlatMaxSmem = 200 * 1024;
__host__ __device__ inline int prolongFlatRowGroups(const Grid& gf) { return (gf.ny + PR - 1) / PR; }

template <typename T>
__device__ __forceinline__ void cpAsync(T* dst, const T* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src), "n"(sizeof(T)) : "memory");
}

// Inverse-diagonal values of a chunk: T, or FP16 (scaled; 8-byte loads).
__device__ __forceinline__ float diagVal(__half h) { return __half2float(h); }
__device__ __forceinline__ float diagVal(float v) { return v; }
template <typename T>
__device__ __forceinline__ void ldDiag12(const T* p, T (&v)[12]) {
#pragma unroll
    for (int q = 0; q < 3; ++q) V4<T>::ld(p + 4 * q, *reinterpret_cast<T(*)[4]>(v + 4 * q));
}
__device__ __forceinline__ void ldDiag12(const __half* p, float (&v)[12]) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const uint2 raw = reinterpret_cast<const uint2*>(p)[q];
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        v[4 * q] = a.x;
        v[4 * q + 1] = a.y;
        v[4 * q + 2] = b.x;
        v[4 * q + 3] = b.y;
    }
}

// The 2x transfers of small grids, one thread per value (coarse value of the
// restriction, fine value of the FP32 up-leg): every load of a thread is in flight at
// once, where the marching kernels above wait for one plane after the other.
// Same operations in the same order as kRestrict2 and kProlongFlat.  Measured,
// FP64 / FP32 us, marching -> this: restriction from 33 x 17 x 17 nodes 18.4 / 6.7 ->
// 6.2 / 4.2, from 65^3 18.5 / 8.2 -> 10.3 / 4.2, from 97^3 30.8 / 9.8 -> 22.6 / 6.2;
// FP32 up-leg to 33 x 17 x 17 10.3 -> 8.3, to 49^3 12.3 -> 12.4, to 65^3 14.4 -> 16.3:
// hence the limits, in fine nodes.
constexpr int64_t kSmallRestrict = 1000000, kSmallProlong = 100000;

template <typename T>
__global__ void __launch_bounds__(256) kRestrictSmall(Grid gf, Grid gc, const T* __restrict__ rf, T* __restrict__ rc,
                                                      const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    if (checkDone == 2 && S->replStamp != S->matvecs) return;
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= 3 * (int)gc.nnode) return;
    const int s = i / 3, c = i - 3 * s, cyz = s / gc.nx, cx = s - cyz * gc.nx, cz = cyz / gc.ny, cy = cyz - cz * gc.ny;
    const T half = T(0.5);
    T v[3][3][3];
#pragma unroll
    for (int dz = 0; dz < 3; ++dz)
#pragma unroll
        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const int fx = 2 * cx - 1 + dx, fy = 2 * cy - 1 + dy, fz = 2 * cz - 1 + dz;
                const bool ok = (unsigned)fx < (unsigned)gf.nx && (unsigned)fy < (unsigned)gf.ny && (unsigned)fz < (unsigned)gf.nz;
                v[dz][dy][dx] = ok ? rf[3 * ((fz * gf.ny + fy) * gf.nx + fx) + c] : T(0);
            }
    T P[3];
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
        T row[3];
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) row[dy] = v[dz][dy][1] + half * (v[dz][dy][0] + v[dz][dy][2]);
        P[dz] = row[1] + half * (row[0] + row[2]);
    }
    rc[i] = P[1] + half * (P[0] + P[2]);
}

template <typename T, typename DT>
__global__ void __launch_bounds__(256)
    kProlongSmall(Grid gf, Grid gc, const T* __restrict__ zc, const T* __restrict__ rf, const DT* __restrict__ dinv,
                  const uint8_t* __restrict__ flags, T* __restrict__ zf, double coef, int maskFixed,
                  const T* __restrict__ aux, int epi, Scalars* S, RedBuf rb, int checkDone) {
    if (checkDone && S->done) return;
    DotAcc<T> d0, d1;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < 3 * (int)gf.nnode; i += gridDim.x * 256) {
        const int s = i / 3, c = i - 3 * s, fyz = s / gf.nx, fx = s - fyz * gf.nx, fz = fyz / gf.ny, fy = fyz - fz * gf.ny;
        const T half = T(0.5);
        const uint32_t fl = flags[s];
        const T rv = rf[i], dv = (T)diagVal(dinv[i]);
        // coarse corners; an odd position has a neighbour one up on its axis
        const int px = 3 * (fx & 1), py = (fy & 1) ? 3 * gc.nx : 0, pz = (fz & 1) ? 3 * gc.nx * gc.ny : 0;
        const T* b = zc + 3 * (((fz >> 1) * gc.ny + (fy >> 1)) * gc.nx + (fx >> 1)) + c;
        T q[2][2][2];
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int x = 0; x < 2; ++x) q[z][y][x] = b[(z ? pz : 0) + (y ? py : 0) + (x ? px : 0)];
        const bool used = (fl & FLAG_USED) != 0;
        const bool zero = !used || (maskFixed && (fl & FLAG_FIXED));
        const T r = used ? rv : T(0);
        T w[2][2];
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x) w[y][x] = (fz & 1) ? half * (q[0][y][x] + q[1][y][x]) : q[0][y][x];
        const T r0 = (fx & 1) ? half * (w[0][0] + w[0][1]) : w[0][0], r1 = (fx & 1) ? half * (w[1][0] + w[1][1]) : w[1][0];
        const T pv = (fy & 1) ? half * (r0 + r1) : r0;
        const T out = zero ? T(0) : pv + (T)coef * dv * r;
        zf[i] = out;
        if (epi != EPI_NONE) {
            d0.add(r * out);
            if (aux) d1.add(out * aux[i]);
        }
    }
    if (epi != EPI_NONE) {
        double v[2] = {d0.get(), d1.get()}, t[2];
        if (gridReduce<256, 2>(v, rb, t)) applyEpi(epi, S, t[0], t[1]);
    }
}

// DT: the type the inverse diagonal is stored in (T, or FP16 scaled so that
// coef already carries the scale).
template <typename T, typename DT>
__global__ void __launch_bounds__(kProlongThreads, 6)
    kProlongFlat(Grid gf, Grid gc, const T* __restrict__ zc, const T* __restrict__ rf, const DT* __restrict__ dinv,
                 const uint8_t* __restrict__ flags, T* __restrict__ zf, double coef, int maskFixed,
                 const T* __restrict__ aux, int epi, int vec, float invNx, Scalars* S, RedBuf rb, int checkDone) {
    if (checkDone && S->done) return;
    extern __shared__ __align__(16) unsigned char prolongSmem[];
    T* C = reinterpret_cast<T*>(prolongSmem);  // [kProlongCoarseRows][3 * gc.nx], then the layer above
    const int groups = prolongFlatRowGroups(gf);
    const int fz = blockIdx.x / groups;
    const int fy0 = (blockIdx.x - fz * groups) * PR, fy1 = min(gf.ny, fy0 + PR);
    const int cw = 3 * gc.nx, cy0 = fy0 >> 1, cz = fz >> 1;
    const int nstage = min(kProlongCoarseRows, gc.ny - cy0) * cw;
    const bool zodd = fz & 1;
    const T half = T(0.5), cf = (T)coef;
    {
        // the block's coarse rows are contiguous in each coarse layer
        const T* src = zc + 3 * gc.store(0, cy0, cz);
        const int64_t up = 3 * ((int64_t)gc.nx * gc.ny);
        for (int j = threadIdx.x; j < nstage; j += blockDim.x) {
            cpAsync(C + j, src + j);
            if (zodd) cpAsync(C + nstage + j, src + up + j);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const int64_t nBeg = gf.store(0, fy0, fz);  // first node of the block
    const int nb = (fy1 - fy0) * gf.nx;
    const int64_t j1 = (nBeg + nb + 3) >> 2;
    DotAcc<T> d0, d1;
    // One chunk of 4 nodes; FULL: all 4 in the block's range and vectors aligned.
    auto chunk = [&](auto fullTag, int64_t n0, int ln0, const T (&rv)[12], const T (&dv)[12], uint32_t fl4) {
        constexpr bool FULL = decltype(fullTag)::value;
        // (ly, fx) of the chunk's first node; fx < 0 for nodes before the range
        const int lnc = max(ln0, 0);
        int ly = __float2int_rz(((float)lnc + 0.5f) * invNx);
        int fx = lnc - ly * gf.nx;
        if (fx < 0) { --ly; fx += gf.nx; }
        if (fx >= gf.nx) { ++ly; fx -= gf.nx; }
        fx -= lnc - ln0;
        T ov[12];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int ln = ln0 + t;
            const bool in = FULL || (ln >= 0 && ln < nb);
            if (in) {
                const uint32_t fl = (fl4 >> (8 * t)) & 0xffu;
                const bool used = (fl & FLAG_USED) != 0;
                const bool zero = !used || (maskFixed && (fl & FLAG_FIXED));
                const T* b = C + (ly >> 1) * cw + 3 * (fx >> 1);
                T pv[3];
                if (fx & 1) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) pv[c] = half * (b[c] + b[c + 3]);
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c) pv[c] = b[c];
                }
                if (ly & 1) {
                    const T* b1 = b + cw;
                    if (fx & 1) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) pv[c] = half * (pv[c] + half * (b1[c] + b1[c + 3]));
                    } else {
#pragma unroll
                        for (int c = 0; c < 3; ++c) pv[c] = half * (pv[c] + b1[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const T r = used ? rv[3 * t + c] : T(0);
                    const T out = zero ? T(0) : pv[c] + cf * dv[3 * t + c] * r;
                    if (epi != EPI_NONE) {
                        d0.add(r * out);
                        if (aux) d1.add(out * aux[3 * (n0 + t) + c]);
                    }
                    if (FULL) ov[3 * t + c] = out;
                    else zf[3 * (n0 + t) + c] = out;
                }
            }
            if (++fx == gf.nx) {
                fx = 0;
                ++ly;
            }
        }
        if (FULL) {
#pragma unroll
            for (int v = 0; v < 3; ++v) V4<T>::st(zf + 3 * n0 + 4 * v, *reinterpret_cast<T(*)[4]>(ov + 4 * v));
        }
    };
    bool staged = false;
    for (int64_t j = (nBeg >> 2) + threadIdx.x;; j += blockDim.x) {
        const bool have = j < j1;
        const int64_t n0 = 4 * j;
        const int ln0 = (int)(n0 - nBeg);  // -3 .. nb - 1
        const bool full = vec && ln0 >= 0 && ln0 + 4 <= nb;
        T rv[12], dv[12];
        uint32_t fl4 = 0;
        if (have) {
            if (full) {
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    V4<T>::ld(rf + 3 * n0 + 4 * v, *reinterpret_cast<T(*)[4]>(rv + 4 * v));
                }
                ldDiag12(dinv + 3 * n0, dv);
                fl4 = *reinterpret_cast<const uint32_t*>(flags + n0);
            } else {
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const bool in = ln0 + t >= 0 && ln0 + t < nb;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        rv[3 * t + c] = in ? rf[3 * (n0 + t) + c] : T(0);
                        dv[3 * t + c] = in ? (T)diagVal(dinv[3 * (n0 + t) + c]) : T(0);
                    }
                    if (in) fl4 |= (uint32_t)flags[n0 + t] << (8 * t);
                }
            }
        }
        if (!staged) {
            // every thread passes here once, after issuing its first chunk's loads
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
            if (zodd) {
                for (int q = threadIdx.x; q < nstage; q += blockDim.x)
                    C[q] = half * (C[q] + C[nstage + q]);
                __syncthreads();
            }
            staged = true;
        }
        if (!have) break;
        if (full) chunk(std::true_type{}, n0, ln0, rv, dv, fl4);
        else chunk(std::false_type{}, n0, ln0, rv, dv, fl4);
    }
    if (epi != EPI_NONE) {
        double v[2] = {d0.get(), d1.get()}, t[2];
        if (gridReduce<kProlongThreads, 2>(v, rb, t)) applyEpi(epi, S, t[0], t[1]);
    }
}

// x * 2^-k (k = 0 .. 3) without an FP64 operation.
__device__ __forceinline__ double scaleDown(double x, int k) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
    if (e - 4u < 0x7ffu - 4u) return __hiloint2double(hi - (k << 20), lo);
    if (((hi & 0x7fffffff) | lo) == 0) return x;
    return x * __hiloint2double((1023 - k) << 20, 0);  // subnormal result, infinity or NaN
}

// The 2x up-leg in FP64, flat like kProlongFlat.  FP64 operations (1.7 a clock and SM)
// bound it, so a value takes about 4 of them: the sums over y are made once per coarse
// column in shared memory (C: the rows summed over z; behind them, once the layer above
// is summed in, the odd fine rows), a warp adds over x only where a lane needs it, the
// weight 2^-k is an integer subtraction from the exponent, and dv * r takes one multiply
// and one multiply-add.  (kProlongFlat's corner sums, up to 7 operations where a warp
// spans two rows.)  A thread takes 2 nodes (4: 617 instead of 580 us to 257^3).
// Measured, us, kProlongFlat in FP64 -> this: up-leg to 257^3 757 -> 580, 129^3 149 ->
// 95, 97^3 70.5 -> 47, 65^3 35 -> 22.6, 34^3 14.5 -> 11.3; FP64 operations alone 405 and
// bytes 193 to 257^3.  Rows and threads of a block: to 65^3 16 rows x 256 threads 26.8,
// 8 x 128 22.6, 4 x 128 24.9; to 97^3 47, 51, 55; to 34^3 12.8, 12.5, 11.3.
template <int ROWS, int NTH>
__global__ void __launch_bounds__(NTH)
    kProlong64(Grid gf, Grid gc, const double* __restrict__ zc, const double* __restrict__ rf,
               const double* __restrict__ dinv, const uint8_t* __restrict__ flags, double* __restrict__ zf, double coef,
               int maskFixed, const double* __restrict__ aux, int epi, int vec, float invNx, Scalars* S, RedBuf rb,
               int checkDone) {
    constexpr int CH = 2;  // nodes a thread takes at a time
    if (checkDone && S->done) return;
    extern __shared__ __align__(16) unsigned char prolongSmem[];
    double* C = reinterpret_cast<double*>(prolongSmem);  // coarse rows; then the layer above, later the row sums
    const int groups = (gf.ny + ROWS - 1) / ROWS;
    const int fz = blockIdx.x / groups;
    const int fy0 = (blockIdx.x - fz * groups) * ROWS, fy1 = min(gf.ny, fy0 + ROWS);
    const int cw = 3 * gc.nx, cy0 = fy0 >> 1, cz = fz >> 1;
    const int nstage = min(ROWS / 2 + 1, gc.ny - cy0) * cw;
    const int nsum = ((fy1 - fy0) >> 1) * cw;  // odd fine rows
    const bool zodd = fz & 1;
    {
        const double* src = zc + 3 * gc.store(0, cy0, cz);
        const int64_t up = 3 * ((int64_t)gc.nx * gc.ny);
        for (int j = threadIdx.x; j < nstage; j += NTH) {
            cpAsync(C + j, src + j);
            if (zodd) cpAsync(C + nstage + j, src + up + j);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const int64_t nBeg = gf.store(0, fy0, fz);
    const int nb = (fy1 - fy0) * gf.nx;
    const int64_t j1 = (nBeg + nb + CH - 1) / CH;
    double d0 = 0.0, d1 = 0.0;
    bool staged = false;
    // sums of 2^1022 and more, which may overflow over x: the block halves every sum instead
    bool big = false;
    int halved = 0;
    auto watch = [&](double s) {
        big = big || (__double2hiint(s) & 0x7ff00000) >= (2045 << 20);
        return s;
    };
    for (int64_t j = nBeg / CH + threadIdx.x;; j += NTH) {
        const bool have = j < j1;
        const int64_t n0 = CH * j;
        const int ln0 = (int)(n0 - nBeg);  // 1 - CH .. nb - 1
        const bool full = vec && ln0 >= 0 && ln0 + CH <= nb;
        double rv[3 * CH], dv[3 * CH];
        uint32_t fl4 = 0;
        if (have) {
            if (full) {
#pragma unroll
                for (int q = 0; q < 3 * CH; q += 2) {
                    const double2 a = *reinterpret_cast<const double2*>(rf + 3 * n0 + q);
                    const double2 b = *reinterpret_cast<const double2*>(dinv + 3 * n0 + q);
                    rv[q] = a.x; rv[q + 1] = a.y;
                    dv[q] = b.x; dv[q + 1] = b.y;
                }
            } else {
#pragma unroll
                for (int t = 0; t < CH; ++t) {
                    const bool in = ln0 + t >= 0 && ln0 + t < nb;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        rv[3 * t + c] = in ? rf[3 * (n0 + t) + c] : 0.0;
                        dv[3 * t + c] = in ? dinv[3 * (n0 + t) + c] : 0.0;
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < CH; ++t)
                if (ln0 + t >= 0 && ln0 + t < nb) fl4 |= (uint32_t)flags[n0 + t] << (8 * t);
        }
        if (!staged) {
            // every thread passes here once, after issuing its first chunk's loads
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
            if (zodd) {
                for (int q = threadIdx.x; q < nstage; q += NTH) C[q] = watch(C[q] + C[nstage + q]);
                __syncthreads();
            }
            for (int q = threadIdx.x; q < nsum; q += NTH) C[nstage + q] = watch(C[q] + C[q + cw]);
            halved = __syncthreads_or(big);
            if (halved) {
                const double* src = zc + 3 * gc.store(0, cy0, cz);
                const int64_t up = 3 * ((int64_t)gc.nx * gc.ny);
                for (int q = threadIdx.x; q < nstage; q += NTH) C[q] = zodd ? 0.5 * (src[q] + src[up + q]) : src[q];
                __syncthreads();
                for (int q = threadIdx.x; q < nsum; q += NTH) C[nstage + q] = 0.5 * (C[q] + C[q + cw]);
                __syncthreads();
            }
            staged = true;
        }
        if (!have) break;
        // (ly, fx) of the chunk's first node; fx < 0 for nodes before the range
        const int lnc = max(ln0, 0);
        int ly = __float2int_rz(((float)lnc + 0.5f) * invNx);
        int fx = lnc - ly * gf.nx;
        if (fx < 0) { --ly; fx += gf.nx; }
        if (fx >= gf.nx) { ++ly; fx -= gf.nx; }
        fx -= lnc - ln0;
#pragma unroll
        for (int t = 0; t < CH; ++t) {
            const bool in = full || (ln0 + t >= 0 && ln0 + t < nb);
            if (in) {
                const uint32_t fl = (fl4 >> (8 * t)) & 0xffu;
                const bool used = (fl & FLAG_USED) != 0;
                const bool zero = !used || (maskFixed && (fl & FLAG_FIXED));
                const double* b = C + ((ly & 1) ? nstage : 0) + (ly >> 1) * cw + 3 * (fx >> 1);
                const int k = (halved ? 0 : (int)zodd + (ly & 1)) + (fx & 1);
                double pv[3] = {b[0], b[1], b[2]};
                if (fx & 1) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) pv[c] += b[c + 3];
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double r = used ? rv[3 * t + c] : 0.0;
                    const double out = zero ? 0.0 : fma(coef, dv[3 * t + c] * r, scaleDown(pv[c], k));
                    if (epi != EPI_NONE) {
                        d0 = fma(r, out, d0);
                        if (aux) d1 = fma(out, aux[3 * (n0 + t) + c], d1);
                    }
                    rv[3 * t + c] = out;
                    if (!full) zf[3 * (n0 + t) + c] = out;
                }
            }
            if (++fx == gf.nx) {
                fx = 0;
                ++ly;
            }
        }
        if (full) {
#pragma unroll
            for (int q = 0; q < 3 * CH; q += 2)
                *reinterpret_cast<double2*>(zf + 3 * n0 + q) = make_double2(rv[q], rv[q + 1]);
        }
    }
    if (epi != EPI_NONE) {
        double v[2] = {d0, d1}, t[2];
        if (gridReduce<NTH, 2>(v, rb, t)) applyEpi(epi, S, t[0], t[1]);
    }
}

// y = Kinv b with the full inverse, one warp per row (FP64: the packed form below
// needs two FMAs per stored value plus FP64 shuffle reductions, which GB300's
// narrow FP64 pipe turns into 1.7x the time of this one-FMA-per-value form).
__global__ void __launch_bounds__(256) kGemv64(const double* __restrict__ K, int64_t n, const double* __restrict__ b,
                                               const int32_t* __restrict__ freeDof, double* __restrict__ zc,
                                               const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    const int lane = threadIdx.x & 31;
    const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (row >= n) return;
    const double* k = K + row * n;
    double acc = 0.0;
    for (int64_t j = lane; j < n; j += 32) acc = fma(k[j], b[j], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) zc[freeDof[row]] = acc;
}

// Small coarsest systems in one kernel: the block gathers the right-hand side into
// shared memory, a warp takes a row of the full inverse (FP64, or FP16 with rows
// padded to 8 values) with independent partial sums.  Gathering, streaming and
// reducing took two kernels in FP64 and three in mixed precision, each mostly
// latency.  Measured, FP64 / mixed us, before -> this: n = 600 11.3 / 15.3 -> 6.3 /
// 5.5, n = 1,944 18.5 / 17.5 -> 14.5 / 8.2 (FP64 FMAs alone 8), n = 2,700 25.7 / 19.6
// -> 24.7 / 8.3, n = 3,993 44.2 / 18.0 -> 47.2 / 12.3, where FP64 is better off with
// kGemv64 and the mixed form, at twice the bytes of the packed half, would soon be
// with that: hence kSmallCoarse.
__device__ __forceinline__ float smallRow(const __half* k, const float* b, int n, int lane) {
    float2 acc[4] = {};
    for (int j = 8 * lane; j < n; j += 256) {
        const uint4 q = *reinterpret_cast<const uint4*>(k + j);
        const float4 b0 = *reinterpret_cast<const float4*>(b + j), b1 = *reinterpret_cast<const float4*>(b + j + 4);
        acc[0] = __ffma2_rn(__half22float2(*reinterpret_cast<const __half2*>(&q.x)), make_float2(b0.x, b0.y), acc[0]);
        acc[1] = __ffma2_rn(__half22float2(*reinterpret_cast<const __half2*>(&q.y)), make_float2(b0.z, b0.w), acc[1]);
        acc[2] = __ffma2_rn(__half22float2(*reinterpret_cast<const __half2*>(&q.z)), make_float2(b1.x, b1.y), acc[2]);
        acc[3] = __ffma2_rn(__half22float2(*reinterpret_cast<const __half2*>(&q.w)), make_float2(b1.z, b1.w), acc[3]);
    }
    const float2 s = __fadd2_rn(__fadd2_rn(acc[0], acc[1]), __fadd2_rn(acc[2], acc[3]));
    return s.x + s.y;
}
__device__ __forceinline__ double smallRow(const double* k, const double* b, int n, int lane) {
    double acc[4] = {};
    int j = lane;
    for (; j + 96 < n; j += 128) {
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = fma(k[j + 32 * q], b[j + 32 * q], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (j + 32 * q < n) acc[q] = fma(k[j + 32 * q], b[j + 32 * q], acc[q]);
    return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}
template <typename T, typename KT>
__global__ void __launch_bounds__(256) kCoarseSmall(const KT* __restrict__ K, int n, int ld, T scale,
                                                    const int32_t* __restrict__ freeDof, const T* __restrict__ rc,
                                                    T* __restrict__ zc, const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    __shared__ __align__(16) T b[kSmallCoarse<T> + 8];
    for (int j = threadIdx.x; j < ((n + 7) & ~7); j += 256) b[j] = j < n ? rc[freeDof[j]] : T(0);
    __syncthreads();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    T sum = smallRow(K + (int64_t)row * ld, b, n, lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) zc[freeDof[row]] = sum * scale;
}

// FP16 rows of the full inverse for kCoarseSmall.
__global__ void __launch_bounds__(256) kPackRowsHalf(const float* __restrict__ K, int n, int ld, float invScale,
                                                     __half* __restrict__ rows) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n * ld; i += gridDim.x * 256) {
        const int r = i / ld, c = i - r * ld;
        rows[i] = __float2half_rn(c < n ? K[(int64_t)r * n + c] * invScale : 0.0f);
    }
}

// ---- coarsest solve of the mixed-precision cycle: y = Kinv b with the
// symmetric inverse stored once, in FP16.  Kinv is kept as the lower block
// triangle of 64 x 64 tiles (tile (I, J <= I) at index I (I + 1) / 2 + J,
// row-major inside, zero-padded past n), a quarter of the bytes of the full
// FP32 matrix.  The stored values are Kinv / scale with scale a power of two
// that maps the largest diagonal entry to 2^14 (|Kinv_ij| <= max diag for an
// SPD inverse), so every entry above 2^-10 of that maximum keeps FP16's 11-bit
// significand; the products accumulate in FP32.  The rounding is symmetric, so
// the coarse operator stays symmetric.  kSymRuns streams runs of consecutive
// tiles: it reads each tile once, accumulates K_IJ b_J for y_I over a row block
// and writes K_IJ^T b_I (for y_J, off-diagonal tiles) per tile; kSymRunsReduce sums the partials per row block in a fixed order
// (deterministic, no atomics) and applies the scale.
__host__ __device__ inline int64_t symTileCount(int64_t nb) { return nb * (nb + 1) / 2; }
// Tile index -> (I, J): FP32 square root, corrected exactly in integers (an FP64
// square root per thread would run on GB300's narrow FP64 pipe).
__device__ inline void symTileDecode(int64_t t, int64_t& I, int64_t& J) {
    int64_t i = (int64_t)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (i > 0 && i * (i + 1) / 2 > t) --i;
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    I = i;
    J = t - i * (i + 1) / 2;
}

__global__ void kPackSymHalf(const float* __restrict__ K, int64_t n, int64_t nb, float invScale,
                             __half* __restrict__ tiles) {
    const int64_t total = symTileCount(nb) * CT * CT;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t I, J;
        symTileDecode(i / (CT * CT), I, J);
        const int e = (int)(i % (CT * CT));
        const int64_t row = I * CT + e / CT, col = J * CT + e % CT;
        tiles[i] = __float2half_rn((row < n && col < n) ? K[row * n + col] * invScale : 0.0f);
    }
}

// *out = max |x_i| as FP32 bits (non-negative floats order like their bits); *out zeroed by the caller.
__global__ void __launch_bounds__(256) kMaxAbs(const float* __restrict__ x, int64_t n, unsigned* __restrict__ out) {
    float m = 0.0f;
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) m = fmaxf(m, fabsf(x[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

__global__ void __launch_bounds__(256) kToHalf(const float* __restrict__ x, int64_t n, float invScale,
                                               __half* __restrict__ y) {
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT)
        y[i] = __float2half_rn(x[i] * invScale);
}

// Largest diagonal entry of a row-major n x n matrix (one block).
__global__ void __launch_bounds__(1024) kMaxDiag(const float* __restrict__ K, int64_t n, float* __restrict__ out) {
    __shared__ float red[32];
    float m = 0.0f;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, K[i * n + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) *out = m;
    }
}

// The tiles, numbered row block after row block, are split evenly over the warps that fit
// on the chip: warp w of W takes tiles symStart(w) .. symStart(w + 1) - 1.  Where a row
// block ends within its range, or the range ends, it writes that row block's sums.
constexpr int SYM_WARPS = 4, SYM_PER_SM = 3, SYM_BLOCKS = SYM_PER_SM * 152;
__host__ __device__ inline int64_t symWarps(int64_t tiles) {
    return tiles < (int64_t)SYM_WARPS * SYM_BLOCKS ? tiles : (int64_t)SYM_WARPS * SYM_BLOCKS;
}
__host__ __device__ inline int64_t symStart(int64_t w, int64_t tiles, int64_t warps) { return w * tiles / warps; }

// A lane holds 8 columns of every fourth row of a tile (16 loads of 16 bytes) and replaces
// each by the next tile's as soon as it is used, so a whole tile per warp is in flight and
// nothing waits on a barrier.  The row sums K_IJ b_J stay in registers until the row block
// ends (part[its last tile][0..63]); the column sums K_IJ^T b_I of an off-diagonal tile
// need two shuffles a value (part[tile][64..127]).  DRAM bound: 183 MB for n = 13,500 in
// 32.6 us (5.6 TB/s); with gather and reduction 47.9 us, where blocks of 256 threads on
// runs of 16 tiles with a barrier per tile took 55.3 and warps on runs of 8 (one wave and
// a half of blocks) 47.5; for n = 4,752 18.1, 21.7 and 19.5.  Two blocks an SM 49.2.
__global__ void __launch_bounds__(32 * SYM_WARPS, SYM_PER_SM)
    kSymRuns(const __half* __restrict__ tiles, const float* __restrict__ b, float* __restrict__ part, int64_t nb,
             const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    const int64_t T = nb * (nb + 1) / 2, W = symWarps(T), w = blockIdx.x * (int64_t)SYM_WARPS + (threadIdx.x >> 5);
    if (w >= W) return;
    int64_t t = symStart(w, T, W);
    const int64_t tEnd = symStart(w + 1, T, W);
    // row block of the first tile: the largest I with I (I + 1) / 2 <= t
    int I = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((int64_t)I * (I + 1) / 2 > t) --I;
    while ((int64_t)(I + 1) * (I + 2) / 2 <= t) ++I;
    int J = (int)(t - (int64_t)I * (I + 1) / 2);
    const int lane = threadIdx.x & 31, tc = lane & 7, tr = lane >> 3;
    float bI[16], rs[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        bI[i] = b[I * CT + 4 * i + tr];
        rs[i] = 0.f;
    }
    const uint4* K = reinterpret_cast<const uint4*>(tiles + t * (CT * CT)) + lane;
    uint4 k[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) k[i] = K[32 * i];
    const float4* bp = reinterpret_cast<const float4*>(b + J * CT + 8 * tc);
    float4 q0 = bp[0], q1 = bp[1];
    for (; t < tEnd; ++t) {
        const float2 bj[4] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y),
                              make_float2(q1.z, q1.w)};
        const bool more = t + 1 < tEnd, diagonal = J == I;
        K += CT * CT / 8;
        J = diagonal ? 0 : J + 1;
        if (more) {
            bp = reinterpret_cast<const float4*>(b + J * CT + 8 * tc);
            q0 = bp[0];
            q1 = bp[1];
        }
        float2 cs[4] = {};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float2 k0 = __half22float2(*reinterpret_cast<const __half2*>(&k[i].x));
            const float2 k1 = __half22float2(*reinterpret_cast<const __half2*>(&k[i].y));
            const float2 k2 = __half22float2(*reinterpret_cast<const __half2*>(&k[i].z));
            const float2 k3 = __half22float2(*reinterpret_cast<const __half2*>(&k[i].w));
            if (more) k[i] = K[32 * i];
            const float2 r2 = __ffma2_rn(k3, bj[3], __ffma2_rn(k2, bj[2], __ffma2_rn(k1, bj[1], __fmul2_rn(k0, bj[0]))));
            rs[i] += r2.x + r2.y;
            const float2 bi = make_float2(bI[i], bI[i]);
            cs[0] = __ffma2_rn(k0, bi, cs[0]);
            cs[1] = __ffma2_rn(k1, bi, cs[1]);
            cs[2] = __ffma2_rn(k2, bi, cs[2]);
            cs[3] = __ffma2_rn(k3, bi, cs[3]);
        }
        if (!diagonal) {
#pragma unroll
            for (int o = 8; o <= 16; o <<= 1)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    cs[j].x += __shfl_xor_sync(0xffffffffu, cs[j].x, o);
                    cs[j].y += __shfl_xor_sync(0xffffffffu, cs[j].y, o);
                }
            if (tr == 0) {
                float4* out = reinterpret_cast<float4*>(part + t * (2 * CT) + CT + 8 * tc);
                out[0] = make_float4(cs[0].x, cs[0].y, cs[1].x, cs[1].y);
                out[1] = make_float4(cs[2].x, cs[2].y, cs[3].x, cs[3].y);
            }
        }
        if (diagonal || !more) {
#pragma unroll
            for (int o = 1; o < 8; o <<= 1)
#pragma unroll
                for (int i = 0; i < 16; ++i) rs[i] += __shfl_xor_sync(0xffffffffu, rs[i], o);
            if (tc == 0) {
#pragma unroll
                for (int i = 0; i < 16; ++i) part[t * (2 * CT) + 4 * i + tr] = rs[i];
            }
            ++I;
            if (more) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    bI[i] = b[I * CT + 4 * i + tr];
                    rs[i] = 0.f;
                }
            }
        }
    }
}

// y_I = scale (sum over the runs of row I of their row partials + sum_{I' > I}
// (K_I'I^T b_I')), in a fixed order.
__global__ void __launch_bounds__(1024) kSymRunsReduce(const float* __restrict__ part, int64_t nb, int64_t n,
                                                       const int32_t* __restrict__ freeDof, float scale,
                                                       float* __restrict__ zc, const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    __shared__ float red[16][CT];
    const int64_t I = blockIdx.x;
    const int r = threadIdx.x & (CT - 1), grp = threadIdx.x >> 6;
    float s = 0.f;
    // row sums of row block I: at its last tile and at the last tile of every warp's range in it
    const int64_t T = nb * (nb + 1) / 2, W = symWarps(T), t0 = I * (I + 1) / 2, t1 = t0 + I + 1;
    if (grp == 0) s = part[(t1 - 1) * (2 * CT) + r];
    for (int64_t w = ((t0 + 1) * W + T - 1) / T + grp;; w += 16) {  // the first w with symStart(w) > t0
        const int64_t t = symStart(w, T, W);
        if (t >= t1) break;
        s += part[(t - 1) * (2 * CT) + r];
    }
#pragma unroll 8
    for (int64_t Ip = I + 1 + grp; Ip < nb; Ip += 16) s += part[(Ip * (Ip + 1) / 2 + I) * (2 * CT) + CT + r];
    red[grp][r] = s;
    __syncthreads();
    if (grp == 0) {
        float y = 0.f;
#pragma unroll
        for (int q = 0; q < 16; ++q) y += red[q][r];
        const int64_t i = I * CT + r;
        if (i < n) zc[freeDof[i]] = y * scale;
    }
}

// x += alpha p; r -= alpha Ap; r.r.  TX = double is the FP64 solution; TX = float
// is the mixed-precision correction accumulated since the last flush.
template <typename TX, typename TV>
__global__ void __launch_bounds__(256) kUpdateXR(int64_t n, TX* __restrict__ x, TV* __restrict__ r,
                                                 const TV* __restrict__ p, const TV* __restrict__ Ap, Scalars* S,
                                                 RedBuf rb) {
    if (S->done) return;
    const TX ax = (TX)S->alpha;
    const TV av = (TV)S->alpha;
    DotAcc<TV> acc;
    const int64_t tid = blockIdx.x * (int64_t)NT + threadIdx.x, stride = (int64_t)gridDim.x * NT;
    const int64_t n4 = n / 4;
    for (int64_t q = tid; q < n4; q += stride) {
        TX xv[4];
        TV rv[4], pv[4], av4[4];
        V4<TX>::ld(x + 4 * q, xv);
        V4<TV>::ld(r + 4 * q, rv);
        V4<TV>::ld(p + 4 * q, pv);
        V4<TV>::ld(Ap + 4 * q, av4);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            xv[k] = fma(ax, (TX)pv[k], xv[k]);
            rv[k] = fma(-av, av4[k], rv[k]);
            acc.add(rv[k] * rv[k]);
        }
        V4<TX>::st(x + 4 * q, xv);
        V4<TV>::st(r + 4 * q, rv);
    }
    for (int64_t i = 4 * n4 + tid; i < n; i += stride) {
        x[i] = fma(ax, (TX)p[i], x[i]);
        const TV ri = fma(-av, Ap[i], r[i]);
        r[i] = ri;
        acc.add(ri * ri);
    }
    double v[1] = {acc.get()}, t[1];
    if (gridReduce<NT, 1>(v, rb, t)) applyEpi(EPI_CONV, S, t[0], 0.0);
}

// Mixed precision: r -= alpha Ap; r.r.  The solution update x += alpha p of
// the same iteration is deferred to kUpdatePX (or kFlushX), which read p anyway.
__global__ void __launch_bounds__(256) kUpdateR(int64_t n, float* __restrict__ r, const float* __restrict__ Ap,
                                                Scalars* S, RedBuf rb) {
    if (S->done) return;
    const float av = (float)S->alpha;
    DotAcc<float> acc;
    const int64_t tid = blockIdx.x * (int64_t)NT + threadIdx.x, stride = (int64_t)gridDim.x * NT;
    const int64_t n4 = n / 4;
    for (int64_t q = tid; q < n4; q += stride) {
        float rv[4], av4[4];
        V4<float>::ld(r + 4 * q, rv);
        V4<float>::ld(Ap + 4 * q, av4);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            rv[k] = fma(-av, av4[k], rv[k]);
            acc.add(rv[k] * rv[k]);
        }
        V4<float>::st(r + 4 * q, rv);
    }
    for (int64_t i = 4 * n4 + tid; i < n; i += stride) {
        const float ri = fma(-av, Ap[i], r[i]);
        r[i] = ri;
        acc.add(ri * ri);
    }
    double v[1] = {acc.get()}, t[1];
    if (gridReduce<NT, 1>(v, rb, t)) applyEpi(EPI_CONV, S, t[0], 0.0);
}

// Mixed precision: fold the FP32 solution correction, and this iteration's
// deferred alpha p, into the FP64 solution.  conditional = 1: only when an FP64
// true-residual pass follows in this iteration (kUpdateR has run, so alpha p is
// pending; the stamp tells kUpdatePX it is folded).  conditional = 0 (after the
// last iteration): alpha p only if kUpdateR ran in the last iteration and
// neither a flush nor kUpdatePX has folded it.
__global__ void __launch_bounds__(256) kFlushX(int64_t n, double* __restrict__ x64, float* __restrict__ x32,
                                               const float* __restrict__ pFirst, const float* __restrict__ pSecond,
                                               Scalars* S, int conditional) {
    if (conditional && (S->done || !trueResidualDue(S))) return;
    const float* __restrict__ p = S->pSel ? pSecond : pFirst;
    const bool pending =
        conditional || (S->rStamp == S->matvecs && S->foldStamp != S->matvecs && S->pxStamp != S->matvecs);
    const double a = pending ? S->alpha : 0.0;
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
        x64[i] += (double)x32[i] + a * (double)p[i];
        x32[i] = 0.f;
    }
    if (conditional && blockIdx.x == 0 && threadIdx.x == 0) S->foldStamp = S->matvecs;
}

// Mixed precision: p = z + beta p, and the deferred x += alpha p (old p) of
// this iteration unless a flush has folded it.
__global__ void __launch_bounds__(256) kUpdatePX(int64_t n, float* __restrict__ p, const float* __restrict__ z,
                                                 float* __restrict__ x, Scalars* S) {
    if (S->done) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) S->pxStamp = S->matvecs;  // read only by kFlushX
    const float beta = (float)S->beta;
    const float ax = S->foldStamp == S->matvecs ? 0.f : (float)S->alpha;
    const int64_t tid = blockIdx.x * (int64_t)NT + threadIdx.x, stride = (int64_t)gridDim.x * NT;
    const int64_t n4 = n / 4;
    for (int64_t q = tid; q < n4; q += stride) {
        float pv[4], zv[4], xv[4];
        V4<float>::ld(p + 4 * q, pv);
        V4<float>::ld(z + 4 * q, zv);
        V4<float>::ld(x + 4 * q, xv);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            xv[k] = fma(ax, pv[k], xv[k]);
            pv[k] = fma(beta, pv[k], zv[k]);
        }
        V4<float>::st(p + 4 * q, pv);
        V4<float>::st(x + 4 * q, xv);
    }
    for (int64_t i = 4 * n4 + tid; i < n; i += stride) {
        x[i] = fma(ax, p[i], x[i]);
        p[i] = fma(beta, p[i], z[i]);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) kUpdateP(int64_t n, T* __restrict__ p, const T* __restrict__ z,
                                                const Scalars* S, int first) {
    if (S->done) return;
    const T beta = first ? T(0) : (T)S->beta;
    const int64_t tid = blockIdx.x * (int64_t)NT + threadIdx.x, stride = (int64_t)gridDim.x * NT;
    const int64_t n4 = n / 4;
    for (int64_t q = tid; q < n4; q += stride) {
        T pv[4], zv[4];
        V4<T>::ld(p + 4 * q, pv);
        V4<T>::ld(z + 4 * q, zv);
#pragma unroll
        for (int k = 0; k < 4; ++k) pv[k] = fma(beta, pv[k], zv[k]);
        V4<T>::st(p + 4 * q, pv);
    }
    for (int64_t i = 4 * n4 + tid; i < n; i += stride) p[i] = fma(beta, p[i], z[i]);
}

template <typename T>
__global__ void __launch_bounds__(256) kDots(int64_t n, const T* __restrict__ a, const T* __restrict__ b,
                                             const T* __restrict__ c, const T* __restrict__ d, int epi, Scalars* S,
                                             RedBuf rb, int checkDone) {
    if (checkDone && S->done) return;
    DotAcc<T> s0, s1;
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
        if (a) s0.add(a[i] * b[i]);
        if (c) s1.add(c[i] * d[i]);
    }
    double v[2] = {s0.get(), s1.get()}, t[2];
    if (gridReduce<NT, 2>(v, rb, t)) applyEpi(epi, S, t[0], t[1]);
}

// Deflation coarse space, part 1: t_j = v_j . r - (K v_j) . z (j < k; z may be
// null), reduced over the grid; the last block stores G^-1 t in the solver scalars.
template <typename T>
__global__ void __launch_bounds__(256) kCoarseDots(int64_t n, int k, const T* __restrict__ V,
                                                   const T* __restrict__ KV, const T* __restrict__ r,
                                                   const T* __restrict__ z, CoarseSpace G, Scalars* S, RedBuf rb,
                                                   int checkDone) {
    if (checkDone && S->done) return;
    DotAcc<T> acc[4];
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
        const T ri = r[i];
        const T zi = z ? z[i] : T(0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < k) {
                acc[j].add(V[(int64_t)j * n + i] * ri);
                if (z) acc[j].add(-KV[(int64_t)j * n + i] * zi);
            }
    }
    double v[4] = {acc[0].get(), acc[1].get(), acc[2].get(), acc[3].get()}, t[4];
    if (gridReduce<NT, 4>(v, rb, t)) {
        for (int a = 0; a < 4; ++a) {
            double sum = 0.0;
            for (int b = 0; b < k; ++b) sum += G.Ginv[4 * a + b] * t[b];
            S->coarseCoef[a] = a < k ? sum : 0.0;
        }
    }
}

// Part 2: z += sum_j coef_j v_j.
template <typename T>
__global__ void __launch_bounds__(256) kCoarseAxpy(int64_t n, int k, const T* __restrict__ V, T* __restrict__ z,
                                                   const Scalars* S, int checkDone) {
    if (checkDone && S->done) return;
    T cf[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) cf[j] = (T)S->coarseCoef[j];
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
        T zi = z[i];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < k) zi = fma(cf[j], V[(int64_t)j * n + i], zi);
        z[i] = zi;
    }
}

// Start projection: x += sum_j mu_j v_j, r -= sum_j mu_j (K v_j).
__global__ void __launch_bounds__(256) kCoarseStart(int64_t n, int k, const double* __restrict__ V,
                                                    const double* __restrict__ KV, const Scalars* S,
                                                    double* __restrict__ x, double* __restrict__ r) {
    double mu[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) mu[j] = S->coarseCoef[j];
    for (int64_t i = blockIdx.x * (int64_t)NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
        double xi = x[i], ri = r[i];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < k) {
                xi = fma(mu[j], V[(int64_t)j * n + i], xi);
                ri = fma(-mu[j], KV[(int64_t)j * n + i], ri);
            }
        x[i] = xi;
        r[i] = ri;
    }
}

template <typename TI, typename TO>
__global__ void kConvert(int64_t n, const TI* __restrict__ x, TO* __restrict__ y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = (TO)x[i];
}

template <typename T>
__global__ void kFill(int64_t n, T* __restrict__ y, T v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = v;
}

// Values between -1 and 1 without a pattern (a multiplicative hash) at used nodes.
__global__ void kNoise(int64_t n, const uint8_t* __restrict__ flags, double* __restrict__ y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        unsigned h = (unsigned)i * 2654435761u;
        h = (h ^ (h >> 15)) * 2246822519u;
        y[i] = (flags[i / 3] & FLAG_USED) ? (double)(int)(h ^ (h >> 13)) * 0x1p-31 : 0.0;
    }
}

template <typename T>
__global__ void kScatterCompressed(int64_t nn, const int32_t* __restrict__ store, const double* __restrict__ comp,
                                   T* __restrict__ dense, unsigned* bad) {
    bool ok = true;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 3 * nn; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = comp[i];
        ok = ok && isfinite(v);
        dense[3 * (int64_t)store[i / 3] + i % 3] = (T)v;
    }
    if (bad && !ok) atomicOr(bad, 1u);
}

template <typename T>
__global__ void kGatherCompressed(int64_t nn, const int32_t* __restrict__ store, const T* __restrict__ dense,
                                  double* __restrict__ comp) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 3 * nn; i += (int64_t)gridDim.x * blockDim.x)
        comp[i] = (double)dense[3 * (int64_t)store[i / 3] + i % 3];
}

// One parity colour of the coarsest-matrix assembly: same-colour elements share
// no node, so plain += is race-free and the summation order is fixed.
template <typename T>
__global__ void kAssembleCoarse(Grid g, const float* __restrict__ E, const int32_t* __restrict__ freeNode,
                                const Kd<double> ke, double scale, T* __restrict__ K, int64_t n, int color) {
    const int hx = (g.ex + 1 - (color & 1)) / 2, hy = (g.ey + 1 - ((color >> 1) & 1)) / 2;
    const int64_t e = blockIdx.x;
    const int ix = (int)(e % hx), iy = (int)((e / hx) % hy), iz = (int)(e / ((int64_t)hx * hy));
    const int x = 2 * ix + (color & 1), y = 2 * iy + ((color >> 1) & 1), z = 2 * iz + (color >> 2);
    if (x >= g.ex || y >= g.ey || z >= g.ez) return;
    const float Ee = E[g.store(x, y, z)];
    if (Ee == 0.f) return;
    for (int ent = threadIdx.x; ent < 576; ent += blockDim.x) {
        const int r = ent / 24, c = ent % 24;
        const int a = r / 3, ci = r % 3, b = c / 3, cj = c % 3;
        const int32_t na = freeNode[g.store(x + (a & 1), y + ((a >> 1) & 1), z + (a >> 2))];
        const int32_t nb = freeNode[g.store(x + (b & 1), y + ((b >> 1) & 1), z + (b >> 2))];
        if (na < 0 || nb < 0) continue;
        K[(3 * (int64_t)na + ci) * n + 3 * (int64_t)nb + cj] += (T)(scale * (double)Ee * ke.v[ent]);
    }
}

template <typename T>
__global__ void kSymmetrize(T* K, int64_t n) {
    // Column-major lower triangle (cuSOLVER) == row-major upper triangle: copy it down.
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / n, c = i % n;
        if (c < r) K[i] = K[c * n + r];
    }
}

__global__ void kInitScalars(Scalars* S, double tol, long long maxIter, int flexible, int mixed, int replaceEvery,
                             double delta, int breakAt) {
    Scalars s = {};
    s.breakAt = breakAt;
    s.tol2 = tol * tol;
    s.maxIter = maxIter;
    s.flexible = flexible;
    s.mixed = mixed;
    s.replaceEvery = replaceEvery;
    s.delta2 = mixed ? delta * delta : 0.0;
    s.rStamp = s.foldStamp = s.pxStamp = s.replStamp = -1;
    *S = s;
}

inline int flatBlocks(int64_t n) {
    int64_t b = (n + NT - 1) / NT;
    if (b > 152 * 8) b = 152 * 8;
    if (b < 1) b = 1;
    return (int)b;
}

// Blocks of the vector updates that also reduce (4 values a thread and step): each block's
// sum costs five FP64 additions a warp and a partial that the last block reads, so 3 an
// SM (8 for kUpdateR on large grids: 103 us to 257^3 instead of 110) and none without work.  kUpdateXR in FP64 with 8 an SM (one thread a value) / 4 / 3 /
// 2, us: 65^3 nodes 16.7 / 14.4 / 13.3 / 12.4, 129^3 61 / 56 / 54 / 58, 257^3 399 / 413 /
// 369 / 385; kUpdateR to 65^3 14.4 -> 9.1.
inline int reduceBlocks(int64_t n, int perSm) { return (int)std::min<int64_t>((n / 4 + NT) / NT, 152 * perSm); }

inline dim3 nodeGrid(const Grid& g) {
    return dim3((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + PZ - 1) / PZ);
}

}  // namespace

// ------------------------------------------------------------------ launchers

cudaError_t setKernelAttributes() {
    const int s64 = (kSuElems + kSyElems) * (int)sizeof(double), s32 = (kSuElems + kSyElems) * (int)sizeof(float);
    const cudaFuncAttribute A = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(kMatvecH<double, double>, A, s64))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<float, float>, A, s32))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<float, float, OUT_CG>, A, s32))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<float, float, OUT_CG_PX>, A, s32))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<float, float, OUT_ANY, Kc<float>>, A, s32))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<float, float, OUT_CG, Kc<float>>, A, s32))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<float, float, OUT_CG_PX, Kc<float>>, A, s32))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<double, double, OUT_CG>, A, s64))) return e;
    if ((e = cudaFuncSetAttribute(kMatvec<double>, A, s64))) return e;
    static_assert(sizeof(df) == sizeof(double), "the same shared memory");
    if ((e = cudaFuncSetAttribute(kMatvecH<double, df, OUT_TRUE>, A, s64))) return e;
    if ((e = cudaFuncSetAttribute(kMatvecH<double, df>, A, s64))) return e;
    if ((e = cudaFuncSetAttribute(kMatvec<double, df>, A, s64))) return e;
    return cudaFuncSetAttribute(kMatvec<float>, A, s32);
}

// Node layers a product block marches: the part count with the least (layers + repeated
// layer, prologue and epilogue) x (blocks an SM gets, at least `sat`: that many share an
// SM without slowing each other).  FP64 at every size, us with parts of up to 32 layers / this /
// the best of 15 lengths from 6 to 65, boxes with voids and moduli, random vectors:
// 65^3 nodes 68 / 45 / 47, 97^3 111 / 94 / 94, 129^3 197 / 180 / 179, 161^3 322 / 320 /
// 311, 193^3 486 / 496 / 486, 225^3 750 / 742 / 742, 257^3 1,077 / 1,050 / 1,050; the dense form 217 /
// 138 / 138, 466 / 386 / 385, 896 / 789 / 788, 1,480 / 1,444 / 1,435 (to 161^3).
int marchLayers(const Grid& g, int sat) {
    const int64_t tiles = (int64_t)((g.nx + MV_TX - 2) / (MV_TX - 1)) * ((g.ny + MV_TY - 2) / (MV_TY - 1));
    int best = g.nz;
    double least = 1e300;
    for (int parts = std::max(1, g.nz / 64); 2 * parts <= g.nz + 1; ++parts) {
        const int zc = (g.nz + parts - 1) / parts;
        const double perSm = std::ceil((double)(tiles * ((g.nz + zc - 1) / zc)) / 152.0);
        const double cost = (zc + 3.0) * std::max((double)sat, perSm);
        if (cost < least) {
            least = cost;
            best = zc;
        }
        if ((perSm > 8.0 && zc < 16) || perSm > 32.0) break;
    }
    return best;
}

// FP32: about 32 layers, in equal parts, where that gives two blocks an SM; longer
// marches wait on memory longer (with the direction update, 33 layers / marchLayers: 129^3
// 69.5 / 74 us, 193^3 187 / 213).  Smaller grids take marchLayers: 33 x 17 x 17 nodes
// 24.6 -> 12.3 us, 65^3 39 -> 21 us.
inline int productLayers(const Grid& g) {
    const int64_t tiles = (int64_t)((g.nx + MV_TX - 2) / (MV_TX - 1)) * ((g.ny + MV_TY - 2) / (MV_TY - 1));
    const int parts = std::max(1, (g.nz + MV_ZC / 2) / MV_ZC);
    return tiles * parts >= 2 * 152 ? (g.nz + parts - 1) / parts : marchLayers(g, 2);
}

// Layers of a march in the products of one type: the FP64 marches are bound by their
// operations, so marchLayers on every grid, with the blocks that share an SM.
template <typename T>
inline int layersFor(const Grid& g, bool structured) {
    if (std::is_same<T, double>::value) return marchLayers(g, structured ? 2 : 1);
    return structured ? productLayers(g) : MV_ZC;
}

// FP32 products with a structured Ke take the cube's constants where it is one.
template <typename T>
int launchMatvec(const LaunchCtx& c, const MatvecArgs<T>& a, bool structured, const void* opconst, const float* cube) {
    const Grid& g = a.g;
    const int zc = layersFor<T>(g, structured);
    dim3 grid((g.nx + MV_TX - 2) / (MV_TX - 1), (g.ny + MV_TY - 2) / (MV_TY - 1), (g.nz + zc - 1) / zc);
    dim3 block(MV_TX, MV_TY);
    size_t smem = (size_t)(kSuElems + kSyElems) * sizeof(T);
    const bool cg = a.mode == MV_AX && a.dot0 == DOT_X_OUT && !a.dot1 && !a.y32;
    auto go = [&](auto kern, const auto& k) { kern<<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb); };
    if (structured) {
        if constexpr (std::is_same<T, float>::value) {
            if (cube) {
                Kc<T> k;
                for (int i = 0; i < 8; ++i) k.v[i] = cube[i];
                if (cg) go(kMatvecH<T, T, OUT_CG, Kc<T>>, k);
                else go(kMatvecH<T, T, OUT_ANY, Kc<T>>, k);
                return 1;
            }
        }
        Ks<T> k;
        const T* src = static_cast<const T*>(opconst);
        for (int i = 0; i < 45; ++i) k.v[i] = src[i];
        if (cg) go(kMatvecH<T, T, OUT_CG>, k);
        else go(kMatvecH<T, T>, k);
    } else {
        Kd<T> k;
        const T* src = static_cast<const T*>(opconst) + 45;
        for (int i = 0; i < 576; ++i) k.v[i] = src[i];
        kMatvec<T><<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb);
    }
    return 1;
}

int launchMatvecDF(const LaunchCtx& c, const MatvecArgs<double>& a, bool structured, const double* opconst) {
    const Grid& g = a.g;
    const int zc = layersFor<float>(g, structured);  // its operations are FP32's
    dim3 grid((g.nx + MV_TX - 2) / (MV_TX - 1), (g.ny + MV_TY - 2) / (MV_TY - 1), (g.nz + zc - 1) / zc);
    dim3 block(MV_TX, MV_TY);
    const size_t smem = (size_t)(kSuElems + kSyElems) * sizeof(df);
    if (structured) {
        Ks<df> k;
        for (int i = 0; i < 45; ++i) k.v[i] = df(opconst[i]);
        if (a.mode == MV_RESID && a.dot0 == DOT_OUT_OUT && !a.dot1 && a.y32)
            kMatvecH<double, df, OUT_TRUE><<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb);
        else
            kMatvecH<double, df><<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb);
    } else {
        Kd<df> k;
        for (int i = 0; i < 576; ++i) k.v[i] = df(opconst[45 + i]);
        kMatvec<double, df><<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb);
    }
    return 1;
}

int launchMatvecPX(const LaunchCtx& c, const MatvecArgs<float>& a, const float* opconst, const float* cube) {
    const Grid& g = a.g;
    const int zc = productLayers(g);
    dim3 grid((g.nx + MV_TX - 2) / (MV_TX - 1), (g.ny + MV_TY - 2) / (MV_TY - 1), (g.nz + zc - 1) / zc);
    dim3 block(MV_TX, MV_TY);
    size_t smem = (size_t)(kSuElems + kSyElems) * sizeof(float);
    if (cube) {
        Kc<float> k;
        for (int i = 0; i < 8; ++i) k.v[i] = cube[i];
        kMatvecH<float, float, OUT_CG_PX, Kc<float>><<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb);
    } else {
        Ks<float> k;
        for (int i = 0; i < 45; ++i) k.v[i] = opconst[i];
        kMatvecH<float, float, OUT_CG_PX><<<grid, block, smem, c.stream>>>(a, k, zc, c.S, c.rb);
    }
    return 1;
}

template <typename T>
int launchRestrict(const LaunchCtx& c, const Grid& gf, const Grid& gc, int div, const T* rf, T* rc, int checkDone) {
    dim3 block(32, 8);
    if (div == 4) {
        kRestrict<T, 4><<<nodeGrid(gc), block, 0, c.stream>>>(gf, gc, rf, rc, c.S, checkDone);
    } else {
        if constexpr (std::is_same<T, float>::value) {
            if ((c.tma & 1) && launchRestrictTma(c, gf, gc, rf, nullptr, nullptr, rc, checkDone)) return 1;
        }
        if (gf.nnode <= kSmallRestrict) {
            kRestrictSmall<T><<<(unsigned)((3 * gc.nnode + 255) / 256), 256, 0, c.stream>>>(gf, gc, rf, rc, c.S, checkDone);
            return 1;
        }
        if constexpr (std::is_same<T, double>::value) {
            dim3 grid((gc.nx + 30) / 31, (gc.ny + 7) / 8, (gc.nz + PZR - 1) / PZR);
            kRestrict64<<<grid, block, 0, c.stream>>>(gf, gc, rf, rc, c.S, checkDone);
        } else {
            dim3 grid((gc.nx + 31) / 32, (gc.ny + 7) / 8, (gc.nz + PZR - 1) / PZR);
            kRestrict2<T, false><<<grid, block, 0, c.stream>>>(gf, gc, rf, nullptr, nullptr, rc, c.S, c.rb, checkDone);
        }
    }
    return 1;
}

int launchUpdateRestrict(const LaunchCtx& c, const Grid& gf, const Grid& gc, const float* rIn, const float* Ap,
                         float* rOut, float* rc) {
    if ((c.tma & 1) && launchRestrictTma(c, gf, gc, rIn, Ap, rOut, rc, 1)) return 1;
    const bool small = gf.nnode <= kSmallRestrict;
    const int pz = small ? 1 : PZR;
    dim3 block(32, 8), grid((gc.nx + 31) / 32, (gc.ny + 7) / 8, (gc.nz + pz - 1) / pz);
    auto kern = small ? kRestrict2<float, true, 1> : kRestrict2<float, true>;
    kern<<<grid, block, 0, c.stream>>>(gf, gc, rIn, Ap, rOut, rc, c.S, c.rb, 1);
    return 1;
}

template <typename T>
int launchProlongSmooth(const LaunchCtx& c, const Grid& gf, const Grid& gc, int div, const T* zc, const T* rf,
                        const T* dinv, const uint8_t* flags, T* zf, double coef, int maskFixed, const T* aux, int epi,
                        int checkDone, HalfDiag hd) {
    dim3 grid = nodeGrid(gf), block(32, 8);
    const int64_t flatBlocksN = (int64_t)prolongFlatRowGroups(gf) * gf.nz;
    const size_t flatSmem = 2 * sizeof(T) * kProlongCoarseRows * 3 * (size_t)gc.nx;
    if (div == 2 && flatBlocksN <= kMaxRedBlocks && flatSmem <= kProlongFlatMaxSmem) {
        auto al = [](const void* q) { return ((uintptr_t)q & 15u) == 0; };
        const bool half = std::is_same<T, float>::value && hd.d != nullptr;
        const int vec = al(rf) && al(zf) && ((uintptr_t)flags & 3u) == 0 &&
                        (half ? ((uintptr_t)hd.d & 7u) == 0 : al(dinv));
        // (FP32)
        auto go = [&](auto kern, const auto* dptr, double cf) {
            typedef typename std::remove_const<typename std::remove_pointer<decltype(dptr)>::type>::type DT;
            if (gf.nnode <= kSmallProlong) {
                // (few enough blocks for a cheap grid reduction)
                const int64_t blocks = std::min<int64_t>((3 * gf.nnode + 255) / 256, 152 * 2);
                kProlongSmall<T, DT><<<(unsigned)blocks, 256, 0, c.stream>>>(
                    gf, gc, zc, rf, dptr, flags, zf, cf, maskFixed, aux, epi, c.S, c.rb, checkDone);
                return;
            }
            if (flatSmem > 48 * 1024)
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProlongFlatMaxSmem);
            kern<<<(unsigned)flatBlocksN, kProlongThreads, flatSmem, c.stream>>>(gf, gc, zc, rf, dptr, flags, zf, cf, maskFixed, aux,
                                                                     epi, vec, 1.0f / gf.nx, c.S, c.rb, checkDone);
        };
        if constexpr (std::is_same<T, float>::value) {
            if (half) {
                if ((c.tma & 2) && launchProlongBulk(c, gf, gc, zc, rf, hd.d, flags, zf, coef * (double)hd.scale, maskFixed,
                                               aux, epi, checkDone))
                    return 1;
                go(kProlongFlat<float, __half>, hd.d, coef * (double)hd.scale);
                return 1;
            }
        }
        if constexpr (std::is_same<T, double>::value) {
            auto go64 = [&](auto rowsTag, auto nthTag) {
                constexpr int ROWS = decltype(rowsTag)::value, NTH = decltype(nthTag)::value;
                const int64_t blocks = (int64_t)((gf.ny + ROWS - 1) / ROWS) * gf.nz;
                const size_t smem = 2 * sizeof(double) * (ROWS / 2 + 1) * 3 * (size_t)gc.nx;
                if (smem > 48 * 1024)
                    cudaFuncSetAttribute(kProlong64<ROWS, NTH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kProlongFlatMaxSmem);
                kProlong64<ROWS, NTH><<<(unsigned)blocks, NTH, smem, c.stream>>>(
                    gf, gc, zc, rf, dinv, flags, zf, coef, maskFixed, aux, epi, vec, 1.0f / gf.nx, c.S, c.rb, checkDone);
            };
            // 16 rows where that gives 4 blocks an SM, else 8 where those give 2, else 4
            using std::integral_constant;
            const auto blocksOf = [&](int rows) { return (int64_t)((gf.ny + rows - 1) / rows) * gf.nz; };
            if (blocksOf(16) >= 4 * 152) go64(integral_constant<int, 16>(), integral_constant<int, 256>());
            else if (blocksOf(8) >= 2 * 152) go64(integral_constant<int, 8>(), integral_constant<int, 128>());
            else go64(integral_constant<int, 4>(), integral_constant<int, 128>());
        } else {
            go(kProlongFlat<float, float>, dinv, coef);
        }
    } else if (div == 2) {
        // grids beyond the flat kernel's block or shared-memory limits (over ~1000^3 nodes)
        dim3 cgrid((gc.nx + 31) / 32, (gc.ny + 7) / 8, (gc.nz + PZC - 1) / PZC);
        kProlongSmooth2<T><<<cgrid, block, 0, c.stream>>>(gf, gc, zc, rf, dinv, flags, zf, coef, maskFixed, aux, epi,
                                                          c.S, c.rb, checkDone);
    } else if (div == 4)
        kProlongSmooth<T, 4><<<grid, block, 0, c.stream>>>(gf, gc, zc, rf, dinv, flags, zf, coef, maskFixed, aux, epi,
                                                             c.S, c.rb, checkDone);
    else
        kProlongSmooth<T, 2><<<grid, block, 0, c.stream>>>(gf, gc, zc, rf, dinv, flags, zf, coef, maskFixed, aux, epi,
                                                             c.S, c.rb, checkDone);
    return 1;
}

template <typename T>
int launchJacobiZero(const LaunchCtx& c, const Grid& g, const T* r, const T* dinv, const uint8_t* flags, T* z,
                     double omega, int checkDone) {
    kJacobiZero<T><<<flatBlocks(g.nnode), NT, 0, c.stream>>>(g.nnode, r, dinv, flags, z, omega, c.S, checkDone);
    return 1;
}

template <typename T>
int launchProlongAdd(const LaunchCtx& c, const Grid& gf, const Grid& gc, int div, const T* zc, const uint8_t* flags,
                     T* zf, int checkDone) {
    dim3 grid = nodeGrid(gf), block(32, 8);
    if (div == 4) kProlongAdd<T, 4><<<grid, block, 0, c.stream>>>(gf, gc, zc, flags, zf, c.S, checkDone);
    else kProlongAdd<T, 2><<<grid, block, 0, c.stream>>>(gf, gc, zc, flags, zf, c.S, checkDone);
    return 1;
}

template <typename T>
int launchCoarseSolve(const LaunchCtx& c, CoarseInv<T> Kinv, int64_t n, const int32_t* freeDof, const T* rc, T* tmp,
                      T* part, T* zc, int checkDone) {
    if (n <= 0) return 0;
    if (n <= kSmallCoarse<T>) {
        const unsigned blocks = (unsigned)((n + 7) / 8);
        if constexpr (std::is_same<T, double>::value)
            kCoarseSmall<double, double><<<blocks, 256, 0, c.stream>>>(Kinv.K, (int)n, (int)n, 1.0, freeDof, rc, zc, c.S,
                                                                       checkDone);
        else
            kCoarseSmall<float, __half><<<blocks, 256, 0, c.stream>>>(Kinv.K, (int)n, (int)coarseLd(n), Kinv.scale,
                                                                      freeDof, rc, zc, c.S, checkDone);
        return 1;
    }
    kCoarseGather<T><<<(int)((n + 255) / 256), 256, 0, c.stream>>>(n, freeDof, rc, tmp, c.S, checkDone);
    if constexpr (std::is_same<T, double>::value) {
        kGemv64<<<(int)((n * 32 + 255) / 256), 256, 0, c.stream>>>(Kinv.K, n, tmp, freeDof, zc, c.S, checkDone);
        return 2;
    } else {
        const int64_t nb = coarseBlocks(n);
        kSymRuns<<<(unsigned)std::min<int64_t>((coarseTiles(n) + SYM_WARPS - 1) / SYM_WARPS, SYM_BLOCKS), 32 * SYM_WARPS, 0,
                   c.stream>>>(Kinv.K, tmp, part, nb, c.S, checkDone);
        kSymRunsReduce<<<(unsigned)nb, 1024, 0, c.stream>>>(part, nb, n, freeDof, Kinv.scale, zc, c.S, checkDone);
        return 3;
    }
}

int launchMaxAbs(cudaStream_t s, const float* x, int64_t n, unsigned* outBits) {
    kMaxAbs<<<flatBlocks(n), NT, 0, s>>>(x, n, outBits);
    return 1;
}

int launchToHalf(cudaStream_t s, const float* x, int64_t n, float invScale, __half* y) {
    kToHalf<<<flatBlocks(n), NT, 0, s>>>(x, n, invScale, y);
    return 1;
}

int launchMaxDiag(cudaStream_t s, const float* K, int64_t n, float* out) {
    kMaxDiag<<<1, 1024, 0, s>>>(K, n, out);
    return 1;
}

int launchPackSymHalf(cudaStream_t s, const float* K, int64_t n, float invScale, __half* tiles) {
    if (n <= kSmallCoarse<float>) {
        kPackRowsHalf<<<flatBlocks(n * coarseLd(n)), NT, 0, s>>>(K, (int)n, (int)coarseLd(n), invScale, tiles);
        return 1;
    }
    const int64_t nb = coarseBlocks(n);
    kPackSymHalf<<<flatBlocks(symTileCount(nb) * CT * CT), NT, 0, s>>>(K, n, nb, invScale, tiles);
    return 1;
}

template <typename TX, typename TV>
int launchUpdateXR(const LaunchCtx& c, int64_t n, TX* x, TV* r, const TV* p, const TV* Ap) {
    kUpdateXR<TX, TV><<<reduceBlocks(n, 3), NT, 0, c.stream>>>(n, x, r, p, Ap, c.S, c.rb);
    return 1;
}

int launchFlushX(const LaunchCtx& c, int64_t n, double* x64, float* x32, const float* p, const float* pAlt,
                 int conditional) {
    kFlushX<<<flatBlocks(n), NT, 0, c.stream>>>(n, x64, x32, p, pAlt ? pAlt : p, c.S, conditional);
    return 1;
}

int launchUpdateR(const LaunchCtx& c, int64_t n, float* r, const float* Ap) {
    kUpdateR<<<reduceBlocks(n, n > 4 * NT * 152 * 8 ? 8 : 3), NT, 0, c.stream>>>(n, r, Ap, c.S, c.rb);
    return 1;
}

int launchUpdatePX(const LaunchCtx& c, int64_t n, float* p, const float* z, float* x) {
    kUpdatePX<<<flatBlocks(n), NT, 0, c.stream>>>(n, p, z, x, c.S);
    return 1;
}

template <typename T>
int launchUpdateP(const LaunchCtx& c, int64_t n, T* p, const T* z, int first) {
    kUpdateP<T><<<flatBlocks(n), NT, 0, c.stream>>>(n, p, z, c.S, first);
    return 1;
}

template <typename T>
int launchDots(const LaunchCtx& c, int64_t n, const T* a, const T* b, const T* cc, const T* d, int epi, int checkDone) {
    kDots<T><<<flatBlocks(n), NT, 0, c.stream>>>(n, a, b, cc, d, epi, c.S, c.rb, checkDone);
    return 1;
}

template <typename T>
int launchCoarseSpace(const LaunchCtx& c, int64_t n, int k, const T* V, const T* KV, const CoarseSpace& G,
                      const T* r, T* z, int checkDone) {
    kCoarseDots<T><<<flatBlocks(n), NT, 0, c.stream>>>(n, k, V, KV, r, z, G, c.S, c.rb, checkDone);
    kCoarseAxpy<T><<<flatBlocks(n), NT, 0, c.stream>>>(n, k, V, z, c.S, checkDone);
    return 2;
}

int launchCoarseStart(const LaunchCtx& c, int64_t n, int k, const double* V, const double* KV, const CoarseSpace& G,
                      double* x, double* r) {
    kCoarseDots<double><<<flatBlocks(n), NT, 0, c.stream>>>(n, k, V, KV, r, nullptr, G, c.S, c.rb, 0);
    kCoarseStart<<<flatBlocks(n), NT, 0, c.stream>>>(n, k, V, KV, c.S, x, r);
    return 2;
}

template <typename TI, typename TO>
int launchConvert(cudaStream_t s, int64_t n, const TI* x, TO* y) {
    kConvert<TI, TO><<<flatBlocks(n), NT, 0, s>>>(n, x, y);
    return 1;
}

template <typename T>
int launchFill(cudaStream_t s, int64_t n, T* y, T v) {
    kFill<T><<<flatBlocks(n), NT, 0, s>>>(n, y, v);
    return 1;
}

int launchNoise(cudaStream_t s, int64_t n, const uint8_t* flags, double* y) {
    kNoise<<<flatBlocks(n), NT, 0, s>>>(n, flags, y);
    return 1;
}

template <typename T>
int launchScatterCompressed(cudaStream_t s, int64_t nn, const int32_t* store, const double* comp, T* dense,
                            unsigned* bad) {
    kScatterCompressed<T><<<flatBlocks(3 * nn), NT, 0, s>>>(nn, store, comp, dense, bad);
    return 1;
}

template <typename T>
int launchGatherCompressed(cudaStream_t s, int64_t nn, const int32_t* store, const T* dense, double* comp) {
    kGatherCompressed<T><<<flatBlocks(3 * nn), NT, 0, s>>>(nn, store, dense, comp);
    return 1;
}

template <typename T>
int launchAssembleCoarse(cudaStream_t s, const Grid& g, const float* E, const int32_t* freeNode, const double* Ke,
                         double scale, T* K, int64_t n) {
    Kd<double> k;
    for (int i = 0; i < 576; ++i) k.v[i] = Ke[i];
    int launches = 0;
    for (int color = 0; color < 8; ++color) {
        const int hx = (g.ex + 1 - (color & 1)) / 2, hy = (g.ey + 1 - ((color >> 1) & 1)) / 2,
                  hz = (g.ez + 1 - (color >> 2)) / 2;
        const int64_t ne = (int64_t)hx * hy * hz;
        if (ne <= 0) continue;
        kAssembleCoarse<T><<<(unsigned)ne, 64, 0, s>>>(g, E, freeNode, k, scale, K, n, color);
        ++launches;
    }
    return launches;
}

template <typename T>
__global__ void kZeroStrictRowMajorLower(T* K, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / n, c = i - r * n;
        if (c < r) K[i] = T(0);
    }
}

template <typename T>
int launchZeroStrictRowMajorLower(cudaStream_t s, T* K, int64_t n) {
    kZeroStrictRowMajorLower<T><<<flatBlocks(n * n), NT, 0, s>>>(K, n);
    return 1;
}

template <typename T>
int launchSymmetrizeLowerToFull(cudaStream_t s, T* K, int64_t n) {
    kSymmetrize<T><<<flatBlocks(n * n), NT, 0, s>>>(K, n);
    return 1;
}

int launchInitScalars(cudaStream_t s, Scalars* S, double tol, long long maxIter, int flexible, int mixed,
                      int replaceEvery, double replaceDelta, int breakAt) {
    kInitScalars<<<1, 1, 0, s>>>(S, tol, maxIter, flexible, mixed, replaceEvery, replaceDelta, breakAt);
    return 1;
}

// ------------------------------------------------------------------ no-allocation product
//
// Scratch of vfem_apply_operator_device_noalloc: the reduction partials, the
// ticket and the scalar block of the fused x.(Kx) dot live in this file-scope
// device array instead of memory from cudaMalloc.  Fixed size: 2 x 65,536 block
// partials + 1 KiB (1,049,600 bytes); every GPU that loads the library holds it
// until the process exits.  All calls share it, so calls that overlap on the GPU
// race; each call clears the ticket and scalars before its kernel.
namespace {
// Partials of the product's grid reduction, which carries two sums per block
// (x.(Kx) and the unused second dot).
constexpr size_t kNoAllocPartialBytes = 2 * (size_t)kMaxRedBlocks * sizeof(double);
constexpr size_t kNoAllocBytes = kNoAllocPartialBytes + 1024;
static_assert(sizeof(Scalars) + 256 <= 1024, "scalar block does not fit the no-allocation scratch");
__device__ __align__(256) unsigned char g_noallocScratch[kNoAllocBytes];
std::mutex g_noallocMutex;
constexpr int kNoAllocMaxDevices = 64;
void* g_noallocAddr[kNoAllocMaxDevices] = {};
}  // namespace

cudaError_t noallocScratchSetup() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noallocMutex);
    if (g_noallocAddr[dev]) return cudaSuccess;
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_noallocScratch);  // the host-side name is not a device address
    if (e != cudaSuccess) return e;
    g_noallocAddr[dev] = ptr;
    return cudaSuccess;
}

cudaError_t launchMatvecNoAlloc(cudaStream_t s, const MatvecArgs<double>& a, bool structured, const void* opconst,
                                const FxOperand& fx, double* xKx, bool* tooLarge) {
    const Grid& g = a.g;
    dim3 grid((g.nx + MV_TX - 2) / (MV_TX - 1), (g.ny + MV_TY - 2) / (MV_TY - 1), (g.nz + MV_ZC - 1) / MV_ZC);
    *tooLarge = (int64_t)grid.x * grid.y * grid.z > kMaxRedBlocks;
    if (*tooLarge) return cudaSuccess;
    cudaError_t e = noallocScratchSetup();
    if (e != cudaSuccess) return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    unsigned char* base = static_cast<unsigned char*>(g_noallocAddr[dev]);
    RedBuf rb{reinterpret_cast<double*>(base), reinterpret_cast<unsigned*>(base + kNoAllocPartialBytes)};
    Scalars* S = reinterpret_cast<Scalars*>(base + kNoAllocPartialBytes + 256);
    // The ticket and the scalars must start at zero; the partials are overwritten.
    if ((e = cudaMemsetAsync(base + kNoAllocPartialBytes, 0, 1024, s)) != cudaSuccess) return e;
    MatvecArgs<double> b = a;
    b.mode = MV_AX;
    b.dot0 = DOT_X_OUT;
    b.dot1 = 0;
    b.epi = EPI_STORE;
    b.checkDone = 0;
    b.condTrue = 0;
    size_t smem = (size_t)(kSuElems + kSyElems) * sizeof(double);
    dim3 block(MV_TX, MV_TY);
    const int zc = layersFor<double>(g, structured);
    grid.z = (g.nz + zc - 1) / zc;
    if (fxEligible(fx, b.scale)) {
        launchMatvecFx(s, b, fx, static_cast<const double*>(opconst), S, rb);
    } else if (structured) {
        Ks<double> k;
        for (int i = 0; i < 45; ++i) k.v[i] = static_cast<const double*>(opconst)[i];
        kMatvecH<double, double><<<grid, block, smem, s>>>(b, k, zc, S, rb);
    } else {
        Kd<double> k;
        for (int i = 0; i < 576; ++i) k.v[i] = static_cast<const double*>(opconst)[45 + i];
        kMatvec<double><<<grid, block, smem, s>>>(b, k, zc, S, rb);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return cudaMemcpyAsync(xKx, &S->red0, sizeof(double), cudaMemcpyDeviceToDevice, s);
}

// ------------------------------------------------------------------ instantiations
#define INST_T(T)                                                                                                     \
    template int launchMatvec<T>(const LaunchCtx&, const MatvecArgs<T>&, bool, const void*, const float*);                            \
    template int launchRestrict<T>(const LaunchCtx&, const Grid&, const Grid&, int, const T*, T*, int);               \
    template int launchProlongSmooth<T>(const LaunchCtx&, const Grid&, const Grid&, int, const T*, const T*,          \
                                        const T*, const uint8_t*, T*, double, int, const T*, int, int, HalfDiag);    \
    template int launchJacobiZero<T>(const LaunchCtx&, const Grid&, const T*, const T*, const uint8_t*, T*, double,  \
                                     int);                                                                           \
    template int launchProlongAdd<T>(const LaunchCtx&, const Grid&, const Grid&, int, const T*, const uint8_t*, T*,  \
                                     int);                                                                           \
    template int launchCoarseSolve<T>(const LaunchCtx&, CoarseInv<T>, int64_t, const int32_t*, const T*, T*, T*,    \
                                      T*, int);                                                                      \
    template int launchUpdateP<T>(const LaunchCtx&, int64_t, T*, const T*, int);                                     \
    template int launchCoarseSpace<T>(const LaunchCtx&, int64_t, int, const T*, const T*, const CoarseSpace&, const T*, T*, int); \
    template int launchDots<T>(const LaunchCtx&, int64_t, const T*, const T*, const T*, const T*, int, int);         \
    template int launchFill<T>(cudaStream_t, int64_t, T*, T);                                                        \
    template int launchScatterCompressed<T>(cudaStream_t, int64_t, const int32_t*, const double*, T*, unsigned*);    \
    template int launchGatherCompressed<T>(cudaStream_t, int64_t, const int32_t*, const T*, double*);               \
    template int launchAssembleCoarse<T>(cudaStream_t, const Grid&, const float*, const int32_t*, const double*,     \
                                         double, T*, int64_t);                                                       \
    template int launchSymmetrizeLowerToFull<T>(cudaStream_t, T*, int64_t);                                          \
    template int launchZeroStrictRowMajorLower<T>(cudaStream_t, T*, int64_t);
INST_T(double)
INST_T(float)
template int launchUpdateXR<double, double>(const LaunchCtx&, int64_t, double*, double*, const double*, const double*);
template int launchConvert<double, float>(cudaStream_t, int64_t, const double*, float*);
template int launchConvert<float, double>(cudaStream_t, int64_t, const float*, double*);
template int launchConvert<double, double>(cudaStream_t, int64_t, const double*, double*);
template int launchConvert<float, float>(cudaStream_t, int64_t, const float*, float*);

}  // namespace vfem
