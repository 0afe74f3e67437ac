// unet.cu -- the learned part of the solver: a small 3-D U-Net on the node grid
// (inputs: occupancy, modulus, fixed mask, load; output: displacement), trained
// and run with this file's own kernels.  No reference counterpart.
//
// Numerics: activations and weights in BF16, every product accumulated in FP32
// on the tensor cores (mma.sync m16n8k16 bf16 -> f32), FP32 master weights and
// Adam moments.  Layout: channels-last [voxel][channel] on an n^3 grid (n a
// multiple of 8), x fastest.
//
// Network (4 levels, 16-32-64-128 channels; every conv is 3x3x3, zero padded):
//   e0 = relu(conv(x, 16->16))        @ n      p1 = avgpool2(e0)
//   e1 = relu(conv(p1, 16->32))       @ n/2    p2 = avgpool2(e1)
//   e2 = relu(conv(p2, 32->64))       @ n/4    p3 = avgpool2(e2)
//   e3 = relu(conv(p3, 64->128))      @ n/8
//   d2 = relu(conv([up2(e3), e2], 192->64))  @ n/4
//   d1 = relu(conv([up2(d2), e1],  96->32))  @ n/2
//   d0 = relu(conv([up2(d1), e0],  48->16))  @ n
//   y  = conv(d0, 16->16)  (channels 0..2 are the prediction)
// Kernels: kConv (implicit GEMM; also the data gradient with flipped, transposed
// weights; reads [up2(a), b] in place), kWGrad (weight and bias gradient, split
// over voxels), pooling, split of the decoder's gradient, ReLU mask, masked MSE,
// Adam.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>
#include <vector>

#include "host_copy.h"
#include "vfem_net.h"

namespace {

thread_local std::string g_netError;

constexpr int kLayers = 8;
// (Cin, Cout, level) of the 8 convolutions; all but the last end in a relu.
constexpr int kCin[kLayers] = {16, 16, 32, 64, 192, 96, 48, 16};
constexpr int kCout[kLayers] = {16, 32, 64, 128, 64, 32, 16, 16};
constexpr int kLevel[kLayers] = {0, 1, 2, 3, 2, 1, 0, 0};
__constant__ int d_cin[kLayers] = {16, 16, 32, 64, 192, 96, 48, 16};
__constant__ int d_cout[kLayers] = {16, 32, 64, 128, 64, 32, 16, 16};

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ----------------------------------------------------------------------------- convolution
// Implicit GEMM: out[v][co] = sum_{tap, ci} in[v + off(tap)][ci] * W[tap][ci][co] (+ bias, relu),
// summed tap by tap and 16 channels at a time (the order every shape keeps).
//
// A block stages the halo of an 8 x 8 x TZ voxel tile, all channels, in shared
// memory once and reads the 27 shifted operands from there with ldmatrix: a
// voxel's 16 channels are one 32-byte row, so a shift is only an address.  A row
// of 16 voxels is two x rows of 8; the voxel stride of 32 CK + 16 bytes puts any
// 8 of them in different banks.  Each of the 2 TZ warps owns 32 voxels and all
// 8 NT output channels of the block.  Weights pass through shared memory in
// stages of TG taps, double-buffered; where all 27 fit (TG = 27) they stay for
// the block's further tiles.  The input may be two tensors: channels [0, Ca)
// from `a` at half resolution (nearest upsampling) and the rest from `b`, which
// spares writing the decoder's concatenation.
//
// The earlier kernel staged 64 x 16 operands for every tap and 16 channels from
// global memory (index arithmetic, two barriers and 2 to 8 MMAs a step).
// Measured on GB300, 16 -> 16 channels at 136^3: 687 -> 134 us; 48 -> 16 there with
// the concatenation: 2,480 -> 441 us; 192 -> 64 at 34^3: 396 -> 138 us; same bits.
// Bound: shared-memory reads of A (512 bytes for 2 NT MMAs) where NT = 2.
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// 16-byte asynchronous copy; zeros when !ok (src must be a valid address all the same).
__device__ __forceinline__ void cpAsync16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cpCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpWait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// An activation tensor read by the GEMM kernels: channels [0, Ca) of `a` at half
// resolution, then Cb of `b` (Ca = 0: b alone).
struct Input {
    const bf16* a;
    const bf16* b;
    int Ca, Cb;
};

constexpr int HALO = 10;  // tile edge 8 and one voxel on each side
template <int CK>
__host__ __device__ constexpr int rowBytes() { return 32 * CK + 16; }

// Copies the halo of the tile at (x0, y0, z0), TZ + 2 layers of 10 x 10 voxels, zeros outside the grid.
template <int CK, int TZ, int NTH>
__device__ __forceinline__ void stageHalo(uint32_t dst, const Input& in, int n, int x0, int y0, int z0) {
    constexpr int Q = 2 * CK, TOT = HALO * HALO * (TZ + 2) * Q;
    const int nh = n >> 1;
    for (int i = threadIdx.x; i < TOT; i += NTH) {
        const int q = i % Q, h = i / Q;
        const int hx = h % HALO, hy = (h / HALO) % HALO, hz = h / (HALO * HALO);
        const int x = x0 + hx - 1, y = y0 + hy - 1, z = z0 + hz - 1;
        const bool ok = x >= 0 && x < n && y >= 0 && y < n && z >= 0 && z < n;
        const bf16* src = in.b;
        if (ok) {
            const int c = 8 * q;
            if (c < in.Ca) src = in.a + ((((int64_t)(z >> 1) * nh + (y >> 1)) * nh + (x >> 1)) * in.Ca + c);
            else src = in.b + ((((int64_t)z * n + y) * n + x) * in.Cb + c - in.Ca);
        }
        cpAsync16(dst + (uint32_t)(h * rowBytes<CK>() + 16 * q), src, ok);
    }
}

// a weight row: 8 NT channels, any 8 rows in different banks
template <int NT>
__host__ __device__ constexpr int wRowBytes() { return NT == 1 ? 48 : 16 * NT + 16; }

template <int CK, int NT, int TG, int TZ>
constexpr size_t convSmem() {
    return (size_t)HALO * HALO * (TZ + 2) * rowBytes<CK>() +
           (size_t)(TG == 27 ? 1 : 2) * TG * 16 * CK * wRowBytes<NT>();
}

// OUT_PRED: the network's 3 output channels, FP32 [V][3] (NT = 1: their 8-channel tile alone).
// OUT_MASKED: the data gradient through the relu of `act` (the tensor it is the gradient of), BF16.
enum ConvOut { OUT_BF16, OUT_F32, OUT_MASKED, OUT_PRED };
template <int CK, int NT, int TG, int TZ, ConvOut OUT>
__global__ void __launch_bounds__(64 * TZ) kConv(const Input in, const bf16* __restrict__ W,
                                                 const float* __restrict__ bias, const bf16* __restrict__ act,
                                                 void* __restrict__ out, int n, int Cout, int relu) {
    constexpr int NTH = 64 * TZ, NS = 27 / TG, ROW = rowBytes<CK>(), WROW = wRowBytes<NT>();
    constexpr uint32_t haloBytes = HALO * HALO * (TZ + 2) * ROW, stageBytes = TG * 16 * CK * WROW;
    extern __shared__ __align__(16) unsigned char convSm[];
    const uint32_t sA = (uint32_t)__cvta_generic_to_shared(convSm), sB = sA + haloBytes;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * (8 * NT);
    const int tx = (n + 7) >> 3, tz = (n + TZ - 1) / TZ, tiles = tx * tx * tz;
    auto stageW = [&](int s, int buf) {
        constexpr int Q = NT, TOT = TG * 16 * CK * Q;  // 16-byte pieces
        for (int i = tid; i < TOT; i += NTH) {
            const int q = i % Q, k = i / Q;
            cpAsync16(sB + buf * stageBytes + k * WROW + 16 * q,
                      W + ((int64_t)s * TG * 16 * CK + k) * Cout + n0 + 8 * q, true);
        }
    };
    // ldmatrix addresses of this lane: A row (lane & 15) of the warp's first 16 voxels,
    // channel half lane >> 4; B row k, column half
    const int wz = warp >> 1, wy = (warp & 1) * 4;
    const uint32_t aLane =
        sA + (uint32_t)(((wz * HALO + wy + ((lane >> 3) & 1)) * HALO + (lane & 7)) * ROW + 16 * (lane >> 4));
    const uint32_t bLane = sB + (uint32_t)(((lane & 7) + 8 * ((lane >> 3) & 1)) * WROW + 16 * (lane >> 4));
    if (NS == 1) stageW(0, 0);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int x0 = (tile % tx) * 8, y0 = (tile / tx) % tx * 8, z0 = tile / (tx * tx) * TZ;
        stageHalo<CK, TZ, NTH>(sA, in, n, x0, y0, z0);
        if (NS > 1) stageW(0, 0);
        cpCommit();
        float acc[2][NT][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][j][e] = 0.f;
        for (int s = 0; s < NS; ++s) {
            cpWait<0>();
            __syncthreads();
            if (s + 1 < NS) {
                stageW(s + 1, (s + 1) & 1);
                cpCommit();
            }
            const uint32_t b0 = bLane + (NS > 1 ? (s & 1) * stageBytes : 0);
#pragma unroll 3
            for (int t = 0; t < TG; ++t) {
                const int tap = s * TG + t;
                const uint32_t aTap =
                    aLane + (uint32_t)((((tap / 9) * HALO + (tap / 3) % 3) * HALO + tap % 3) * ROW);
#pragma unroll
                for (int c = 0; c < CK; ++c) {
                    uint32_t A[2][4];
                    ldsm4(A[0], aTap + 32 * c);
                    ldsm4(A[1], aTap + 32 * c + 2 * HALO * ROW);
#pragma unroll
                    for (int j = 0; j < NT; j += 2) {
                        uint32_t B[4];  // (NT = 1: the upper half is the row's padding, unused)
                        ldsm4t(B, b0 + (uint32_t)((t * CK + c) * 16 * WROW + 16 * j));
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            mma16816(acc[m][j], A[m][0], A[m][1], A[m][2], A[m][3], B[0], B[1]);
                            if constexpr (NT > 1)
                                mma16816(acc[m][j + 1], A[m][0], A[m][1], A[m][2], A[m][3], B[2], B[3]);
                        }
                    }
                }
            }
        }
        const int g = lane >> 2, t4 = lane & 3, x = x0 + g, z = z0 + wz;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int hrow = 0; hrow < 2; ++hrow) {
                const int y = y0 + wy + 2 * m + hrow;
                if (x >= n || y >= n || z >= n) continue;
                const int64_t v = ((int64_t)z * n + y) * n + x;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const int co = n0 + 8 * j + 2 * t4;
                    float r0 = acc[m][j][2 * hrow] + (bias ? bias[co] : 0.f);
                    float r1 = acc[m][j][2 * hrow + 1] + (bias ? bias[co + 1] : 0.f);
                    if (relu) {
                        r0 = fmaxf(r0, 0.f);
                        r1 = fmaxf(r1, 0.f);
                    }
                    if (OUT == OUT_MASKED) {
                        const uint32_t y = *reinterpret_cast<const uint32_t*>(act + v * Cout + co);
                        if (!(__uint_as_float(y << 16) > 0.f)) r0 = 0.f;
                        if (!(__uint_as_float(y & 0xffff0000u) > 0.f)) r1 = 0.f;
                    }
                    if (OUT == OUT_PRED) {
                        float* o = static_cast<float*>(out) + v * 3 + co;
                        if (co < 3) o[0] = r0;
                        if (co + 1 < 3) o[1] = r1;
                    } else if (OUT == OUT_F32)
                        *reinterpret_cast<float2*>(static_cast<float*>(out) + v * Cout + co) = make_float2(r0, r1);
                    else
                        *reinterpret_cast<__nv_bfloat162*>(static_cast<bf16*>(out) + v * Cout + co) =
                            __floats2bfloat162_rn(r0, r1);
                }
            }
        __syncthreads();  // the halo is free for the next tile
    }
}

// Weight and bias gradient: dW[tap][ci][co] = sum_v in[v + off(tap)][ci] g[v][co], db[co] = sum_v g[v][co].
//
// A warp owns 16 MT x 8 NT (ci, co) of the three dx taps of one (dy, dz) over
// WG_CHUNK consecutive voxels, WG_SUB at a time; a block is the three dy of one dz
// (blockIdx.z).  With voxels in storage order a tap is a shift by dx + n dy +
// n^2 dz, so a warp stages a run of WG_SUB + 2 input voxels and WG_SUB of g for
// itself, in a ring of WG_BUFS buffers, and needs no block barrier.  A step is 16 voxels as the MMA's
// K, both operands by transposing ldmatrix, whose per-row addresses send a voxel
// without that neighbour to a row of zeros.  The bias is one more MMA against
// ones, in the (0, 0) warp of the first ci block.  The chunk's sums go to its
// slice of part ([chunk][27 Cin Cout weights, Cout biases], the parameters'
// layout) and kGradSum adds the slices in order: the order of the sums depends
// on the voxel numbering alone, so the gradient is bit-reproducible.
//
// The earlier kernel staged both operands for every tap, element by element for
// the transpose, and the bias ran in one block per channel.  Measured on GB300 at
// 72^3, weights and bias: 16 x 16 channels 855 -> 64 us, 48 x 16 1,024 -> 104 us,
// 96 x 32 (36^3) 297 -> 75 us; the weights with the same bits.  8 x 8 x 2 tiles
// with a halo instead of runs (40, 106 and 58 us) change the order of the sums: a
// weight whose gradient nearly cancels then takes another first Adam step.
// Bound: the serial chain of 128 steps of a warp, few warps where a level is small.
constexpr int WG_CHUNK = 2048, WG_SUB = 32, WG_BUFS = 3, WG_THREADS = 96;  // 2 buffers: 5% slower, 4: 48 x 16 60%

// v / n for 0 <= v < 2^31 and n <= 512: mul = ceil(2^40 / n)
__device__ __forceinline__ int divBy(int v, unsigned long long mul) {
    return (int)(((unsigned long long)(unsigned)v * mul) >> 40);
}

template <int MT, int NT>
__host__ __device__ constexpr int wgBufBytes() { return (WG_SUB + 2) * rowBytes<MT>() + WG_SUB * (16 * NT + 16); }
template <int MT, int NT>
__host__ __device__ constexpr int wgSmem() { return rowBytes<MT>() + 3 * WG_BUFS * wgBufBytes<MT, NT>(); }

template <int MT, int NT>
__global__ void __launch_bounds__(WG_THREADS) kWGrad(const Input in, const bf16* __restrict__ g,
                                                     float* __restrict__ part, int n, unsigned long long mul, int Cout) {
    constexpr int ROW = rowBytes<MT>(), GROW = 16 * NT + 16, Q = 2 * MT, BUF = wgBufBytes<MT, NT>();
    constexpr uint32_t gOff = (WG_SUB + 2) * ROW;
    extern __shared__ __align__(16) unsigned char wgSm[];
    const uint32_t sm = (uint32_t)__cvta_generic_to_shared(wgSm);
    const int tid = threadIdx.x, lane = tid & 31, dy = tid >> 5, dz = blockIdx.z, warp = 3 * dz + dy;
    const int Cin = in.Ca + in.Cb, coParts = Cout / (8 * NT);
    const int ci0 = (int)(blockIdx.y / coParts) * 16 * MT, co0 = (int)(blockIdx.y % coParts) * 8 * NT;
    const int V = n * n * n, vb = blockIdx.x * WG_CHUNK, ve = min(V, vb + WG_CHUNK), nh = n >> 1;
    for (int i = tid; i < ROW / 4; i += WG_THREADS) reinterpret_cast<uint32_t*>(wgSm)[i] = 0u;
    __syncthreads();
    const uint32_t mine = sm + ROW + dy * WG_BUFS * BUF;
    const int shift = n * (dy - 1) + n * n * (dz - 1) - 1;  // first voxel of the staged run, from the first of g
    // Pieces of 8 channels: `count` of them a voxel from channel c of a tensor with C channels, to
    // byte `at` of each row.  row(r, src): the tensor's row of run voxel r (src = its number on the grid).
    auto stagePieces = [&](auto count, uint32_t to, int first, const bf16* t, int C, int c, int at, auto row) {
        constexpr int P = decltype(count)::value, PER = 32 / P;
        const int r0 = lane / P, q = lane % P;
#pragma unroll
        for (int j = 0; j < (WG_SUB + 2 + PER - 1) / PER; ++j) {
            const int r = r0 + j * PER, src = first + r, tr = row(r, src);  // row() shuffles: all lanes
            if (r < WG_SUB + 2) {
                const bool ok = (unsigned)src < (unsigned)V;
                cpAsync16(to + r * ROW + at + 16 * q, ok ? t + (tr * (int64_t)C + c + 8 * q) : t, ok);
            }
        }
    };
    auto same = [](int, int src) { return src; };
    auto stage = [&](int v0, uint32_t to) {
        const int first = v0 + shift;
        if (ci0 < in.Ca) {
            // rows of the half-resolution tensor: one lane a voxel, two for lanes 0 and 1
            auto half = [&](int src) {
                const int yz = divBy(max(src, 0), mul), z = divBy(yz, mul), x = src - yz * n, y = yz - z * n;
                return ((z >> 1) * nh + (y >> 1)) * nh + (x >> 1);
            };
            const int h0 = half(first + lane), h1 = half(first + 32 + (lane & 1));
            auto up = [&](int r, int) {
                const int a0 = __shfl_sync(0xffffffffu, h0, r & 31), a1 = __shfl_sync(0xffffffffu, h1, r & 1);
                return r < 32 ? a0 : a1;
            };
            if constexpr (MT == 3) {
                stagePieces(std::integral_constant<int, 4>(), to, first, in.a, in.Ca, ci0, 0, up);
                stagePieces(std::integral_constant<int, 2>(), to, first, in.b, in.Cb, 0, 64, same);
            } else {
                stagePieces(std::integral_constant<int, Q == 6 ? 2 : Q>(), to, first, in.a, in.Ca, ci0, 0, up);
            }
        } else {
            stagePieces(std::integral_constant<int, Q == 6 ? 2 : Q>(), to, first, in.b, in.Cb, ci0 - in.Ca, 0, same);
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int r = lane / NT + j * (32 / NT), v = v0 + r;
            const bool ok = v < ve;
            cpAsync16(to + gOff + r * GROW + 16 * (lane % NT),
                      ok ? g + (v * (int64_t)Cout + co0 + 8 * (lane % NT)) : g, ok);
        }
        cpCommit();
    };
    float acc[3][MT][NT][4], accB[NT][4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            accB[j][e] = 0.f;
#pragma unroll
            for (int t = 0; t < 3; ++t)
#pragma unroll
                for (int m = 0; m < MT; ++m) acc[t][m][j][e] = 0.f;
        }
    const bool bias = warp == 4 && ci0 == 0;
    const int lv = (lane & 7) + 8 * (lane >> 4);  // this lane's voxel row of A in a step
    const uint32_t aHalf = 16 * ((lane >> 3) & 1), aZero = sm + aHalf;
    const uint32_t bLane = gOff + (uint32_t)(((lane & 7) + 8 * ((lane >> 3) & 1)) * GROW + 16 * (lane >> 4));
    // runs past the chunk's end are staged too (g as zeros, never used): a group per run keeps the count
#pragma unroll
    for (int i = 0; i < WG_BUFS - 1; ++i) stage(vb + i * WG_SUB, mine + i * BUF);
    uint32_t cur = 0, put = (WG_BUFS - 1) * BUF;
    int x, y, z;  // of this lane's voxel in the step
    {
        const int yz = divBy(vb + lv, mul);
        z = divBy(yz, mul);
        x = vb + lv - yz * n;
        y = yz - z * n;
    }
    for (int v0 = vb; v0 < ve; v0 += WG_SUB) {
        stage(v0 + (WG_BUFS - 1) * WG_SUB, mine + put);
        cpWait<WG_BUFS - 1>();
        __syncwarp();
        const uint32_t base = mine + cur;
        const int steps = (min(WG_SUB, ve - v0) + 15) >> 4;
#pragma unroll
        for (int k = 0; k < WG_SUB / 16; ++k) {
            if (k >= steps) break;
            uint32_t B[NT / 2][4];
#pragma unroll
            for (int j = 0; j < NT / 2; ++j) ldsm4t(B[j], base + bLane + k * 16 * GROW + 32 * j);
            const bool row = v0 + 16 * k + lv < ve && (unsigned)(y + dy - 1) < (unsigned)n && (unsigned)(z + dz - 1) < (unsigned)n;
            const uint32_t ak = base + (uint32_t)((16 * k + lv) * ROW) + aHalf;
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const uint32_t at = row && (unsigned)(x + t - 1) < (unsigned)n ? ak + t * ROW : aZero;
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    uint32_t A[4];
                    ldsm4t(A, at + 32 * m);
#pragma unroll
                    for (int j = 0; j < NT; ++j)
                        mma16816(acc[t][m][j], A[0], A[1], A[2], A[3], B[j >> 1][2 * (j & 1)], B[j >> 1][2 * (j & 1) + 1]);
                }
            }
            if (bias) {
                constexpr uint32_t one = 0x3f803f80u;
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    mma16816(accB[j], one, one, one, one, B[j >> 1][2 * (j & 1)], B[j >> 1][2 * (j & 1) + 1]);
            }
            for (x += 16; x >= n;) {
                x -= n;
                if (++y == n) {
                    y = 0;
                    ++z;
                }
            }
        }
        __syncwarp();  // every lane has read this buffer before a later stage fills it
        cur = cur + BUF == WG_BUFS * BUF ? 0 : cur + BUF;
        put = put + BUF == WG_BUFS * BUF ? 0 : put + BUF;
    }
    const int64_t per = 27LL * Cin * Cout + Cout;
    float* d = part + blockIdx.x * per;
    const int r = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int co = co0 + 8 * j + 2 * t4;
#pragma unroll
        for (int t = 0; t < 3; ++t)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<float2*>(d + ((int64_t)(3 * warp + t) * Cin + ci0 + 16 * m + r + 8 * h) * Cout + co) =
                        make_float2(acc[t][m][j][2 * h], acc[t][m][j][2 * h + 1]);
        if (bias && r == 0) *reinterpret_cast<float2*>(d + 27LL * Cin * Cout + co) = make_float2(accB[j][0], accB[j][1]);
    }
}

// dW[e] += sum over the slices of part, in order (16 loads in flight, then their additions).
__global__ void __launch_bounds__(64) kGradSum(const float* __restrict__ part, float* __restrict__ dW, int64_t per,
                                               int slices) {
    const int64_t e = blockIdx.x * 64LL + threadIdx.x;
    if (e >= per) return;
    float sum = 0.f;
    int c = 0;
    for (; c + 16 <= slices; c += 16) {
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = part[(int64_t)(c + q) * per + e];
#pragma unroll
        for (int q = 0; q < 16; ++q) sum += v[q];
    }
    for (; c < slices; ++c) sum += part[(int64_t)c * per + e];
    dW[e] += sum;
}

// ----------------------------------------------------------------------------- elementwise
// 8 channels (16 bytes) a thread forward, 4 backward.  Measured at 72^3 with 16
// channels: pooling 11 -> 5 us; the backward passes of a sample 213 -> 60 us: gradient
// sums, ReLU mask and BF16 rounding in one pass each instead of FP32 intermediates.
__device__ __forceinline__ void unpack8(const uint4& r, float (&v)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// out at n/2 = nc: mean of the 2x2x2 children.
__global__ void kPool(const bf16* __restrict__ in, bf16* __restrict__ out, int nc, int C) {
    const int Q = C / 8, total = nc * nc * nc * Q, nf = 2 * nc;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int q = i % Q, v = i / Q;
        const int x = v % nc, y = v / nc % nc, z = v / (nc * nc);
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            const int64_t f = ((int64_t)(2 * z + (d >> 2)) * nf + 2 * y + ((d >> 1) & 1)) * nf + 2 * x + (d & 1);
            float u[8];
            unpack8(*reinterpret_cast<const uint4*>(in + f * C + 8 * q), u);
#pragma unroll
            for (int c = 0; c < 8; ++c) s[c] += u[c];
        }
        *reinterpret_cast<uint4*>(out + (int64_t)v * C + 8 * q) =
            make_uint4(bf16x2(0.125f * s[0], 0.125f * s[1]), bf16x2(0.125f * s[2], 0.125f * s[3]),
                       bf16x2(0.125f * s[4], 0.125f * s[5]), bf16x2(0.125f * s[6], 0.125f * s[7]));
    }
}

// Gradient g through relu (y its output) as the BF16 operand of the backward GEMMs, 4 channels.
__device__ __forceinline__ void storeMasked4(bf16* out, int64_t i, const float (&g)[4], const bf16* y) {
    const uint2 r = *reinterpret_cast<const uint2*>(y + i);
    const float y0 = __uint_as_float(r.x << 16), y1 = __uint_as_float(r.x & 0xffff0000u);
    const float y2 = __uint_as_float(r.y << 16), y3 = __uint_as_float(r.y & 0xffff0000u);
    *reinterpret_cast<uint2*>(out + i) = make_uint2(bf16x2(y0 > 0.f ? g[0] : 0.f, y1 > 0.f ? g[1] : 0.f),
                                                    bf16x2(y2 > 0.f ? g[2] : 0.f, y3 > 0.f ? g[3] : 0.f));
}

// The upsampled part of a decoder input's gradient g ([.][C] at 2 nc): the sum of
// the 8 children's first Ca channels, through the relu of its source y ([.][Ca] at nc).
__global__ void kUpGrad(const float* __restrict__ g, const bf16* __restrict__ y, bf16* __restrict__ out, int nc, int Ca,
                        int C) {
    const int Q = Ca / 4, total = nc * nc * nc * Q, nf = 2 * nc;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int q = i % Q, v = i / Q;
        const int x = v % nc, yy = v / nc % nc, z = v / (nc * nc);
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            const int64_t f = ((int64_t)(2 * z + (d >> 2)) * nf + 2 * yy + ((d >> 1) & 1)) * nf + 2 * x + (d & 1);
            const float4 u = *reinterpret_cast<const float4*>(g + f * C + 4 * q);
            s[0] += u.x; s[1] += u.y; s[2] += u.z; s[3] += u.w;
        }
        storeMasked4(out, (int64_t)v * Ca + 4 * q, s, y);
    }
}

// The gradient of an encoder output y ([.][Cb] at 2 nc): the skip part of g
// (channels [Ca, Ca + Cb)) plus the pooling's, gp / 8 ([.][Cb] at nc), through y's relu.
__global__ void kSkipGrad(const float* __restrict__ g, const float* __restrict__ gp, const bf16* __restrict__ y,
                          bf16* __restrict__ out, int nc, int Ca, int Cb) {
    const int Q = Cb / 4, nf = 2 * nc, total = nf * nf * nf * Q, C = Ca + Cb;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int q = i % Q, v = i / Q;
        const int x = v % nf, yy = v / nf % nf, z = v / (nf * nf);
        const float4 u = *reinterpret_cast<const float4*>(g + (int64_t)v * C + Ca + 4 * q);
        const int64_t pv = ((int64_t)(z >> 1) * nc + (yy >> 1)) * nc + (x >> 1);
        const float4 w = *reinterpret_cast<const float4*>(gp + pv * Cb + 4 * q);
        // (the additions are kept apart from the products: no contraction into FMAs)
        const float s[4] = {__fadd_rn(u.x, __fmul_rn(0.125f, w.x)), __fadd_rn(u.y, __fmul_rn(0.125f, w.y)),
                            __fadd_rn(u.z, __fmul_rn(0.125f, w.z)), __fadd_rn(u.w, __fmul_rn(0.125f, w.w))};
        storeMasked4(out, (int64_t)v * Cb + 4 * q, s, y);
    }
}

// The loss's factor 1 / (3 sum of the mask) (one block, beside the previous sample's kernels).
__global__ void __launch_bounds__(1024) kMaskCount(const float* __restrict__ m, int64_t V, float* __restrict__ invCount) {
    __shared__ double s[1024];
    double acc = 0.0;
    for (int64_t v = 4 * (int64_t)threadIdx.x; v < V; v += 4096) {  // V is a multiple of 512
        const float4 q = *reinterpret_cast<const float4*>(m + v);
        acc += ((double)q.x + q.y) + ((double)q.z + q.w);
    }
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 512; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *invCount = s[0] > 0.0 ? (float)(1.0 / (3.0 * s[0])) : 0.f;
}

// Masked MSE of the prediction y: loss = sum m (y - t)^2 / count; its gradient as the BF16
// operand g (16 channels, 0 beyond 2).  Partial sums in part[blockIdx], invCount behind them.
constexpr int kLossBlocks = 1024;
__global__ void kMse(const float* __restrict__ y, const float* __restrict__ t, const float* __restrict__ m,
                     bf16* __restrict__ g, double* __restrict__ part, int64_t V, const float* __restrict__ inv) {
    __shared__ double s[256];
    const float invCount = *inv;
    double acc = 0.0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
        const float mv = m[v];
        float gr[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float d = y[v * 3 + c] - t[v * 3 + c];
            acc += (double)(mv * d * d);
            gr[c] = 2.f * mv * d * invCount;
        }
        uint4* o = reinterpret_cast<uint4*>(g + v * 16);
        o[0] = make_uint4(bf16x2(gr[0], gr[1]), bf16x2(gr[2], 0.f), 0u, 0u);
        o[1] = make_uint4(0u, 0u, 0u, 0u);
    }
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s[0];
        if (blockIdx.x == 0) part[kLossBlocks] = invCount;
    }
}

// y = x / by
__global__ void kDivide(const float* __restrict__ x, float* __restrict__ y, int64_t n, float by) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = x[i] / by;
}

__global__ void kAdam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                      int64_t n, float lr, float b1, float b2, float eps, float c1, float c2, float gscale) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i] * gscale;
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// Working BF16 weights from the FP32 master, layer blockIdx.y: W (as is) and
// Wt[26 - tap][co][ci] for the data gradient.
struct CastArgs {
    bf16 *wb[kLayers], *wt[kLayers];
    int64_t off[kLayers];
};
__global__ void kCastWeights(const float* __restrict__ params, const CastArgs a) {
    const int l = blockIdx.y, Cin = d_cin[l], Cout = d_cout[l], n = 27 * Cin * Cout;
    const float* w = params + a.off[l];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int co = i % Cout, ci = i / Cout % Cin, tap = i / (Cin * Cout);
        const bf16 b = __float2bfloat16(w[i]);
        a.wb[l][i] = b;
        a.wt[l][((26 - tap) * Cout + co) * Cin + ci] = b;
    }
}

// n a multiple of 8.
__global__ void kF32ToBf16(const float* __restrict__ x, bf16* __restrict__ y, int64_t n) {
    for (int64_t i = 8 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x); i < n; i += 8 * (int64_t)gridDim.x * blockDim.x) {
        const float4 a = *reinterpret_cast<const float4*>(x + i), b = *reinterpret_cast<const float4*>(x + i + 4);
        *reinterpret_cast<uint4*>(y + i) = make_uint4(bf16x2(a.x, a.y), bf16x2(a.z, a.w), bf16x2(b.x, b.y), bf16x2(b.z, b.w));
    }
}

inline int blocks(int64_t n) {
    int64_t b = (n + 255) / 256;
    return (int)(b > 4096 ? 4096 : (b < 1 ? 1 : b));
}

}  // namespace

// ----------------------------------------------------------------------------- network object
constexpr int kLossRing = 64;  // samples between two reads of their losses

struct vfem_net {
    int n = 0;  // finest grid size (multiple of 8)
    int64_t V[4] = {};
    cudaStream_t stream = nullptr;
    // parameters: per layer weights [27][Cin][Cout] then bias [Cout], packed FP32
    int64_t woff[kLayers] = {}, boff[kLayers] = {}, nparam = 0;
    float *w = nullptr, *gw = nullptr, *m = nullptr, *v = nullptr;
    bf16 *wb[kLayers] = {}, *wt[kLayers] = {};
    int64_t step = 0;
    // activations (bf16) and gradients (f32)
    bf16 *x = nullptr, *e[4] = {}, *p[4] = {}, *d[3] = {};
    float* y = nullptr;  // prediction [V][3]
    // a sample's host inputs on the device, twice: one is copied in while the other is trained on
    float *xin[2] = {}, *t[2] = {}, *mask[2] = {}, *inv = nullptr;
    cudaStream_t copyStream = nullptr;
    cudaEvent_t copied[2] = {}, consumed[2] = {};
    float *gp[4] = {}, *gc[3] = {};  // gradients of the pooled and the decoder inputs
    bf16* gm[2] = {};                // gradient operands: of the last layer, of the others (largest layer)
    float* wgPart = nullptr;  // per-block weight and bias gradients (largest layer)
    vfem::PinnedRing ring;  // for samples above kDirectMax
    double *part = nullptr, *hostPart = nullptr;  // loss sums of kLossRing samples; pinned copy
};

namespace {

vfem_status netFail(vfem_status s, const std::string& m) {
    g_netError = m;
    return s;
}

#define NCK(call)                                                                                    \
    do {                                                                                             \
        cudaError_t e_ = (call);                                                                     \
        if (e_ != cudaSuccess) return netFail(VFEM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Zeroed device allocation, complete on return (the memset runs on the legacy
// default stream, which the network's non-blocking stream does not wait for).
template <typename T>
cudaError_t nalloc(T** p, int64_t n) {
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * (size_t)(n > 0 ? n : 1));
    if (e != cudaSuccess) return e;
    e = cudaMemset(*p, 0, sizeof(T) * (size_t)(n > 0 ? n : 1));
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(cudaStreamLegacy);
}

// A kernel's set-up on each device it is launched on (a kernel's attributes belong to one
// device): make() on the first launch there, its result (not 0) afterwards.
struct PerDevice {
    std::atomic<int> value[64] = {};
    template <typename F>
    int get(F make) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return make();
        int v = value[dev].load(std::memory_order_acquire);
        if (!v) value[dev].store(v = make(), std::memory_order_release);
        return v;
    }
};

// One convolution at level lvl: (Cin, Cout) as the network has them, forward and data gradient.
// TZ: 8 x 8 x 4 tiles, or 8 x 8 x 2 where the halo is large (Cin >= 128) or the level
// has too few voxels to fill the GPU's 152 SMs with the taller ones.
template <int CK, int NT, int TG, int TZ, ConvOut OUT>
void launchConv(vfem_net* N, const Input& in, const bf16* W, const float* b, const bf16* act, void* out, int n, int Cout,
                int relu) {
    constexpr size_t smem = convSmem<CK, NT, TG, TZ>();
    static_assert(smem <= 227 * 1024, "tile too large");
    auto kern = kConv<CK, NT, TG, TZ, OUT>;
    static PerDevice blocksPerSm;
    const int perSm = blocksPerSm.get([&] {
        int k = 0;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, kern, 64 * TZ, smem);
        return std::max(1, k);
    });
    const int tx = (n + 7) / 8, tiles = tx * tx * ((n + TZ - 1) / TZ), parts = std::max(1, Cout / (8 * NT) / (OUT == OUT_PRED ? 2 : 1));
    const dim3 grid((unsigned)std::min(tiles, std::max(1, 152 * perSm / parts)), (unsigned)parts);
    kern<<<grid, 64 * TZ, smem, N->stream>>>(in, W, b, act, out, n, Cout, relu);
}

template <ConvOut OUT>
void conv(vfem_net* N, const Input& in, const bf16* W, const float* b, const bf16* act, void* out, int lvl, int Cout,
          int relu) {
    const int n = N->n >> lvl, Cin = in.Ca + in.Cb;
    const bool low = (int64_t)n * n * n < 152 * 256;  // fewer tall tiles than SMs
#define CONV_CASE(ci, co, nt, tg, tz)                                                                  \
    if (Cin == ci && Cout == co) {                                                                     \
        if (low) return launchConv<ci / 16, nt, tg, 2, OUT>(N, in, W, b, act, out, n, Cout, relu);     \
        return launchConv<ci / 16, nt, tg, tz, OUT>(N, in, W, b, act, out, n, Cout, relu);            \
    }
    if constexpr (OUT == OUT_BF16) {
        CONV_CASE(16, 32, 4, 27, 4)
        CONV_CASE(32, 64, 8, 3, 4)
        CONV_CASE(64, 128, 8, 1, 4)
        CONV_CASE(192, 64, 8, 1, 2)
        CONV_CASE(96, 32, 4, 1, 4)
        CONV_CASE(48, 16, 2, 3, 4)
    } else if constexpr (OUT == OUT_F32) {
        CONV_CASE(16, 48, 6, 27, 4)
        CONV_CASE(32, 96, 6, 3, 4)
        CONV_CASE(64, 192, 8, 1, 4)
        CONV_CASE(128, 64, 8, 1, 2)
        CONV_CASE(64, 32, 4, 1, 4)
        CONV_CASE(32, 16, 2, 27, 4)
    }
    if constexpr (OUT == OUT_PRED) {
        CONV_CASE(16, 16, 1, 27, 4)
    } else {
        CONV_CASE(16, 16, 2, 27, 4)
    }
#undef CONV_CASE
}

// BF16 working weights of the current master weights (after set_params and every Adam step).
void castWeights(vfem_net* N) {
    CastArgs a;
    for (int l = 0; l < kLayers; ++l) {
        a.wb[l] = N->wb[l];
        a.wt[l] = N->wt[l];
        a.off[l] = N->woff[l];
    }
    kCastWeights<<<dim3(152, kLayers), 256, 0, N->stream>>>(N->w, a);
}

// The input of convolution l.
Input layerInput(const vfem_net* N, int l) {
    switch (l) {
        case 0: return {nullptr, N->x, 0, 16};
        case 1: case 2: case 3: return {nullptr, N->p[l], 0, kCin[l]};
        case 4: return {N->e[3], N->e[2], 128, 64};
        case 5: return {N->d[2], N->e[1], 64, 32};
        case 6: return {N->d[1], N->e[0], 32, 16};
        default: return {nullptr, N->d[0], 0, 16};
    }
}

void forward(vfem_net* N) {
    const int64_t* V = N->V;
    auto layer = [&](int l, bf16* out) {
        conv<OUT_BF16>(N, layerInput(N, l), N->wb[l], N->w + N->boff[l], nullptr, out, kLevel[l], kCout[l], 1);
    };
    layer(0, N->e[0]);
    kPool<<<blocks(V[1] * 2), 256, 0, N->stream>>>(N->e[0], N->p[1], N->n / 2, 16);
    layer(1, N->e[1]);
    kPool<<<blocks(V[2] * 4), 256, 0, N->stream>>>(N->e[1], N->p[2], N->n / 4, 32);
    layer(2, N->e[2]);
    kPool<<<blocks(V[3] * 8), 256, 0, N->stream>>>(N->e[2], N->p[3], N->n / 8, 64);
    layer(3, N->e[3]);
    layer(4, N->d[2]);
    layer(5, N->d[1]);
    layer(6, N->d[0]);
    conv<OUT_PRED>(N, layerInput(N, 7), N->wb[7], N->w + N->boff[7], nullptr, N->y, 0, 16, 0);
}

int wgChunks(int64_t V) { return (int)((V + WG_CHUNK - 1) / WG_CHUNK); }

template <int MT, int NT>
void launchWGrad(vfem_net* N, const Input& in, const bf16* g, int n, int Cout, int chunks) {
    static PerDevice ready;
    ready.get([] {
        cudaFuncSetAttribute(kWGrad<MT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, wgSmem<MT, NT>());
        return 1;
    });
    const dim3 grid((unsigned)chunks, (unsigned)((in.Ca + in.Cb) / (16 * MT) * (Cout / (8 * NT))), 3);
    const unsigned long long mul = ((1ull << 40) + n - 1) / n;
    kWGrad<MT, NT><<<grid, WG_THREADS, wgSmem<MT, NT>(), N->stream>>>(in, g, N->wgPart, n, mul, Cout);
}

// Weight and bias gradient of convolution l, accumulated, from g = dL/d(its sums) (BF16).
void weightGrad(vfem_net* N, int l, const bf16* g) {
    const int Cin = kCin[l], Cout = kCout[l], n = N->n >> kLevel[l];
    const int64_t per = 27LL * Cin * Cout + Cout;
    // (ci, co) of a block: large ones read each operand least often; few chunks (V below
    // 16 x 2,048 at the coarse levels) take small ones, to have blocks for the 152 SMs
    const int chunks = wgChunks(N->V[kLevel[l]]);
    const Input in = layerInput(N, l);
    if (Cin == 48) launchWGrad<3, 2>(N, in, g, n, Cout, chunks);
    else if (Cout == 16) launchWGrad<1, 2>(N, in, g, n, Cout, chunks);
    else if (Cin == 16 || chunks < 16) launchWGrad<1, 4>(N, in, g, n, Cout, chunks);
    else launchWGrad<2, 4>(N, in, g, n, Cout, chunks);
    kGradSum<<<(unsigned)((per + 63) / 64), 64, 0, N->stream>>>(N->wgPart, N->gw + N->woff[l], per, chunks);
}

// dL/d(input) of convolution l from g.
void dataGrad(vfem_net* N, int l, const bf16* g, float* gin) {
    conv<OUT_F32>(N, Input{nullptr, g, 0, kCout[l]}, N->wt[l], nullptr, nullptr, gin, kLevel[l], kCin[l], 0);
}

// From gm[0] = dL/dy (kMse).  gm[1] holds the operand of every other layer in turn.
void backward(vfem_net* N) {
    const int64_t* V = N->V;
    bf16* g = N->gm[1];
    weightGrad(N, 7, N->gm[0]);
    conv<OUT_MASKED>(N, Input{nullptr, N->gm[0], 0, 16}, N->wt[7], nullptr, N->d[0], g, 0, 16, 0);
    // decoder: layer 6 - l reads [up(upper source), e[l]]
    const bf16* src[3] = {N->d[1], N->d[2], N->e[3]};
    const int up[3] = {32, 64, 128}, skip[3] = {16, 32, 64};
    for (int l = 0; l < 3; ++l) {
        weightGrad(N, 6 - l, g);
        dataGrad(N, 6 - l, g, N->gc[l]);
        kUpGrad<<<blocks(V[l + 1] * up[l] / 4), 256, 0, N->stream>>>(N->gc[l], src[l], g, N->n >> (l + 1), up[l],
                                                                      up[l] + skip[l]);
    }
    // encoder: layer l reads pool(e[l - 1])
    for (int l = 3; l > 0; --l) {
        weightGrad(N, l, g);
        dataGrad(N, l, g, N->gp[l]);
        kSkipGrad<<<blocks(V[l - 1] * skip[l - 1] / 4), 256, 0, N->stream>>>(N->gc[l - 1], N->gp[l], N->e[l - 1], g,
                                                                              N->n >> l, up[l - 1], skip[l - 1]);
    }
    weightGrad(N, 0, g);
}

}  // namespace

extern "C" {

const char* vfem_net_last_error_message(void) { return g_netError.c_str(); }

vfem_status vfem_net_create(int32_t n, vfem_net** out) {
    if (!out || n < 8 || n % 8 != 0 || n > 512) return netFail(VFEM_ERR_INVALID_ARGUMENT, "grid size must be a multiple of 8 in [8, 512]");
    *out = nullptr;
    vfem_net* N = new vfem_net();
    N->n = n;
    for (int l = 0; l < 4; ++l) N->V[l] = (int64_t)(n >> l) * (n >> l) * (n >> l);
    int64_t off = 0;
    for (int l = 0; l < kLayers; ++l) {
        N->woff[l] = off;
        off += 27LL * kCin[l] * kCout[l];
        N->boff[l] = off;
        off += kCout[l];
    }
    N->nparam = off;
    auto bail = [&](cudaError_t e) {
        vfem_net_destroy(N);
        return netFail(VFEM_ERR_CUDA, std::string("allocation: ") + cudaGetErrorString(e));
    };
#define NA(call)                    \
    do {                            \
        cudaError_t e_ = (call);    \
        if (e_ != cudaSuccess) return bail(e_); \
    } while (0)
    NA(cudaStreamCreateWithFlags(&N->stream, cudaStreamNonBlocking));
    NA(nalloc(&N->w, off)); NA(nalloc(&N->gw, off)); NA(nalloc(&N->m, off)); NA(nalloc(&N->v, off));
    for (int l = 0; l < kLayers; ++l) {
        NA(nalloc(&N->wb[l], 27LL * kCin[l] * kCout[l]));
        NA(nalloc(&N->wt[l], 27LL * kCin[l] * kCout[l]));
    }
    const int64_t* V = N->V;
    NA(nalloc(&N->x, V[0] * 16));
    const int ec[4] = {16, 32, 64, 128};
    for (int l = 0; l < 4; ++l) {
        NA(nalloc(&N->e[l], V[l] * ec[l]));
    }
    const int pc[4] = {0, 16, 32, 64};
    for (int l = 1; l < 4; ++l) {
        NA(nalloc(&N->p[l], V[l] * pc[l]));
        NA(nalloc(&N->gp[l], V[l] * pc[l]));
    }
    const int cc[3] = {48, 96, 192}, dc[3] = {16, 32, 64};
    for (int l = 0; l < 3; ++l) {
        NA(nalloc(&N->gc[l], V[l] * cc[l]));
        NA(nalloc(&N->d[l], V[l] * dc[l]));
    }
    NA(nalloc(&N->y, V[0] * 3));
    for (int i = 0; i < 2; ++i) {
        NA(nalloc(&N->xin[i], V[0] * 16));
        NA(nalloc(&N->t[i], V[0] * 3));
        NA(nalloc(&N->mask[i], V[0]));
        NA(cudaEventCreateWithFlags(&N->copied[i], cudaEventDisableTiming));
        NA(cudaEventCreateWithFlags(&N->consumed[i], cudaEventDisableTiming));
    }
    NA(nalloc(&N->inv, 2));
    NA(cudaStreamCreateWithFlags(&N->copyStream, cudaStreamNonBlocking));
    int64_t gmax = 0;
    for (int l = 0; l < kLayers; ++l) gmax = std::max<int64_t>(gmax, V[kLevel[l]] * kCout[l]);
    NA(nalloc(&N->gm[0], V[0] * 16));
    NA(nalloc(&N->gm[1], gmax));
    int64_t wmax = 0;
    for (int l = 0; l < kLayers; ++l)
        wmax = std::max<int64_t>(wmax, wgChunks(V[kLevel[l]]) * (27LL * kCin[l] * kCout[l] + kCout[l]));
    NA(nalloc(&N->wgPart, std::max(wmax, off)));  // also the batch mean on its way to the caller
    NA(nalloc(&N->part, kLossRing * (kLossBlocks + 1)));
    NA(cudaMallocHost((void**)&N->hostPart, sizeof(double) * kLossRing * (kLossBlocks + 1)));
#undef NA
    *out = N;
    return VFEM_OK;
}

void vfem_net_destroy(vfem_net* N) {
    if (!N) return;
    cudaFree(N->w); cudaFree(N->gw); cudaFree(N->m); cudaFree(N->v);
    for (int l = 0; l < kLayers; ++l) { cudaFree(N->wb[l]); cudaFree(N->wt[l]); }
    cudaFree(N->x);
    for (int l = 0; l < 4; ++l) { cudaFree(N->e[l]); cudaFree(N->p[l]); cudaFree(N->gp[l]); }
    for (int l = 0; l < 3; ++l) { cudaFree(N->gc[l]); cudaFree(N->d[l]); }
    cudaFree(N->y); cudaFree(N->inv); cudaFree(N->gm[0]); cudaFree(N->gm[1]);
    for (int i = 0; i < 2; ++i) {
        cudaFree(N->xin[i]); cudaFree(N->t[i]); cudaFree(N->mask[i]);
        if (N->copied[i]) cudaEventDestroy(N->copied[i]);
        if (N->consumed[i]) cudaEventDestroy(N->consumed[i]);
    }
    cudaFree(N->part); cudaFree(N->wgPart);
    if (N->hostPart) cudaFreeHost(N->hostPart);
    if (N->copyStream) cudaStreamDestroy(N->copyStream);
    if (N->stream) cudaStreamDestroy(N->stream);
    delete N;
}

int64_t vfem_net_num_params(const vfem_net* N) { return N ? N->nparam : 0; }

vfem_status vfem_net_set_params(vfem_net* N, const float* params) {
    if (!N || !params) return netFail(VFEM_ERR_INVALID_ARGUMENT, "null argument");
    NCK(cudaMemcpyAsync(N->w, params, sizeof(float) * N->nparam, cudaMemcpyHostToDevice, N->stream));
    NCK(cudaMemsetAsync(N->m, 0, sizeof(float) * N->nparam, N->stream));
    NCK(cudaMemsetAsync(N->v, 0, sizeof(float) * N->nparam, N->stream));
    castWeights(N);
    N->step = 0;
    NCK(cudaStreamSynchronize(N->stream));
    return VFEM_OK;
}

vfem_status vfem_net_get_params(vfem_net* N, float* params) {
    if (!N || !params) return netFail(VFEM_ERR_INVALID_ARGUMENT, "null argument");
    NCK(vfem::copyToHost(N->ring, params, N->w, sizeof(float) * N->nparam, N->stream));
    return VFEM_OK;
}

// input: [n^3][16] FP32 features (channels beyond the used ones zero); output [n^3][3].
vfem_status vfem_net_forward(vfem_net* N, const float* input, float* output) {
    if (!N || !input || !output) return netFail(VFEM_ERR_INVALID_ARGUMENT, "null argument");
    const int64_t V = N->V[0];
    NCK(vfem::copyToDevice(N->ring, N->xin[0], input, sizeof(float) * V * 16, N->stream));
    kF32ToBf16<<<blocks(V * 2), 256, 0, N->stream>>>(N->xin[0], N->x, V * 16);
    forward(N);
    NCK(cudaGetLastError());
    NCK(vfem::copyToHost(N->ring, output, N->y, sizeof(float) * V * 3, N->stream));
    return VFEM_OK;
}

// Forward + backward of a batch of `batch` samples; gradients (summed over the
// batch, divided by it) to grads (host, nparam) if given, Adam step with lr if
// lr > 0.  loss_out: mean masked MSE.  Sample b + 1 is copied to the device while
// sample b is trained on; nothing waits for the host until the batch is through.
vfem_status vfem_net_train_batch(vfem_net* N, const float* inputs, const float* targets, const float* masks,
                                 int32_t batch, float lr, float* grads, float* loss_out) {
    if (!N || !inputs || !targets || !masks || batch < 1) return netFail(VFEM_ERR_INVALID_ARGUMENT, "bad argument");
    const int64_t V = N->V[0];
    NCK(cudaMemsetAsync(N->gw, 0, sizeof(float) * N->nparam, N->stream));
    double lossSum = 0.0;
    auto copyIn = [&](int b) -> cudaError_t {
        const int i = b & 1;
        cudaError_t e;
        if (b >= 2 && (e = cudaStreamWaitEvent(N->copyStream, N->consumed[i], 0)) != cudaSuccess) return e;
        auto in = [&](float* dst, const float* src, int64_t per) {
            return vfem::copyToDevice(N->ring, dst, src + b * V * per, sizeof(float) * V * per, N->copyStream);
        };
        if ((e = in(N->xin[i], inputs, 16)) || (e = in(N->t[i], targets, 3)) || (e = in(N->mask[i], masks, 1))) return e;
        kMaskCount<<<1, 1024, 0, N->copyStream>>>(N->mask[i], V, N->inv + i);
        return cudaEventRecord(N->copied[i], N->copyStream);
    };
    NCK(copyIn(0));
    for (int b = 0; b < batch; ++b) {
        const int i = b & 1, slot = b % kLossRing;
        double* part = N->part + slot * (kLossBlocks + 1);
        NCK(cudaStreamWaitEvent(N->stream, N->copied[i], 0));
        kF32ToBf16<<<blocks(V * 2), 256, 0, N->stream>>>(N->xin[i], N->x, V * 16);
        forward(N);
        kMse<<<kLossBlocks, 256, 0, N->stream>>>(N->y, N->t[i], N->mask[i], N->gm[0], part, V, N->inv + i);
        NCK(cudaEventRecord(N->consumed[i], N->stream));
        backward(N);
        if (b + 1 < batch) NCK(copyIn(b + 1));
        if (b + 1 == batch || slot + 1 == kLossRing) {
            NCK(cudaMemcpyAsync(N->hostPart, N->part, sizeof(double) * (slot + 1) * (kLossBlocks + 1),
                                cudaMemcpyDeviceToHost, N->stream));
            NCK(cudaStreamSynchronize(N->stream));
            for (int q = 0; q <= slot; ++q) {
                const double* h = N->hostPart + q * (kLossBlocks + 1);
                double s = 0.0;
                for (int k = 0; k < kLossBlocks; ++k) s += h[k];
                lossSum += s * (float)h[kLossBlocks];
            }
        }
    }
    NCK(cudaGetLastError());
    if (loss_out) *loss_out = (float)(lossSum / batch);
    if (grads) {
        kDivide<<<blocks(N->nparam), 256, 0, N->stream>>>(N->gw, N->wgPart, N->nparam, (float)batch);
        NCK(vfem::copyToHost(N->ring, grads, N->wgPart, sizeof(float) * N->nparam, N->stream));
    }
    if (lr > 0.f) {
        N->step++;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - std::pow(b1, (float)N->step), c2 = 1.f - std::pow(b2, (float)N->step);
        kAdam<<<blocks(N->nparam), 256, 0, N->stream>>>(N->w, N->gw, N->m, N->v, N->nparam, lr, b1, b2, 1e-8f, c1, c2,
                                                        1.f / (float)batch);
        castWeights(N);
        NCK(cudaGetLastError());
        NCK(cudaStreamSynchronize(N->stream));
    }
    return VFEM_OK;
}

}  // extern "C"
