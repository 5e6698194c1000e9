// tw_eval.cu -- TPS evaluation at the coarse control-grid nodes (FP32,
// compensated landmark sums) on sm_100a.
//
// Reference: get_cd (weiyijisuan.cu:91-114) keeps a float xmxn_K1[20000]
// per thread (80 KB of local memory) and launches once per z plane; the CPU
// loops are q_imgwarp_tps_quicksmallmemory.cpp:620-648 and :1117-1146.
//
// Here one launch covers the whole grid.  Landmarks (negated centres and
// coefficients) are staged through shared memory in tiles and read as
// warp-wide broadcasts; a thread evaluates 2 or 4 nodes of one (x, y) column, so
// dx^2 + dy^2 is computed once per landmark for all of them.  Per landmark and
// two nodes what is left is one add, one multiply-add, two square roots and
// three multiply-adds, the node pairs in FP32x2 instructions.  (Grids a few
// nodes deep: nodes of one row, see eval_form.)  What bounds it:
// the square roots, 16 per SM and clock (1.15 M nodes x 2000 landmarks: 0.51
// ms of them; the call takes 648 us, 826 when each node had its own dx and dy
// and the landmarks' components were staged twice over: a broadcast of 16
// bytes to a warp takes 4 cycles of the shared memory's return path, and three
// of them per landmark and four nodes were more than the square roots).  Sums
// are two-level: plain FP32 FMA chains over 32 landmarks, then
// Kahan-compensated accumulation of those partials.
//
// Coordinates are taken relative to an origin o near the landmarks so the
// FP32 magnitudes stay small; the affine part is folded (in FP64, on the
// device) into a0 + alin * p' with the identity already subtracted, so the
// kernel writes the displacement f(p) - p directly without cancelling two
// large numbers.

#include "tw_internal.h"

namespace tw {

namespace {

constexpr int kEvalThreads = 256;
constexpr int kTile = 256;   // landmarks staged per shared-memory tile
constexpr int kSub = 32;     // landmarks per plain FP32 partial sum

__device__ __forceinline__ float fast_sqrt(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void kahan_add(float &s, float &c, float x)
{
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

// NPT: nodes per thread, consecutive along axis AX (z, or x).  SPLIT: groups of threads that
// share the 32-landmark partial sums of the same nodes out among themselves,
// turn by turn; the partials then meet in shared memory and are added in
// landmark order, so the sums are the same whatever the split.
template <int NPT, int SPLIT, int AX>
__global__ void __launch_bounds__(kEvalThreads) k_tps_eval(EvalParams p)
{
    static_assert(AX == 0 || AX == 2, "runs along x or z");
    constexpr int UNITS = kEvalThreads / SPLIT, P2 = NPT / 2;
    static_assert(kTile / kSub == 8 && 8 % SPLIT == 0 && UNITS % 32 == 0, "whole warps, whole turns");
    __shared__ float4 s_a[kTile];  // -cx, -cy, -cz, wx
    __shared__ float2 s_b[kTile];  // wy, wz
    __shared__ float s_part[SPLIT > 1 ? SPLIT : 1][3 * NPT][SPLIT > 1 ? UNITS : 1];
    const int unit = threadIdx.x % UNITS, grp = threadIdx.x / UNITS;
    const int64_t U = (int64_t)blockIdx.x * UNITS + unit;
    // units: x (or runs of NPT columns) fastest, then y, then z (or runs of NPT
    // planes); past the end: some node again, not stored
    const int64_t nx = AX == 0 ? (p.gsz[0] + NPT - 1) / NPT : p.gsz[0];
    const int64_t ix = U % nx * (AX == 0 ? NPT : 1), iy = U / nx % p.gsz[1];
    const int64_t iz = U / (nx * p.gsz[1]) * (AX == 2 ? NPT : 1);
    const auto coord = [&](int a, int64_t i) { return (float)(p.node_o[a] + min(i, p.gsz[a] - 1) * p.g); };
    const float px = coord(0, ix), py = coord(1, iy), pz = coord(2, iz);
    float pr[NPT];  // along the run
    float s[3][NPT], c[3][NPT];
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
        pr[j] = coord(AX, (AX == 0 ? ix : iz) + j);
#pragma unroll
        for (int q = 0; q < 3; ++q) s[q][j] = c[q][j] = 0.f;
    }

    for (int t0 = 0; t0 < p.n; t0 += kTile) {
        const int cnt = min(kTile, p.n - t0);
        __syncthreads();
        for (int l = threadIdx.x; l < kTile; l += kEvalThreads) {
            float4 e = make_float4(0.f, 0.f, 0.f, 0.f), w = e;  // zero weight pads the tile
            if (l < cnt) {
                e = p.ctr[t0 + l];
                w = p.coef[t0 + l];
            }
            s_a[l] = make_float4(-e.x, -e.y, -e.z, w.x);
            s_b[l] = make_float2(w.y, w.z);
        }
        __syncthreads();
        const int nsub = (cnt + kSub - 1) / kSub;
        for (int sb0 = 0; sb0 < nsub; sb0 += SPLIT) {
            const int sb = sb0 + grp;
            // two nodes per instruction: the same operations, in the same
            // order, as one FP32 instruction per node and landmark
            float2 a[3][P2];
#pragma unroll
            for (int k = 0; k < P2; ++k) a[0][k] = a[1][k] = a[2][k] = make_float2(0.f, 0.f);
            if (SPLIT == 1 || sb < nsub) {
#pragma unroll 4
                for (int l = sb * kSub; l < sb * kSub + kSub; ++l) {
                    const float4 A = s_a[l];
                    const float2 B = s_b[l];
                    // dx^2 + dy^2 + dz^2, added in this order whatever the run
                    const float dy = __fadd_rn(py, A.y);
                    float2 r02, dy2, dz2;
                    if (AX == 2) {
                        const float dx = __fadd_rn(px, A.x), r0 = __fmaf_rn(dy, dy, __fmul_rn(dx, dx));
                        r02 = make_float2(r0, r0);
                    } else {
                        const float dz = __fadd_rn(pz, A.z);
                        dy2 = make_float2(dy, dy);
                        dz2 = make_float2(dz, dz);
                    }
                    const float nc = AX == 0 ? A.x : A.z;
                    const float2 wx = make_float2(A.w, A.w), wy = make_float2(B.x, B.x), wz = make_float2(B.y, B.y);
#pragma unroll
                    for (int k = 0; k < P2; ++k) {
                        const float2 dr = __fadd2_rn(make_float2(pr[2 * k], pr[2 * k + 1]), make_float2(nc, nc));
                        const float2 r2 = AX == 2 ? __ffma2_rn(dr, dr, r02)
                                                  : __ffma2_rn(dz2, dz2, __ffma2_rn(dy2, dy2, __fmul2_rn(dr, dr)));
                        const float2 r = make_float2(fast_sqrt(r2.x), fast_sqrt(r2.y));
                        a[0][k] = __ffma2_rn(r, wx, a[0][k]);
                        a[1][k] = __ffma2_rn(r, wy, a[1][k]);
                        a[2][k] = __ffma2_rn(r, wz, a[2][k]);
                    }
                }
            }
            if constexpr (SPLIT == 1) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int j = 0; j < NPT; ++j) kahan_add(s[q][j], c[q][j], (j & 1) ? a[q][j >> 1].y : a[q][j >> 1].x);
            } else {
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int j = 0; j < NPT; ++j) s_part[grp][q * NPT + j][unit] = (j & 1) ? a[q][j >> 1].y : a[q][j >> 1].x;
                __syncthreads();
                // sum e of a unit belongs to group e % SPLIT
                const int have = min(SPLIT, nsub - sb0);
#pragma unroll
                for (int e = 0; e < 3 * NPT; e += SPLIT)
                    if (e + grp < 3 * NPT)
                        for (int k = 0; k < have; ++k)
                            kahan_add(s[0][e / SPLIT], c[0][e / SPLIT], s_part[k][e + grp][unit]);
                __syncthreads();
            }
        }
    }
    if constexpr (SPLIT > 1) {  // the sums, less their compensation, to group 0
        static_assert(3 * NPT <= SPLIT * NPT, "a group's sums fit in s[0]");
#pragma unroll
        for (int e = 0; e < 3 * NPT; e += SPLIT)
            if (e + grp < 3 * NPT) s_part[0][e + grp][unit] = s[0][e / SPLIT] - c[0][e / SPLIT];
        __syncthreads();
        if (grp != 0) return;
    }

    // affine part: f_c(q) = d[0][c] + sum_r q_r d[r+1][c]; with q = o + p:
    // DF_c = (d[0][c] + o.d[1:4][c] - o_c) + sum_r p_r (d[r+1][c] - delta),
    // folded in FP64 without contraction, then rounded once to float
    float a0[3], alin[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double s = __ldg(&p.aff[c + 1]);
#pragma unroll
        for (int r = 0; r < 3; ++r) s = __dadd_rn(s, __dmul_rn(p.o[r], __ldg(&p.aff[(r + 1) * 4 + c + 1])));
        a0[c] = (float)__dsub_rn(s, p.o[c]);
#pragma unroll
        for (int r = 0; r < 3; ++r) alin[r][c] = (float)__dsub_rn(__ldg(&p.aff[(r + 1) * 4 + c + 1]), r == c ? 1.0 : 0.0);
    }
#pragma unroll
    for (int j = 0; j < NPT; ++j) {
        const int64_t i = AX == 0 ? ix + j : ix, k = AX == 2 ? iz + j : iz;
        if (i >= p.gsz[0] || k >= p.gsz[2]) break;
        const float x = AX == 0 ? pr[j] : px, z = AX == 2 ? pr[j] : pz;
        float dfx = __fmaf_rn(alin[2][0], z, __fmaf_rn(alin[1][0], py, __fmaf_rn(alin[0][0], x, a0[0])));
        float dfy = __fmaf_rn(alin[2][1], z, __fmaf_rn(alin[1][1], py, __fmaf_rn(alin[0][1], x, a0[1])));
        float dfz = __fmaf_rn(alin[2][2], z, __fmaf_rn(alin[1][2], py, __fmaf_rn(alin[0][2], x, a0[2])));
        // the running compensation holds minus the lost low-order part
        if constexpr (SPLIT > 1) {
            dfx += s_part[0][j][unit];
            dfy += s_part[0][NPT + j][unit];
            dfz += s_part[0][2 * NPT + j][unit];
        } else {
            dfx += s[0][j] - c[0][j];
            dfy += s[1][j] - c[1][j];
            dfz += s[2][j] - c[2][j];
        }
        p.out[(k * p.gsz[1] + iy) * p.gsz[0] + i] = make_float4(dfx, dfy, dfz, 0.f);
    }
}

template <int NPT, int SPLIT, int AX>
cudaError_t launch_eval_along(const EvalParams &p, cudaStream_t st)
{
    int64_t n[3] = {p.gsz[0], p.gsz[1], p.gsz[2]};
    n[AX] = (n[AX] + NPT - 1) / NPT;
    const int64_t per = kEvalThreads / SPLIT, grid = (n[0] * n[1] * n[2] + per - 1) / per;
    if (grid > 0x7fffffff) return cudaErrorInvalidValue;
    k_tps_eval<NPT, SPLIT, AX><<<(unsigned)grid, kEvalThreads, 0, st>>>(p);
    return cudaGetLastError();
}

template <int NPT, int SPLIT>
cudaError_t launch_eval(const EvalParams &p, cudaStream_t st, int axis)
{
    return axis == 0 ? launch_eval_along<NPT, SPLIT, 0>(p, st) : launch_eval_along<NPT, SPLIT, 2>(p, st);
}

}  // namespace

EvalForm eval_form(const int64_t gsz[3], int n, int sm_count)
{
    const int64_t nnodes = gsz[0] * gsz[1] * gsz[2];
    EvalForm f;
    // A grid that fills the chip runs one thread per four nodes.  Smaller ones
    // share the landmarks of 32-node units out over a block's eight warps, if
    // there are enough of them (calls with 2000 landmarks: 847 nodes 129 us
    // unsplit, 49 split, 23,000 129 and 58 with two nodes a thread, 61 with
    // four; 157,000 201, 150 and 134; 1.15 M 649, 793 and 677; 292,000 227, -
    // and 211, but with 300 landmarks 55, - and 58).
    if (nnodes >= (int64_t)sm_count * (n > 512 ? 2048 : 1792)) f = {4, 1, 2};
    else if (nnodes >= (int64_t)sm_count * 256) f = {4, n > 128 ? 8 : 1, 2};
    else f = {2, 8, 2};
    // The nodes of a thread lie along z, unless rounding the grid's depth up to
    // whole runs costs clearly more than rounding its width up (2000 landmarks,
    // us along z and along x: 515 x 515 x 1 607 and 198, x 3 632 and 521, x 5
    // 1151 and 766, 259 x 259 x 9 481 and 361; a run along x has two more
    // instructions per pair: 131 x 131 x 67 634 and 716)
    const auto rounded = [&](int a) { return (double)((gsz[a] + f.npt - 1) / f.npt * f.npt) / (double)gsz[a]; };
    if (rounded(2) > 1.1 * rounded(0)) f.axis = 0;
    return f;
}

cudaError_t launch_tps_eval(const EvalParams &p, cudaStream_t st, int sm_count)
{
    if (p.gsz[0] * p.gsz[1] * p.gsz[2] <= 0) return cudaSuccess;
    const EvalForm f = eval_form(p.gsz, p.n, sm_count);
    if (f.npt == 2) return launch_eval<2, 8>(p, st, f.axis);
    return f.split == 8 ? launch_eval<4, 8>(p, st, f.axis) : launch_eval<4, 1>(p, st, f.axis);
}

}  // namespace tw
