// tw_solve.cu -- FP64 landmark solves on sm_100a: the regularised TPS system
// and the 3-D affine DLT fit.
//
// TPS (reference: compute_df_stps_subsampled_volume_4bspline,
// q_imgwarp_tps_quicksmallmemory.cpp:377-588, whose GPU branch runs cuSOLVER
// Sgeqrf on an N x N zero-padded copy of X (qr.cu:8-130), N-4 host round trips
// of Gram-Schmidt (extendornormal.cu:55-150), four cublasSgemm calls with a
// handle created per call (aff.cu:37-133) and an unpivoted FP32 Gauss-Jordan
// inverse with 3(N-4) launches (GET_A_i.cu:80-161), all in FP32):
//
//   c = q2 (q2' K q2 + lambda I)^-1 q2' Y,   d = r^-1 q1' (Y - K c)
//
// is computed here entirely in FP64 without ever forming K, Q or A^-1:
//   1. Householder QR of X = [1 s] (n x 4): 4 reflectors H_k = I - tau v v'.
//      Q = H1 H2 H3 H4; q1 = Q(:,0:4), q2 = Q(:,4:n).  c and d do not depend
//      on which orthonormal basis q2 is (the reference completes q1 by
//      Gram-Schmidt instead), only on span(q2) = span(X)^perp.
//   2. Q' K Q by four symmetric rank-2 updates: H K H = K - v w' - w v' with
//      w = tau p - (tau^2 v'p / 2) v, p = K v.  All four p come from one
//      product P0 = K V over the implicit K_ij = -|s_i - s_j|.
//   3. A = (Q' K Q)(4:,4:) + lambda I is symmetric positive definite (-|r| is
//      conditionally positive definite of order 1 in 3-D and q2 is orthogonal
//      to the polynomials), so it is factored by a blocked Cholesky in
//      64 x 64 FP64 tiles (tw_chol.cu).
//   4. z = Q' Y; w = A^-1 z(4:): the forward substitution rides along in the
//      factorisation (z(4:)' is an extra row block of the panel solves and
//      trailing updates), the back substitution follows in the same kernel;
//      c = Q [0; w]; d = R^-1 (Q' (Y - K c))(0:4).
//
// Affine (reference: q_affine_compute_affinmatrix_3D,
// q_warp_affine_tps.cpp:649-731, newmat SVD of the 3N x 13 DLT matrix):
// one CTA normalises both point sets, accumulates the 13 x 13 normal matrix
// in FP64 and takes the eigenvector of its smallest eigenvalue by cyclic
// Jacobi, which is the right singular vector the reference uses.

#include "tw_internal.h"
#include "tw_kdist.h"

#include <cmath>
#include <cstring>
#include <vector>

namespace tw {

namespace {

constexpr int kRedThreads = 1024;

// status word bits
constexpr int kStSingularX = 1;
constexpr int kStNotSPD = 2;   // set by the Cholesky kernel (tw_chol.cu)
constexpr int kStTimeout = 4;

// The vector kernels below run as one CTA and are a chain of block-wide sums;
// their time is the latency of those rounds.  Sums that do not depend on one
// another share a round (the four right-hand sides, the dot products of one
// reflector), and one thread per sum adds the warps' parts, where every thread
// adding all 32 of them took 2000 cycles a round in shared-memory loads.  Each
// sum still adds the same terms in the same order: lanes as a tree, then warps
// 0, 1, ... (warps past the last landmark hold zeros and are left out).
constexpr int kMostSums = 12;
struct SumSmem {
    double part[kMostSums][33];
    double sum[kMostSums];
};

template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], int n, SumSmem &S)
{
    static_assert(N <= kMostSums, "sums per round");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < N; ++i) S.part[i][warp] = v[i];
    __syncthreads();
    if (threadIdx.x < N) {
        double t = 0.0;
        const int nw = min((int)blockDim.x >> 5, (n + 31) >> 5);
#pragma unroll 8
        for (int w = 0; w < nw; ++w) t += S.part[threadIdx.x][w];
        S.sum[threadIdx.x] = t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = S.sum[i];
}

// Reflector k of the QR below: the rows' column k is turned into V's, and the
// columns from k on are updated.
template <int K>
__device__ __forceinline__ void qr_step(int n, double nrm2, double colnorm, double *Xw, double *V, double *tau, double *R,
                                        int *status, SumSmem &S)
{
    const double nrm = sqrt(nrm2);
    const double xkk = Xw[K * 4 + K];
    const double alpha = xkk > 0 ? -nrm : nrm;
    const double vk = xkk - alpha;
    const double vv = nrm2 - xkk * xkk + vk * vk;
    const double t = vv > 0 ? 2.0 / vv : 0.0;
    double d[4 - K];
#pragma unroll
    for (int j = 0; j < 4 - K; ++j) d[j] = 0.0;
#pragma unroll 4
    for (int i = K + threadIdx.x; i < n; i += blockDim.x) {
        const double v = i == K ? vk : Xw[i * 4 + K];
        V[i * 4 + K] = v;
#pragma unroll
        for (int j = 0; j < 4 - K; ++j) d[j] += v * Xw[i * 4 + K + j];
    }
    if (threadIdx.x < K) V[threadIdx.x * 4 + K] = 0.0;
    block_sums(d, n, S);
    if (threadIdx.x == 0) {
        tau[K] = t;
        R[K * 4 + K] = alpha;
        for (int j = 0; j < K; ++j) R[K * 4 + j] = 0.0;
        if (!(fabs(alpha) > 1e-10 * (colnorm + 1e-300))) atomicOr(status, kStSingularX);
    }
#pragma unroll 4
    for (int i = K + threadIdx.x; i < n; i += blockDim.x) {
        const double v = i == K ? vk : Xw[i * 4 + K];
#pragma unroll
        for (int j = 4 - K - 1; j >= 0; --j) {  // column K last: it is v itself
            const double sj = t * d[j];
            const double x = Xw[i * 4 + K + j] - sj * v;
            Xw[i * 4 + K + j] = x;
            if (i == K && j > 0) R[K * 4 + K + j] = x;
        }
    }
    __syncthreads();
}

// 1. Householder QR of X = [1 s].  Xw (n x 4) is a work copy; V (n x 4) gets
// the reflectors (zeros above the diagonal), tau[4], R[16].
__global__ void k_qr(const double *ctr, int n, double *Xw, double *V, double *tau, double *R, int *status)
{
    __shared__ SumSmem S;
    double s[4] = {0.0, 0.0, 0.0, 0.0};  // squared column norms; the first is also the first reflector's
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double x[4] = {1.0, ctr[3 * i], ctr[3 * i + 1], ctr[3 * i + 2]};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            Xw[i * 4 + j] = x[j];
            s[j] += x[j] * x[j];
        }
    }
    block_sums(s, n, S);
    double c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = sqrt(s[j]);
    qr_step<0>(n, s[0], c[0], Xw, V, tau, R, status, S);
    auto norm2 = [&](int k) {
        double q[1] = {0.0};
        for (int i = k + threadIdx.x; i < n; i += blockDim.x) q[0] += Xw[i * 4 + k] * Xw[i * 4 + k];
        block_sums(q, n, S);
        return q[0];
    };
    qr_step<1>(n, norm2(1), c[1], Xw, V, tau, R, status, S);
    qr_step<2>(n, norm2(2), c[2], Xw, V, tau, R, status, S);
    qr_step<3>(n, norm2(3), c[3], Xw, V, tau, R, status, S);
}

// out (n x 4) = K B for the implicit K_ij = -|s_i - s_j|; one warp per row.
// The eight rows of a CTA share the other side's landmarks and B, staged in
// shared memory component by component (read from global memory, each lane's
// seven strided loads per term bounded it: 91 us at n = 4096); what is left is
// the FP64 pipe's square roots.
constexpr int kKmulTile = 256;
__global__ void __launch_bounds__(256) k_kmul(const double *__restrict__ ctr, int n, const double *__restrict__ B,
                                              double *__restrict__ out)
{
    __shared__ double c[3][kKmulTile], q[4][kKmulTile];
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int r = min(row, n - 1);
    const double x = ctr[3 * r], y = ctr[3 * r + 1], z = ctr[3 * r + 2];
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    for (int j0 = 0; j0 < n; j0 += kKmulTile) {
        const int cnt = min(kKmulTile, n - j0);
        __syncthreads();
        for (int e = threadIdx.x; e < 3 * cnt; e += 256) c[e % 3][e / 3] = ctr[3 * (size_t)j0 + e];
        for (int e = threadIdx.x; e < 4 * cnt; e += 256) q[e & 3][e >> 2] = B[4 * (size_t)j0 + e];
        __syncthreads();
#pragma unroll 4
        for (int j = lane; j < cnt; j += 32) {
            const double k = kdist(x, y, z, c[0][j], c[1][j], c[2][j]);
            a0 += k * q[0][j];
            a1 += k * q[1][j];
            a2 += k * q[2][j];
            a3 += k * q[3][j];
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        a3 += __shfl_xor_sync(0xffffffffu, a3, o);
    }
    if (lane == 0 && row < n) {
        out[row * 4 + 0] = a0;
        out[row * 4 + 1] = a1;
        out[row * 4 + 2] = a2;
        out[row * 4 + 3] = a3;
    }
}

// Applies reflector k to the four columns of Z's rows; d: its sums V_k . Z_c.
__device__ __forceinline__ void reflect(int n, int k, const double *V, double tau, const double (&d)[4], double *Z)
{
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = V[i * 4 + k];
#pragma unroll
        for (int c = 0; c < 4; ++c) Z[i * 4 + c] -= tau * d[c] * v;
    }
}

// Step K of k_wvec: w_K, and reflector K applied to Z.
template <int K>
__device__ __forceinline__ void wvec_step(int n, const double *V, const double *tau, const double *P0, double *W, double *Z,
                                          SumSmem &S)
{
    // p_K = P0_K - sum_{j<K} [ v_j (w_j . v_K) + w_j (v_j . v_K) ]; the sums
    // V_K . Z_c ride along
    double s[2 * K + 4];
#pragma unroll
    for (int j = 0; j < 2 * K + 4; ++j) s[j] = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = V[i * 4 + K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
            s[2 * j] += W[i * 4 + j] * v;
            s[2 * j + 1] += V[i * 4 + j] * v;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) s[2 * K + c] += v * Z[i * 4 + c];
    }
    block_sums(s, n, S);
    double beta[1] = {0.0};
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double p = P0[i * 4 + K];
#pragma unroll
        for (int j = 0; j < K; ++j) p -= V[i * 4 + j] * s[2 * j] + W[i * 4 + j] * s[2 * j + 1];
        W[i * 4 + K] = p;  // temporarily p
        beta[0] += V[i * 4 + K] * p;
    }
    const double d[4] = {s[2 * K], s[2 * K + 1], s[2 * K + 2], s[2 * K + 3]};
    reflect(n, K, V, tau[K], d, Z);
    block_sums(beta, n, S);
    const double t = tau[K];
    const double cf = 0.5 * t * t * beta[0];
    for (int i = threadIdx.x; i < n; i += blockDim.x) W[i * 4 + K] = t * W[i * 4 + K] - cf * V[i * 4 + K];
}

// 2. From P0 = K V derive the rank-2 update vectors W (n x 4), and Z = Q' Y.
// (A thread reads only rows that it wrote.)
__global__ void k_wvec(int n, const double *V, const double *tau, const double *P0, double *W, const double *Y,
                       double *Z)
{
    __shared__ SumSmem S;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        for (int c = 0; c < 4; ++c) Z[i * 4 + c] = Y[i * 4 + c];
    wvec_step<0>(n, V, tau, P0, W, Z, S);
    wvec_step<1>(n, V, tau, P0, W, Z, S);
    wvec_step<2>(n, V, tau, P0, W, Z, S);
    wvec_step<3>(n, V, tau, P0, W, Z, S);
}

__device__ __forceinline__ void reflector_sums(int n, int k, const double *V, const double *Z, double (&d)[4], SumSmem &S)
{
#pragma unroll
    for (int c = 0; c < 4; ++c) d[c] = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = V[i * 4 + k];
#pragma unroll
        for (int c = 0; c < 4; ++c) d[c] += v * Z[i * 4 + c];
    }
    block_sums(d, n, S);
}

// 4c. c = H1 H2 H3 H4 [0; w]  (Z rows 0..3 are replaced by zeros)
__global__ void k_apply_q(int n, const double *V, const double *tau, const double *Z, double *C)
{
    __shared__ SumSmem S;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        for (int c = 0; c < 4; ++c) C[i * 4 + c] = i < 4 ? 0.0 : Z[i * 4 + c];
    for (int k = 3; k >= 0; --k) {
        double d[4];
        reflector_sums(n, k, V, C, d, S);
        reflect(n, k, V, tau[k], d, C);
    }
}

// 4d. d = R^-1 (Q' (Y - K c))(0:4); KC = K c precomputed.
__global__ void k_finish_d(int n, const double *V, const double *tau, const double *R, const double *Y, double *KC,
                           double *d_out)
{
    __shared__ SumSmem S;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        for (int c = 0; c < 4; ++c) KC[i * 4 + c] = Y[i * 4 + c] - KC[i * 4 + c];
    for (int k = 0; k < 4; ++k) {
        double d[4];
        reflector_sums(n, k, V, KC, d, S);
        reflect(n, k, V, tau[k], d, KC);
    }
    __syncthreads();
    if (threadIdx.x < 4) {  // one thread per right-hand side
        const int c = threadIdx.x;
        double x[4];
#pragma unroll
        for (int a = 3; a >= 0; --a) {
            double s = KC[a * 4 + c];
#pragma unroll
            for (int b = a + 1; b < 4; ++b) s -= R[a * 4 + b] * x[b];
            x[a] = s / R[a * 4 + a];
            d_out[a * 4 + c] = x[a];
        }
    }
}

// 5. FP32 evaluation arrays: centres relative to the origin o, and the
// negated non-affine coefficients (-c_x, -c_y, -c_z, 0).
__global__ void k_eval_arrays(int n, const double *ctr, const double *C, double ox, double oy, double oz,
                              float4 *ctr32, float4 *coef32)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ctr32[i] = make_float4((float)(ctr[3 * i] - ox), (float)(ctr[3 * i + 1] - oy), (float)(ctr[3 * i + 2] - oz), 0.f);
    coef32[i] = make_float4((float)(-C[4 * i + 1]), (float)(-C[4 * i + 2]), (float)(-C[4 * i + 3]), 0.f);
}

// ----------------------------------------------------------- affine DLT
//
// One CTA.  The fit is a serial chain -- the cyclic Jacobi iteration's angles,
// each two square roots and three divisions after the one before -- so its
// time is latency.  One thread doing every rotation, with the 39 element
// pairs of each in a loop, took 580 of the kernel's 622 us at 16 pairs of
// landmarks (8 sweeps).  Here the operations on every matrix element are the
// same and in the same order, but spread over a wavefront:
//  - the angle of rotation (p, q) needs only the elements of rows and columns
//    p and q against each other, so (p, q) runs at step 2p + q of the sweep, 34
//    steps instead of 78, up to four rotations a step, one warp each;
//  - a rotation is applied at once to the indices p < k <= q + 1, to a later
//    index k just before (p, k) needs it (by a second warp, while the angles of
//    that step are computed), and to the indices k < p at the end of the sweep:
//    no angle of the same sweep reads those;
//  - the eigenvector matrix follows one sweep behind, on a warp of its own.
// Every element so meets its rotations in the sequential order, and the matrix
// is the same to the last bit.  Four warps compute angles, four catch up, one
// keeps the vectors (one angle warp per SM sub-partition; 16 warps made every
// barrier dearer and left too few registers for the rows).  169 us at 16 pairs:
// 110 of them are the 34 x 7 angles' own square roots and divisions.

constexpr int kFitRed = 256;                        // threads that hold landmarks in the sums
constexpr int kFitAgents = 4;                       // warps computing angles: p and p + 4 are never active together
constexpr int kFitThreads = 32 * (2 * kFitAgents + 1);  // + as many catch-up warps + the eigenvector warp
constexpr int kFitDim = 13;
constexpr int kFitUpper = kFitDim * (kFitDim + 1) / 2;  // entries of the normal matrix

struct FitSmem {
    double sh[6][kFitRed / 32];
    double part[kFitRed / 32][kFitUpper];
    double A[kFitDim][kFitDim], V[kFitDim][kFitDim];
    double2 R[2][kFitDim - 1][kFitDim];             // (cos, sin) of rotation (p, q), this sweep's and the last one's
    double one;                                     // 1.0, the homogeneous coordinate of every point
    int go;
};

// N sums over the first kFitRed threads' values (the others pass zeros): a
// tree inside each warp, then the warps in order.
template <int N>
__device__ __forceinline__ void fit_sums(double (&v)[N], FitSmem &S)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0 && warp < kFitRed / 32)
#pragma unroll
        for (int i = 0; i < N; ++i) S.sh[i][warp] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kFitRed / 32; ++w) t += S.sh[i][w];
        v[i] = t;
    }
}

// The angle of the rotation that zeroes apq; kFitSkip when it is zero already.
constexpr double kFitSkip = 2.0;  // in place of a cosine: the rotation is left out
__device__ __forceinline__ double2 fit_angle(double app, double aqq, double apq)
{
    if (fabs(apq) < 1e-300) return make_double2(kFitSkip, 0.0);
    const double theta = (aqq - app) / (2.0 * apq);
    const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(fma(theta, theta, 1.0)));
    const double cs = 1.0 / sqrt(fma(t, t, 1.0));
    return make_double2(cs, t * cs);
}

__device__ __forceinline__ bool fit_used(double2 r) { return __double2hiint(r.x) != 0x40000000; }

__device__ __forceinline__ void fit_rot(double &x, double &y, double2 r)
{
    const double a = x, b = y;
    x = fma(r.x, a, -__dmul_rn(r.y, b));
    y = fma(r.y, a, __dmul_rn(r.x, b));
}

// The same where `on`, without a branch: a chain of these stays a chain of
// multiply-adds.
__device__ __forceinline__ void fit_rot_if(double &x, double &y, double2 r, bool on)
{
    double a = x, b = y;
    fit_rot(a, b, r);
    x = on ? a : x;
    y = on ? b : y;
}

// Rotations (p, q), p < q < qe, in order, on the pairs (row[p], row[q]) of a
// row or column with element stride `st`; the loads come first, so that only
// the chain through row[p] is serial.
__device__ __forceinline__ void fit_catch_up(double *row, int st, int p, int qe, const double2 *R)
{
    constexpr int kMost = kFitDim - 3;
    double x = row[p * st], y[kMost];
    double2 r[kMost];
#pragma unroll
    for (int j = 0; j < kMost; ++j) {
        const int q = min(p + 1 + j, kFitDim - 1);
        y[j] = row[q * st];
        r[j] = R[q];
    }
#pragma unroll
    for (int j = 0; j < kMost; ++j) fit_rot_if(x, y[j], r[j], p + 1 + j < qe && fit_used(r[j]));
#pragma unroll
    for (int j = 0; j < kMost; ++j)
        if (p + 1 + j < qe) row[(p + 1 + j) * st] = y[j];
    row[p * st] = x;
}

// All rotations of a sweep with p >= p0 (p0 uniform or not), in order, on one
// row or column with element stride `st`, held in registers.
__device__ __forceinline__ void fit_replay(double *row, int st, int p0, const double2 (*R)[kFitDim])
{
    double v[kFitDim];
#pragma unroll
    for (int k = 0; k < kFitDim; ++k) v[k] = row[k * st];
#pragma unroll
    for (int p = 0; p < kFitDim - 1; ++p)
#pragma unroll
        for (int q = p + 1; q < kFitDim; ++q) {
            const double2 r = R[p][q];
            fit_rot_if(v[p], v[q], r, p >= p0 && fit_used(r));
        }
#pragma unroll
    for (int k = 0; k < kFitDim; ++k) row[k * st] = v[k];
}

// One sweep on A (warps 0 .. 2 kFitAgents - 1); R / skip get its rotations.
__device__ __forceinline__ void fit_sweep(FitSmem &S, double2 (*R)[kFitDim])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int agent = warp % kFitAgents;
    const bool angles = warp < kFitAgents;
    for (int s = 1; s <= 2 * (kFitDim - 2) + kFitDim - 1; ++s) {
        // the agent's rotation of this step: (p, s - 2p) with p < s - 2p < kFitDim
        int p = agent;
        while (s - 2 * p >= kFitDim) p += kFitAgents;
        const int q = s - 2 * p;
        const bool on = p < kFitDim - 1 && q > p && q < kFitDim;
        double2 r = make_double2(kFitSkip, 0.0);
        double app = 0, aqq = 0, apq = 0, aqp = 0;
        if (on && angles) {
            app = S.A[p][p];
            aqq = S.A[q][q];
            apq = S.A[p][q];
            aqp = S.A[q][p];
            r = fit_angle(app, aqq, apq);
            if (lane == 0) R[p][q] = r;
        } else if (on && q + 1 < kFitDim && q > p + 1 && (lane & 15) == 0) {
            const int k = q + 1;
            fit_catch_up(lane == 0 ? &S.A[k][0] : &S.A[0][k], lane == 0 ? 1 : kFitDim, p, q, R[p]);
        }
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(64 * kFitAgents) : "memory");
        if (on && angles && fit_used(r)) {
            const int k = lane & 15;
            const bool mine = k > p && k <= q + 1 && k < kFitDim && k != q;
            const int kk = mine ? k : p;
            double *x = lane < 16 ? &S.A[kk][p] : &S.A[p][kk];
            double *y = lane < 16 ? &S.A[kk][q] : &S.A[q][kk];
            double u = *x, v = *y;
            fit_rot(u, v, r);
            // the rotation's own 2 x 2 block: columns, then rows
            fit_rot(app, apq, r);
            fit_rot(aqp, aqq, r);
            fit_rot(app, aqp, r);
            fit_rot(apq, aqq, r);
            __syncwarp();
            if (mine) {
                *x = u;
                *y = v;
            }
            if (lane == 0) {
                S.A[p][p] = app;
                S.A[p][q] = apq;
                S.A[q][p] = aqp;
                S.A[q][q] = aqq;
            }
        }
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(64 * kFitAgents) : "memory");
    }
    // the indices below each rotation's p
    if (warp == 0) {
        const int k = lane & 15;
        if (k < kFitDim - 2) fit_replay(lane < 16 ? &S.A[k][0] : &S.A[0][k], lane < 16 ? 1 : kFitDim, k + 1, R);
    }
}

__device__ __forceinline__ void fit_vectors(FitSmem &S, int buf)
{
    const int k = threadIdx.x & 31;
    if (k < kFitDim) fit_replay(&S.V[k][0], 1, 0, S.R[buf]);
}

// tar and sub are the call's own copies and are normalised in place.
__global__ void __launch_bounds__(kFitThreads) k_affine_fit(double *tar, double *sub, int n, double *out, int *status)
{
    __shared__ FitSmem S;
    const int tid = threadIdx.x;
    const int i0 = tid < kFitRed ? tid : n;  // threads past kFitRed hold no landmark
    // Hartley normalisation of both sets (0: tar, 1: sub): centroid, 1 / mean distance
    double c[6] = {0, 0, 0, 0, 0, 0}, scale[2] = {0, 0};
    for (int i = i0; i < n; i += kFitRed)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            c[q] += tar[3 * i + q];
            c[3 + q] += sub[3 * i + q];
        }
    if (tid == 0) S.one = 1.0;
    fit_sums(c, S);
#pragma unroll
    for (int q = 0; q < 6; ++q) c[q] /= n;
    for (int i = i0; i < n; i += kFitRed)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double *p = s == 0 ? tar : sub;
            const double dx = p[3 * i] - c[3 * s], dy = p[3 * i + 1] - c[3 * s + 1], dz = p[3 * i + 2] - c[3 * s + 2];
            scale[s] += sqrt(fma(dz, dz, fma(dx, dx, __dmul_rn(dy, dy))));
        }
    fit_sums(scale, S);
#pragma unroll
    for (int s = 0; s < 2; ++s) scale[s] = 1.0 / (scale[s] / n);
    for (int i = i0; i < n; i += kFitRed)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            tar[3 * i + q] = (tar[3 * i + q] - c[q]) * scale[0];
            sub[3 * i + q] = (sub[3 * i + q] - c[3 + q]) * scale[1];
        }
    __syncthreads();
    // normal matrix of the 3n x 13 DLT system, three rows per point,
    // [a 1 0 0 -bx], [0 a 1 0 -by], [0 0 a 1 -bz] with a = (ax, ay, az): one
    // thread per entry (r, c) and warp's share of the points, summed as the
    // lanes of that warp would (products with a zero add nothing)
    const int nw = min(kFitRed / 32, (n + 31) / 32);
    for (int t = tid; t < kFitUpper * nw; t += kFitThreads) {
        const int e = t % kFitUpper, w = t / kFitUpper;
        int r = 0, f = e;
        while (f >= kFitDim - r) {
            f -= kFitDim - r;
            ++r;
        }
        const int cc = r + f;
        double v[32];
#pragma unroll
        for (int l = 0; l < 32; ++l) v[l] = 0.0;
        if (cc == 12 || r / 4 == cc / 4) {
            // the entry's factors: element k of a (1 for k = 3), or -b[k]
            const bool bu = r == 12, bv = cc == 12;
            const int kv = r / 4 % 3;  // of -b, for r < 12
            const double *pu = bu ? sub : (r % 4 == 3 ? &S.one : tar + r % 4);
            const double *pv = bv ? sub + (bu ? 0 : kv) : (cc % 4 == 3 ? &S.one : tar + cc % 4);
            const int su = !bu && r % 4 == 3 ? 0 : 3, sv = !bv && cc % 4 == 3 ? 0 : 3;
            const double sg = bv && !bu ? -1.0 : 1.0;
            for (int b = 32 * w; b < n; b += kFitRed) {
#pragma unroll
                for (int l = 0; l < 32; ++l) {
                    const int i = min(b + l, n - 1);
                    const double x = pu[i * su], y = sg * pv[i * sv];
                    double t = fma(x, y, v[l]);
                    if (bu) {
                        t = fma(pu[i * 3 + 1], pv[i * 3 + 1], t);
                        t = fma(pu[i * 3 + 2], pv[i * 3 + 2], t);
                    }
                    if (b + l < n) v[l] = t;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int l = 0; l < o; ++l) v[l] += v[l + o];
        S.part[w][e] = v[0];
    }
    __syncthreads();
    if (tid < kFitUpper) {
        int r = 0, f = tid;
        while (f >= kFitDim - r) {
            f -= kFitDim - r;
            ++r;
        }
        double acc = 0.0;
        for (int w = 0; w < nw; ++w) acc += S.part[w][tid];
        S.A[r][r + f] = acc;
        S.A[r + f][r] = acc;
    }
    for (int e = tid; e < kFitDim * kFitDim; e += kFitThreads) S.V[e / kFitDim][e % kFitDim] = e % (kFitDim + 1) == 0 ? 1.0 : 0.0;
    __syncthreads();
    const int warp = tid >> 5;
    int sweep = 0;
    for (; sweep < 100; ++sweep) {
        if (tid == 0) {
            double off = 0, diag = 0;
#pragma unroll
            for (int p = 0; p < kFitDim; ++p) {
                diag += S.A[p][p] * S.A[p][p];
#pragma unroll
                for (int q = p + 1; q < kFitDim; ++q) off += S.A[p][q] * S.A[p][q];
            }
            S.go = !(off <= 1e-30 * diag);
        }
        __syncthreads();
        if (!S.go) break;
        if (warp < 2 * kFitAgents) fit_sweep(S, S.R[sweep & 1]);
        else if (sweep > 0) fit_vectors(S, (sweep - 1) & 1);
        __syncthreads();
    }
    if (warp == 2 * kFitAgents && sweep > 0) fit_vectors(S, (sweep - 1) & 1);
    __syncthreads();
    if (tid == 0) {
        int best = 0;
        for (int p = 1; p < kFitDim; ++p)
            if (S.A[p][p] < S.A[best][best]) best = p;
        double h[kFitDim];
        for (int i = 0; i < kFitDim; ++i) h[i] = S.V[i][best];
        if (h[12] == 0.0) {
            atomicOr(status, kStSingularX);
            return;
        }
        for (int i = 0; i < kFitDim; ++i) h[i] /= h[12];
        // T = NB^-1 H NA with N = [s I, -s c; 0 1]:  NB^-1 = [I/sB, cB; 0 1]
        const double sA = scale[0], sB = scale[1];
        double H[3][4];
        for (int r = 0; r < 3; ++r)
            for (int k = 0; k < 4; ++k) H[r][k] = h[r * 4 + k];
        for (int r = 0; r < 3; ++r) {
            // (H NA)(r,:) = [sA H(r,0:3), H(r,3) - sA H(r,0:3).cA]
            double lin[3], tr = H[r][3];
            for (int k = 0; k < 3; ++k) {
                lin[k] = sA * H[r][k];
                tr = fma(-lin[k], c[k], tr);
            }
            for (int k = 0; k < 3; ++k) out[r * 4 + k] = lin[k] / sB;
            out[r * 4 + 3] = tr / sB + c[3 + r];
        }
        out[12] = 0; out[13] = 0; out[14] = 0; out[15] = 1;
    }
}

struct StreamBuf {
    tw_ctx *ctx = nullptr;
    cudaStream_t st = nullptr;
    void *p = nullptr;
    size_t bytes = 0;
    ~StreamBuf() { if (p) dfree_on(ctx, p, bytes, st); }
};

}  // namespace

// The status word of a solve as a tw_status.
static tw_status status_of(tw_ctx *ctx, int status)
{
    if (status & kStSingularX)
        return fail(ctx, TW_ERR_SINGULAR, "TPS centres are degenerate: [1 s] is rank deficient (coplanar or < 4 distinct points)");
    if (status & kStTimeout)
        return fail(ctx, TW_ERR_TIMEOUT, "TPS solve: a wait on another block of the solve timed out");
    if (status & kStNotSPD)
        return fail(ctx, TW_ERR_SINGULAR, "projected TPS system is not positive definite");
    return TW_OK;
}

tw_status solve_tps_device(tw_ctx *ctx, const double *h_ctr, const double *h_val, int n, double lambda,
                           double *d_c_out, double *d_d_out, int *d_status_out, double *h_d_out, const double o[3],
                           float4 *ctr32_out, float4 *coef32_out, cudaStream_t st, double *h_stage)
{
    const int m = n - 4;
    // workspace: ctr 3n, Y/Xw/V/P/W/Z/KC 4n each, tau 4, R 16
    const size_t small = 3 * (size_t)n + 7 * 4 * (size_t)n + 4 + 16;
    // stream-ordered workspace on `st`, returned to the pool on `st` when this
    // function exits (after the final wait, or with the error)
    StreamBuf ws{ctx, st}, abuf{ctx, st};
    ws.bytes = small * sizeof(double);
    TW_TRY(dmalloc_on(ctx, &ws.p, ws.bytes, st));
    double *base = static_cast<double *>(ws.p);
    double *d_ctr = base;
    double *d_Y = d_ctr + 3 * (size_t)n;
    double *d_Xw = d_Y + 4 * (size_t)n;
    double *d_V = d_Xw + 4 * (size_t)n;
    double *d_P = d_V + 4 * (size_t)n;
    double *d_W = d_P + 4 * (size_t)n;
    double *d_Z = d_W + 4 * (size_t)n;
    double *d_KC = d_Z + 4 * (size_t)n;
    double *d_tau = d_KC + 4 * (size_t)n;
    double *d_R = d_tau + 4;
    double *d_d = d_d_out;
    int *d_status = d_status_out;
    if (m > 0) {
        abuf.bytes = chol_work_bytes(m);
        TW_TRY(dmalloc_on(ctx, &abuf.p, abuf.bytes, st));
    }

    std::vector<double> hY(4 * (size_t)n);
    for (int i = 0; i < n; ++i) {
        hY[4 * i + 0] = 1.0;
        hY[4 * i + 1] = h_val[3 * i + 0];
        hY[4 * i + 2] = h_val[3 * i + 1];
        hY[4 * i + 3] = h_val[3 * i + 2];
    }
    if (h_stage) {
        std::memcpy(h_stage, h_ctr, sizeof(double) * 3 * n);
        std::memcpy(h_stage + 3 * (size_t)n, hY.data(), sizeof(double) * 4 * n);
        TW_CUDA_TRY(cudaMemcpyAsync(d_ctr, h_stage, sizeof(double) * 7 * n, cudaMemcpyHostToDevice, st));
    } else {  // (centres and values are consecutive in the workspace)
        hY.insert(hY.begin(), h_ctr, h_ctr + 3 * (size_t)n);
        TW_TRY(upload(ctx, d_ctr, hY.data(), sizeof(double) * 7 * n, st));
    }
    // d, and the status word after it
    TW_CUDA_TRY(cudaMemsetAsync(d_d, 0, sizeof(double) * 16 + sizeof(int), st));

    uint64_t nl = 0;
    k_qr<<<1, kRedThreads, 0, st>>>(d_ctr, n, d_Xw, d_V, d_tau, d_R, d_status);
    ++nl;
    const int warps_per_block = 8;
    const unsigned kgrid = (unsigned)((n + warps_per_block - 1) / warps_per_block);
    k_kmul<<<kgrid, 32 * warps_per_block, 0, st>>>(d_ctr, n, d_V, d_P);
    k_wvec<<<1, kRedThreads, 0, st>>>(n, d_V, d_tau, d_P, d_W, d_Y, d_Z);
    nl += 2;
    if (m > 0) {
        TW_CUDA_TRY(launch_chol_solve(d_ctr, n, d_V, d_W, d_Z, lambda, abuf.p, d_status, ctx->solve_barrier_ns.load(),
                                      ctx->sm_count, st));
        nl += 2;
    }
    k_apply_q<<<1, kRedThreads, 0, st>>>(n, d_V, d_tau, d_Z, d_c_out);
    k_kmul<<<kgrid, 32 * warps_per_block, 0, st>>>(d_ctr, n, d_c_out, d_KC);
    k_finish_d<<<1, kRedThreads, 0, st>>>(n, d_V, d_tau, d_R, d_Y, d_KC, d_d);
    nl += 3;
    if (ctr32_out && coef32_out) {
        k_eval_arrays<<<(n + 255) / 256, 256, 0, st>>>(n, d_ctr, d_c_out, o[0], o[1], o[2], ctr32_out, coef32_out);
        ++nl;
    }
    TW_CUDA_TRY(cudaGetLastError());
    count_launch(ctx, nl);
    if (!h_d_out) return TW_OK;  // the caller reads the status later
    // d and the status word after it in one copy
    struct { double d[16]; int status; } h;
    TW_CUDA_TRY(cudaMemcpyAsync(&h, d_d, sizeof(double) * 16 + sizeof(int), cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaStreamSynchronize(st));
    std::memcpy(h_d_out, h.d, sizeof(h.d));
    return status_of(ctx, h.status);
}

tw_status solve_status(tw_ctx *ctx, const int *d_status, cudaStream_t st)
{
    int status = 0;
    TW_CUDA_TRY(cudaMemcpyAsync(&status, d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaStreamSynchronize(st));
    return status_of(ctx, status);
}

tw_status fit_affine_device(tw_ctx *ctx, const double *h_tar, const double *h_sub, int n, double M[16],
                            cudaStream_t st)
{
    StreamBuf ws{ctx, st};
    ws.bytes = sizeof(double) * (6 * (size_t)n + 16 + 2);
    TW_TRY(dmalloc_on(ctx, &ws.p, ws.bytes, st));
    double *d_tar = static_cast<double *>(ws.p);
    double *d_sub = d_tar + 3 * (size_t)n;
    double *d_out = d_sub + 3 * (size_t)n;
    int *d_status = reinterpret_cast<int *>(d_out + 16);
    // landmarks, a zero matrix and a zero status word in one upload
    std::vector<double> h(6 * (size_t)n + 18, 0.0);
    std::memcpy(h.data(), h_tar, sizeof(double) * 3 * n);
    std::memcpy(h.data() + 3 * (size_t)n, h_sub, sizeof(double) * 3 * n);
    TW_TRY(upload(ctx, ws.p, h.data(), ws.bytes, st));
    k_affine_fit<<<1, kFitThreads, 0, st>>>(d_tar, d_sub, n, d_out, d_status);
    TW_CUDA_TRY(cudaGetLastError());
    count_launch(ctx, 1);
    struct { double M[16]; int status; } r;
    TW_CUDA_TRY(cudaMemcpyAsync(&r, d_out, sizeof(double) * 16 + sizeof(int), cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaStreamSynchronize(st));
    std::memcpy(M, r.M, sizeof(r.M));
    if (r.status) return fail(ctx, TW_ERR_SINGULAR, "affine DLT is degenerate (h13 = 0)");
    return TW_OK;
}

cudaError_t launch_affine_fit(double *d_tar, double *d_sub, int n, double *d_out, int *d_status,
                              cudaStream_t st)
{
    k_affine_fit<<<1, kFitThreads, 0, st>>>(d_tar, d_sub, n, d_out, d_status);
    return cudaGetLastError();
}

}  // namespace tw
