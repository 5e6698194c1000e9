// tw_chol.cu -- the FP64 Cholesky factorisation and the two triangular solves
// of the projected TPS system, one cooperative kernel.
//
// A (m x m, symmetric positive definite) is held as 64 x 64 tiles of its lower
// triangle, each stored with a row pitch of 68 doubles: a tile is one
// contiguous 34,816-byte block that a single bulk copy moves between global
// and shared memory, already in the layout whose 16-byte row loads are free of
// bank conflicts.  Column 64 of a factored diagonal tile holds the reciprocals
// of its diagonal and its upper triangle the transpose of the lower, so the
// panel solves read both along rows.  The four right-hand sides are an extra
// row block of 4 x 68 tiles, so the forward substitution is part of the
// factorisation; the back substitution overwrites the same tiles.
//
// Roles.  CTA 0 runs the critical chain POTRF(k-1) -> TRSM(k, k-1) ->
// SYRK(k, k, k-1) -> POTRF(k) with its tiles in shared memory and registers.
// The other CTAs take tiles in column order from a counter; a tile's owner
// holds it in registers, subtracts L(i,k) L(j,k)' for k = 0, 1, ... as the
// panels become available (each product summed over its 64 columns first,
// then subtracted), solves it against the factored diagonal tile and
// publishes it.  The tiles (j, j) and (j+1, j) go to the chain instead, one
// update and the solve short.  A task waits only for the chain and for tasks
// before it in the order, and every CTA is resident (cooperative launch), so
// the lowest unfinished task can always run.
//
// In each CTA 8 warps compute, one warp fetches tiles ahead of them (bulk
// copies into a ring of shared-memory buffers, after the flag that publishes
// each tile) and one warp stores results and publishes them.  In the chain
// neither a flag's round trip nor a store's completion stands on the compute
// warps' path.  A helper's warps all meet between tasks, after its tile is
// published: there a store's completion, the claim of the next task and that
// task's first fetch do.  What bounds it: latency up to about 3000 landmarks -- per 64 columns
// the chain takes some 25,000 cycles (diagonal tile 14,000: 64 dependent
// pivots, each a reciprocal square root, a product and a multiply-add, and
// three hand-overs between panels; panel tile's solution 5,000; its product
// 2,500), and a tile needs about as long from a diagonal tile's publication
// through a helper's solution and the next helper's product to the chain -- and
// the helpers' FP64 matrix instructions beyond (64 multiply-adds per SM and
// clock).  Solve of 500 / 2000 / 4096 landmarks: 337 / 1074 / 2452 us with
// scalar multiply-adds for products and solutions, 300 / 932 / 1984 now.
//
// Every element sees the operations of the plain right-looking tiled
// factorisation in the same order, whatever the schedule.
//
// Every wait is bounded: a wait that gives up sets the error flag, and from
// then on no wait of any CTA blocks, so every CTA runs to its end (indices do
// not depend on data) and the host reports the time-out.

#include "tw_internal.h"
#include "tw_kdist.h"

namespace tw {

namespace {

constexpr int kNB = 64;                        // tile
constexpr int kTP = 68;                        // tile row pitch, doubles
constexpr int kTileD = kNB * kTP;              // doubles of a tile
constexpr uint32_t kTileB = kTileD * 8;        // bytes
constexpr int kRhsD = 4 * kTP;                 // a right-hand-side tile
constexpr uint32_t kRhsB = kRhsD * 8;
constexpr int kCompute = 256;                  // compute threads
constexpr int kThreads = kCompute + 64;        // + the fetching warp + the publishing warp
constexpr int kFetchWarp = kCompute / 32, kPublishWarp = kFetchWarp + 1;
constexpr int kBufs = 6;                       // tile buffers in shared memory
constexpr int kPotBars = 23;                   // barriers inside a diagonal tile's factorisation

// status word bits
constexpr int kStNotSPD = 2;
constexpr int kStTimeout = 4;

static_assert(kTP - kNB == 4 && kTileB % 16 == 0 && kRhsB % 16 == 0, "bulk copies move multiples of 16 bytes");

// Flags (zeroed before the launch).  tdone[i]: panel tiles of row block i that
// are final (row block nblk: the right-hand sides); pre_d[j], pre_s[j]: tile
// (j, j) / (j+1, j) has been handed to the chain; bcnt[i]: block i of the right-hand sides has
// been handed to the chain's back substitution.
struct Flags {
    int err;    // a wait gave up
    int pdone;  // diagonal tiles factored
    int ddone;  // back-substitution blocks solved, from the last one down
    int next;   // tasks claimed
};

struct Ctl {
    double *tiles;  // lower-triangle tiles, column after column
    double *rhs;    // nblk tiles of 4 x 68
    double *x;      // the solution, 4 per row (rows 0 .. m-1)
    int m, nblk;
    int *status;
    Flags *F;
    int *tdone, *pre_d, *pre_s, *bcnt;
    unsigned long long limit_ns;
};

__device__ __forceinline__ size_t tile_index(int i, int j, int nblk)
{
    return (size_t)j * nblk - (size_t)j * (j - 1) / 2 + (i - j);
}
__device__ __forceinline__ double *tile_ptr(const Ctl &C, int i, int j)
{
    return C.tiles + tile_index(i, j, C.nblk) * kTileD;
}

struct Smem {
    double buf[kBufs][kTileD];
    double z[4][kRhsD];        // back substitution: right-hand sides of the blocks in flight (block & 3)
    double xs[4][kRhsD];       // and their solutions
    double small[kRhsD];       // helpers: right-hand-side tile of a panel / x of a block
    unsigned long long full[kBufs], empty[kBufs];
    unsigned long long zfull[4];
    unsigned long long post[2], freed[2];  // results handed to the publishing warp / their buffers read
    unsigned long long xdone;
    unsigned long long pot[kPotBars];
    // a result to publish: shared source, global destination, bytes, flag and its value
    struct Mail {
        const double *src;
        double *dst;
        uint32_t bytes;
        int *flag;
        int value;
    } mail[2];
    uint32_t issued[kBufs], zissued[4];  // copies begun into each buffer (fetching warp)
    int task;
    int abort;
};

static_assert(sizeof(Smem) <= 232448, "one CTA per SM");

// ------------------------------------------------------------ small helpers

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// The warp's index through a shuffle, so that the compiler knows it to be the
// same in all lanes: below a branch on threadIdx.x / 32 it guards shuffles and
// matrix instructions against lanes that went the other way (factor16 in a
// kernel of its own: 3,280 cycles instead of 2,350).
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }
__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// c ? a : b as one selection.  Written as a
// conditional expression it becomes a branch (one side's arithmetic sinks
// into them), and in the chains below a branch costs more than the arithmetic:
// solve4 210 cycles with, 86 without.
__device__ __forceinline__ double sel(int c, double a, double b)
{
    double r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.f64 %0, %1, %2, p;\n\t}" : "=d"(r) : "d"(a), "d"(b), "r"(c));
    return r;
}
__device__ __forceinline__ int ld_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int *p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void bar_init(unsigned long long *b, uint32_t n)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}
// Arrival of lane 0, without a branch.
__device__ __forceinline__ void bar_arrive_lane0(unsigned long long *b)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(saddr(b)),
                 "r"(threadIdx.x & 31)
                 : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned long long *b, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(saddr(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_copy(double *dst, const double *src, uint32_t bytes, unsigned long long *b)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(saddr(dst)),
                 "l"(src), "r"(bytes), "r"(saddr(b))
                 : "memory");
}
// One tile into buffer b, counted on its "full" barrier.
__device__ __forceinline__ void load_buf(Smem &S, int b, const double *src, uint32_t bytes)
{
    ++S.issued[b];
    bar_expect(&S.full[b], bytes);
    bulk_copy(S.buf[b], src, bytes, &S.full[b]);
}
// barrier of the compute warps
__device__ __forceinline__ void sync_compute()
{
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(kCompute) : "memory");
}

__device__ __noinline__ void give_up(const Ctl &C, Smem &S)
{
    atomicOr(&C.F->err, 1);
    atomicOr(C.status, kStTimeout);
    *reinterpret_cast<volatile int *>(&S.abort) = 1;
}

__device__ __noinline__ void bar_wait_slow(const Ctl &C, Smem &S, unsigned long long *b, uint32_t parity)
{
    const unsigned long long t0 = now_ns();
    for (unsigned i = 1;; ++i) {
        if (bar_try(b, parity) || *reinterpret_cast<volatile int *>(&S.abort)) return;
        if ((i & 15u) == 0 && now_ns() - t0 > C.limit_ns) {
            give_up(C, S);
            return;
        }
    }
}
// The n-th completion of the mbarrier (n counts from 0).  Returns at once
// when the CTA has given up.
__device__ __forceinline__ void bar_wait(const Ctl &C, Smem &S, unsigned long long *b, uint32_t n)
{
    if (!bar_try(b, n & 1u)) bar_wait_slow(C, S, b, n & 1u);
}
// A buffer's n-th reuse: the (n-1)-th release has happened (n = 0: it is free).
__device__ __forceinline__ void bar_wait_free(const Ctl &C, Smem &S, unsigned long long *b, uint32_t n)
{
    if (n > 0) bar_wait(C, S, b, n - 1);
}

// The same for the fetching warp, before it copies into a buffer: false once the
// CTA has given up.  The compute warps then no longer wait for what they read
// and release, so a release says nothing about the buffer any more, and a second
// copy counted on a "full" barrier whose phase is still open would let the CTA
// end before its copies have landed.
__device__ __forceinline__ bool claim_buf(const Ctl &C, Smem &S, unsigned long long *b, uint32_t n)
{
    bar_wait_free(C, S, b, n);
    return *reinterpret_cast<volatile int *>(&S.abort) == 0;
}

// Waits (one thread) until *flag >= want; false once anyone has given up.
__device__ bool flag_wait(const Ctl &C, Smem &S, const int *flag, int want)
{
    if (ld_acquire(flag) >= want) return *reinterpret_cast<volatile int *>(&S.abort) == 0;
    const unsigned long long t0 = now_ns();
    for (;;) {
        if (ld_acquire(flag) >= want) return *reinterpret_cast<volatile int *>(&S.abort) == 0;
        if (*reinterpret_cast<volatile int *>(&S.abort)) return false;
        if (*reinterpret_cast<volatile int *>(&C.F->err) || now_ns() - t0 > C.limit_ns) {
            give_up(C, S);
            return false;
        }
    }
}

// Hands a result in shared memory to the publishing warp (every compute
// thread calls it after its last write; thread 0 describes the result).
__device__ __forceinline__ void post(Smem &S, int b, const double *src, double *dst, uint32_t bytes, int *flag, int value)
{
    fence_async();
    if (threadIdx.x == 0) S.mail[b] = {src, dst, bytes, flag, value};
    __syncwarp();
    bar_arrive_lane0(&S.post[b]);
}

// The publishing warp's lane 0: stores the n-th result of mailbox b and
// raises its flag; false at the end.
__device__ bool publish(const Ctl &C, Smem &S, int b, uint32_t n)
{
    bar_wait(C, S, &S.post[b], n);
    if (*reinterpret_cast<volatile int *>(&S.abort)) return false;
    const Smem::Mail M = S.mail[b];
    if (!M.flag) return false;
    if (M.bytes) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(M.dst), "r"(saddr(M.src)), "r"(M.bytes)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    bar_arrive(&S.freed[b]);
    if (M.bytes) {
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        fence_async();
    }
    __threadfence();
    st_release(M.flag, M.value);
    return true;
}

// ------------------------------------------------------------- tile kernels
//
// Tile products run on the FP64 matrix instruction (m8n8k4): each element is
// the same chain of fused multiply-adds, in ascending order of k, that scalar
// code would run, so its bits do not depend on which of the two computes it.
// A compute warp owns eight rows of a tile, row block wr, as eight 8 x 8
// fragments: lane (lr, lc) = (lane / 4, lane % 4) holds the columns
// 8 f + 2 lc + {0, 1} of row 8 wr + lr.  The rows of a tile are 68 doubles
// apart, so the 8 x 4 operand fragments (row lr, column lc) are free of bank
// conflicts, and per four k's a warp loads nine of them for eight products:
// 144 of the 256 cycles that the products take.

using Frags = double[8][2];

// row block of a compute warp; the two warps of a sub-partition (w, w + 4)
// have nine lower fragments together
__device__ __forceinline__ int row_block()
{
    const int w = warp_index();
    return w < 4 ? w : 11 - w;
}
// element (row lr, column 2 lc) of row block wr of the tile T
__device__ __forceinline__ int frag_at(int wr)
{
    const int lane = threadIdx.x & 31;
    return (8 * wr + (lane >> 2)) * kTP + 2 * (lane & 3);
}
__device__ __forceinline__ void load_frags(const double *T, int wr, Frags &a)
{
    const double *p = T + frag_at(wr);
#pragma unroll
    for (int f = 0; f < 8; ++f) {
        const double2 v = *reinterpret_cast<const double2 *>(p + 8 * f);
        a[f][0] = v.x;
        a[f][1] = v.y;
    }
}
__device__ __forceinline__ void store_frags(double *T, int wr, const Frags &a)
{
    double *p = T + frag_at(wr);
#pragma unroll
    for (int f = 0; f < 8; ++f) *reinterpret_cast<double2 *>(p + 8 * f) = make_double2(a[f][0], a[f][1]);
}
// c += A B' for an 8 x 4 A and B fragment
__device__ __forceinline__ void mma4(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// The first N fragments of acc = Li Lj', summed over the 64 columns in order;
// the others 0.
template <int N>
__device__ __forceinline__ void product_n(const double *__restrict__ A, const double *__restrict__ B, Frags &acc)
{
#pragma unroll
    for (int f = 0; f < 8; ++f) acc[f][0] = acc[f][1] = 0.0;
#pragma unroll 4
    for (int p = 0; p < kNB; p += 4) {
        const double x = A[p];
#pragma unroll
        for (int f = 0; f < N; ++f) mma4(acc[f], x, B[8 * f * kTP + p]);
    }
}
// DIAG: only the lower fragments (f <= wr), in a loop of their own for each wr
// (a test per fragment in one loop keeps its loads from moving ahead of the
// products: 4,800 cycles for the two warps of a sub-partition).
template <bool DIAG>
__device__ __forceinline__ void tile_product(const double *__restrict__ Li, const double *__restrict__ Lj, int wr, Frags &acc)
{
    const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
    const double *A = Li + (8 * wr + lr) * kTP + lc, *B = Lj + lr * kTP + lc;
    if (!DIAG) return product_n<8>(A, B, acc);
    switch (wr) {
    case 0: return product_n<1>(A, B, acc);
    case 1: return product_n<2>(A, B, acc);
    case 2: return product_n<3>(A, B, acc);
    case 3: return product_n<4>(A, B, acc);
    case 4: return product_n<5>(A, B, acc);
    case 5: return product_n<6>(A, B, acc);
    case 6: return product_n<7>(A, B, acc);
    default: return product_n<8>(A, B, acc);
    }
}

// What a group of four columns c0 .. c0 + 3 is solved with: the reciprocal
// pivots and the block below the diagonal (its transpose lies above it).
struct Group {
    double r[4], l10, l20, l30, l21, l31, l32;
};
__device__ __forceinline__ void load_group(Group &G, const double *__restrict__ D)
{
    G.l10 = D[1];
    const double2 t = *reinterpret_cast<const double2 *>(D + 2), u = *reinterpret_cast<const double2 *>(D + kTP + 2);
    G.l20 = t.x;
    G.l30 = t.y;
    G.l21 = u.x;
    G.l31 = u.y;
    G.l32 = D[2 * kTP + 3];
}
// Four columns (half h of the fragment `own`) of X = A L^-T for the eight rows
// of a fragment row: a row's four lanes gather its four values, and all solve
// them.  Returns lane (lr, lc)'s operand element x(row lr, column c0 + lc).
__device__ __forceinline__ void gather4(const double (&own)[2], int h, double (&w)[4])
{
    const unsigned full = 0xffffffffu;
    const int from = (threadIdx.x & 28) + 2 * h;
    w[0] = __shfl_sync(full, own[0], from);
    w[1] = __shfl_sync(full, own[1], from);
    w[2] = __shfl_sync(full, own[0], from + 1);
    w[3] = __shfl_sync(full, own[1], from + 1);
}
__device__ __forceinline__ double solve4(double (&own)[2], int h, const double (&w)[4], const Group &G)
{
    const int odd = threadIdx.x & 1, high = threadIdx.x & 2, mine = (high >> 1) == h;
    const double w0 = w[0] * G.r[0];
    double w1 = fma(-w0, G.l10, w[1]), w2 = fma(-w0, G.l20, w[2]), w3 = fma(-w0, G.l30, w[3]);
    w1 = w1 * G.r[1];
    w2 = fma(-w1, G.l21, w2);
    w3 = fma(-w1, G.l31, w3);
    w2 = w2 * G.r[2];
    w3 = fma(-w2, G.l32, w3);
    w3 = w3 * G.r[3];
    own[0] = sel(mine, sel(odd, w2, w0), own[0]);
    own[1] = sel(mine, sel(odd, w3, w1), own[1]);
    return sel(high, sel(odd, w3, w2), sel(odd, w1, w0));
}
// Subtracts solved columns (x: operand elements) from the other half of their
// own fragment; b: L's element (row lr of the fragment, column c0 + lc).
__device__ __forceinline__ void other_half(double (&own)[2], int h, double x, double b)
{
    const int mine = ((int)(threadIdx.x & 3) >> 1) == h;
    double t[2] = {own[0], own[1]};
    mma4(t, -x, b);
    own[0] = sel(mine, own[0], t[0]);
    own[1] = sel(mine, own[1], t[1]);
}

// X = A L^-T for the tile held in fragments, L a factored diagonal tile in
// shared memory; each warp solves its own rows, so nothing is waited for.  In
// groups of four columns, each subtracted from the later ones as soon as it is
// solved: x(c) l(., c) in ascending order of c for every element.  The next
// group's columns come first; the others' products are issued after the next
// group's values have been gathered, so that they run under its solution
// instead of before it.
__device__ __forceinline__ void tile_solve(Frags &a, const double *__restrict__ L)
{
    const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
    const auto load = [&](Group &G, int c0) {
        const double *R = L + c0 * kTP + kNB;
#pragma unroll
        for (int k = 0; k < 4; ++k) G.r[k] = R[k * kTP];
        load_group(G, L + c0 * kTP + c0);
    };
    Group G[2];
    load(G[0], 0);
    double x = 0.0;
#pragma unroll
    for (int g = 0; g < 16; ++g) {
        const int f = g >> 1, h = g & 1, c0 = 4 * g;
        double w[4];
        gather4(a[f], h, w);
        if (g < 15) load(G[(g + 1) & 1], c0 + 4);
        if (g > 0) {  // the previous group's other fragments
#pragma unroll
            for (int k = f + 1; k < 8; ++k) mma4(a[k], -x, L[(8 * k + lr) * kTP + c0 - 4 + lc]);
        }
        x = solve4(a[f], h, w, G[g & 1]);
        if (g == 15) break;
        const double *B = L + lr * kTP + c0 + lc;
        if (h == 0) other_half(a[f], h, x, B[8 * f * kTP]);
        else mma4(a[f + 1], -x, B[8 * (f + 1) * kTP]);
    }
}

// Solves one row's 16 columns x (shared memory) against the 16 x 16 diagonal
// block at D (its transpose in the upper triangle, reciprocals at rd, pitch
// kTP): one thread per row, everything in registers, so a column costs a
// multiply and a multiply-add of latency instead of a shuffle between lanes.
__device__ __forceinline__ void solve_row16(double *x, const double *D, const double *rd)
{
    double v[16], r[16];
#pragma unroll
    for (int k = 0; k < 16; k += 2) {
        const double2 t = *reinterpret_cast<const double2 *>(x + k);
        v[k] = t.x;
        v[k + 1] = t.y;
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) r[c] = rd[c * kTP];
    double2 l[8], ln[8];  // row c of the transpose, and the next one on its way
#pragma unroll
    for (int k = 0; k < 8; ++k) l[k] = *reinterpret_cast<const double2 *>(D + 2 * k);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
#pragma unroll
        for (int k = (c + 2) >> 1; k < 8; ++k) ln[k] = *reinterpret_cast<const double2 *>(D + (c + 1) * kTP + 2 * k);
        v[c] = v[c] * r[c];
#pragma unroll
        for (int k = (c + 1) >> 1; k < 8; ++k) {
            if (2 * k > c) v[2 * k] = fma(-v[c], l[k].x, v[2 * k]);
            v[2 * k + 1] = fma(-v[c], l[k].y, v[2 * k + 1]);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) l[k] = ln[k];
    }
#pragma unroll
    for (int k = 0; k < 16; k += 2) *reinterpret_cast<double2 *>(x + k) = make_double2(v[k], v[k + 1]);
}

// Reciprocal square root of a pivot; one that is not positive is replaced by 1.
__device__ __forceinline__ double pivot_root(double &d, int &bad)
{
    const int ok = d > 0.0;
    bad |= ok ^ 1;
    d = sel(ok, d, 1.0);
    return rsqrt(d);
}

// Cholesky of a 16 x 16 block held by one warp as the fragments (0, 0), (1, 0),
// (1, 1).  Four columns at a time: every lane factors the 4 x 4 block on the
// diagonal for itself, so a pivot costs the chain a reciprocal square root, a
// product and a multiply-add and no shuffle, all rows are solved against it
// (times the reciprocal roots), and products subtract the four columns from the
// later ones.  Solved columns are stored above the diagonal of the block B in
// shared memory (transposed; what that puts below it is overwritten at the
// end) and announced on cols[q] (if any).  (2,080 cycles in a kernel of its own,
// 2,220 with one row per lane and a shuffle per column and element.)
__device__ __forceinline__ void factor16(double (&a)[3][2], int &bad, double *B, unsigned long long *cols)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
    double x[4][2];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int h = q & 1, c0 = 4 * q, fd = q < 2 ? 0 : 2, at = 18 * h;  // (lane of the 4 x 4 block's first element)
        double a00 = __shfl_sync(full, a[fd][0], at);
        double a10 = __shfl_sync(full, a[fd][0], at + 4), a11 = __shfl_sync(full, a[fd][1], at + 4);
        double a20 = __shfl_sync(full, a[fd][0], at + 8), a21 = __shfl_sync(full, a[fd][1], at + 8);
        double a30 = __shfl_sync(full, a[fd][0], at + 12), a31 = __shfl_sync(full, a[fd][1], at + 12);
        double a22 = __shfl_sync(full, a[fd][0], at + 9), a32 = __shfl_sync(full, a[fd][0], at + 13);
        double a33 = __shfl_sync(full, a[fd][1], at + 13);
        double w[2][4];  // each row's four values, rows of fragment row e
#pragma unroll
        for (int e = q < 2 ? 0 : 1; e < 2; ++e) gather4(a[q < 2 ? e : 2], h, w[e]);
        Group G;
        double p[4];
        G.r[0] = pivot_root(a00, bad);
        p[0] = a00 * G.r[0];
        G.l10 = a10 * G.r[0];
        G.l20 = a20 * G.r[0];
        G.l30 = a30 * G.r[0];
        a11 = fma(-G.l10, G.l10, a11);
        a21 = fma(-G.l20, G.l10, a21);
        a31 = fma(-G.l30, G.l10, a31);
        a22 = fma(-G.l20, G.l20, a22);
        a32 = fma(-G.l30, G.l20, a32);
        a33 = fma(-G.l30, G.l30, a33);
        G.r[1] = pivot_root(a11, bad);
        p[1] = a11 * G.r[1];
        G.l21 = a21 * G.r[1];
        G.l31 = a31 * G.r[1];
        a22 = fma(-G.l21, G.l21, a22);
        a32 = fma(-G.l31, G.l21, a32);
        a33 = fma(-G.l31, G.l31, a33);
        G.r[2] = pivot_root(a22, bad);
        p[2] = a22 * G.r[2];
        G.l32 = a32 * G.r[2];
        a33 = fma(-G.l32, G.l32, a33);
        G.r[3] = pivot_root(a33, bad);
        p[3] = a33 * G.r[3];
#pragma unroll
        for (int e = q < 2 ? 0 : 1; e < 2; ++e) {
            double w0 = w[e][0] * G.r[0];
            double w1 = fma(-w0, G.l10, w[e][1]), w2 = fma(-w0, G.l20, w[e][2]), w3 = fma(-w0, G.l30, w[e][3]);
            w1 = w1 * G.r[1];
            w2 = fma(-w1, G.l21, w2);
            w3 = fma(-w1, G.l31, w3);
            w2 = w2 * G.r[2];
            w3 = fma(-w2, G.l32, w3);
            w3 = w3 * G.r[3];
            if (e == fd >> 1) {  // the pivots themselves
                w0 = sel(lr == 4 * h, p[0], w0);
                w1 = sel(lr == 4 * h + 1, p[1], w1);
                w2 = sel(lr == 4 * h + 2, p[2], w2);
                w3 = sel(lr == 4 * h + 3, p[3], w3);
            }
            x[q][e] = sel(lc & 2, sel(lc & 1, w3, w2), sel(lc & 1, w1, w0));
            B[(c0 + lc) * kTP + 8 * e + lr] = x[q][e];
        }
        __syncwarp();
        if (cols) bar_arrive_lane0(cols + q);
        if (q == 0) {
            mma4(a[0], -x[0][0], x[0][0]);
            mma4(a[1], -x[0][1], x[0][0]);
        }
        if (q < 3) mma4(a[2], -x[q][1], x[q][1]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = q < 2 ? 0 : 1; e < 2; ++e)
            if (8 * e + lr > 4 * q + lc) B[(8 * e + lr) * kTP + 4 * q + lc] = x[q][e];
    __syncwarp();
}

// barriers of tile_potrf, each completed once per tile: four columns of panel
// P factored; rows 16 g .. of panel P solved (P < 2); block (i, j) has all its
// products subtracted
__device__ __forceinline__ int pot_cols(int P) { return 4 * P; }
__device__ __forceinline__ int pot_rows(int P, int g) { return 12 + 3 * P + g - 1; }
__device__ __forceinline__ int pot_block(int i, int j) { return i == 2 ? 16 + 2 * j : 17 + 2 * j - (j == 3); }

// block (i, j) -= its rows' and columns' parts of panel P (one warp)
__device__ __forceinline__ void block_update(double *__restrict__ W, int i, int j, int P)
{
    const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
    double acc[2][2][2] = {};
    const double *A = W + (16 * i + lr) * kTP + 16 * P + lc, *B = W + (16 * j + lr) * kTP + 16 * P + lc;
#pragma unroll
    for (int p = 0; p < 16; p += 4) {
        const double a0 = A[p], a1 = A[8 * kTP + p], b0 = B[p], b1 = B[8 * kTP + p];
        mma4(acc[0][0], a0, b0);
        mma4(acc[0][1], a0, b1);
        mma4(acc[1][0], a1, b0);
        mma4(acc[1][1], a1, b1);
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            double2 *c = reinterpret_cast<double2 *>(W + (16 * i + 8 * a + lr) * kTP + 16 * j + 8 * b + 2 * lc);
            double2 v = *c;
            v.x -= acc[a][b][0];
            v.y -= acc[a][b][1];
            *c = v;
        }
}

// Cholesky of the diagonal tile W (shared memory, lower triangle in; out: the
// factor, the transposes of its 16 x 16 diagonal blocks above them, the
// reciprocals in column 64), n tiles having been factored before.  Four panels
// of 16 columns.  Warp g < 4 owns the rows 16 g ..: it solves them against
// panel P < g while warp P is still factoring that panel, four columns behind,
// sums its own diagonal block's part of the last panel (P = g - 1) on the way,
// and so goes on to factor its own panel a few hundred cycles after the one
// before: the chain is 64 pivots and little else.  The products for the other
// blocks are warps 4 .. 7's.  A panel's product is summed over its 16 columns
// first, then subtracted.  (14,000 cycles: four times 2,650 in factor16 and
// three times 850 from one panel's last column to the next panel's first;
// 22,900 panel after panel, with barriers of all warps between factoring,
// solving and updating.)
__device__ __forceinline__ void tile_potrf(const Ctl &C, Smem &S, double *__restrict__ W, uint32_t n)
{
    const unsigned full = 0xffffffffu;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const auto wait = [&](int b) {
        bar_wait(C, S, &S.pot[b], n);
        __syncwarp();
    };
    const auto done = [&](int b) {
        __syncwarp();
        bar_arrive_lane0(&S.pot[b]);
    };
    if (warp < 4) {
        const int g = warp, l = lane & 15, lr = lane >> 2, lc = lane & 3;
        double s[3][2] = {};  // fragments (0, 0), (1, 0), (1, 1) of the diagonal block's part of the last panel
        double *const mine = W + (16 * g + lr) * kTP + 2 * lc;  // row lr, column 2 lc of the warp's rows
#pragma unroll 1
        for (int P = 0; P < g; ++P) {
            if (P > 0) wait(pot_block(g, P));
            double v[2][2][2];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double2 x = *reinterpret_cast<const double2 *>(mine + 8 * (e >> 1) * kTP + 16 * P + 8 * (e & 1));
                v[e >> 1][e & 1][0] = x.x;
                v[e >> 1][e & 1][1] = x.y;
            }
            const double *D = W + 16 * P * kTP + 16 * P;  // panel P's diagonal block, its transpose above
            const bool last = P == g - 1;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int f = q >> 1, h = q & 1, c0 = 4 * q;
                wait(pot_cols(P) + q);
                const double rl = 1.0 / D[(c0 + lc) * kTP + c0 + lc];
                double x[2];
                Group G;
                load_group(G, D + c0 * kTP + c0);
#pragma unroll
                for (int k = 0; k < 4; ++k) G.r[k] = __shfl_sync(full, rl, k);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    double w[4];
                    gather4(v[e][f], h, w);
                    x[e] = solve4(v[e][f], h, w, G);
                }
                const double *B = D + (c0 + lc) * kTP + lr;  // (L's elements from their transpose)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (h == 0) other_half(v[e][f], h, x[e], B[8 * f]);
                    if (f == 0) mma4(v[e][1], -x[e], B[8]);
                }
                if (last) {  // (a product's second operand is held as its first)
                    mma4(s[0], x[0], x[0]);
                    mma4(s[1], x[1], x[0]);
                    mma4(s[2], x[1], x[1]);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                *reinterpret_cast<double2 *>(mine + 8 * (e >> 1) * kTP + 16 * P + 8 * (e & 1)) =
                    make_double2(v[e >> 1][e & 1][0], v[e >> 1][e & 1][1]);
            if (P < 2) done(pot_rows(P, g));
        }
        if (g >= 2) wait(pot_block(g, g));
        double d[3][2];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const double2 x = *reinterpret_cast<const double2 *>(mine + (e > 0 ? 8 * kTP : 0) + 16 * g + (e > 1 ? 8 : 0));
            d[e][0] = x.x - s[e][0];
            d[e][1] = x.y - s[e][1];
        }
        __syncwarp();
        int bad = 0;
        factor16(d, bad, W + 16 * g * kTP + 16 * g, g < 3 ? &S.pot[pot_cols(g)] : nullptr);
        if (bad && lane == 0) atomicOr(C.status, kStNotSPD);
        double *row = W + (16 * g + l) * kTP;
        if (lane < 16) row[kNB] = 1.0 / row[16 * g + l];
    } else if (warp == 4) {
        wait(pot_rows(0, 1));
        wait(pot_rows(0, 2));
        block_update(W, 2, 1, 0);
        done(pot_block(2, 1));
        wait(pot_rows(0, 3));
        block_update(W, 3, 2, 0);
        wait(pot_rows(1, 2));
        wait(pot_rows(1, 3));
        block_update(W, 3, 2, 1);
        done(pot_block(3, 2));
    } else if (warp == 5) {
        wait(pot_rows(0, 1));
        wait(pot_rows(0, 3));
        block_update(W, 3, 1, 0);
        done(pot_block(3, 1));
    } else if (warp == 6) {
        wait(pot_rows(0, 2));
        block_update(W, 2, 2, 0);
        done(pot_block(2, 2));
    } else {
        wait(pot_rows(0, 3));
        block_update(W, 3, 3, 0);
        wait(pot_rows(1, 3));
        block_update(W, 3, 3, 1);
        done(pot_block(3, 3));
    }
    sync_compute();
}

// ------------------------------------------------------------------ chain

// The chain's buffers: 0, 1 the next step's tiles (k, k-1) and (k, k), 2 the
// diagonal tile being factored, 5 the solved panel tile.  The back
// substitution then uses all six as one ring.
constexpr int kBufX = 0, kBufD = 1, kBufW = 2, kBufOut = 5;

// The ring of the back substitution: per block kb, in order, the tiles
// (kb+1, kb) and (kb, kb) of the chain warps and (kb+2, kb-1), (kb+1, kb-1)
// of the look-ahead warps, as far as they exist.
__device__ __forceinline__ bool back_tile(const Ctl &C, int kb, int which, const double *&p)
{
    int i, j;
    if (which == 0) { i = kb + 1; j = kb; }
    else if (which == 1) { i = kb; j = kb; }
    else if (which == 2) { i = kb + 2; j = kb - 1; }
    else { i = kb + 1; j = kb - 1; }
    if (i >= C.nblk || j < 0) return false;
    p = tile_ptr(C, i, j);
    return true;
}

__device__ void chain_fetch(const Ctl &C, Smem &S)
{
    const int nblk = C.nblk;
    for (int k = 1; k < nblk; ++k) {
        const uint32_t n = (uint32_t)(k - 1);
        if (k >= 2 && !flag_wait(C, S, &C.pre_s[k - 1], 1)) return;
        if (!claim_buf(C, S, &S.empty[kBufX], n)) return;
        fence_async();
        load_buf(S, kBufX, tile_ptr(C, k, k - 1), kTileB);
        if (k >= 2 && !flag_wait(C, S, &C.pre_d[k], 1)) return;
        if (!claim_buf(C, S, &S.empty[kBufD], n)) return;
        fence_async();
        load_buf(S, kBufD, tile_ptr(C, k, k), kTileB);
    }
    // back substitution: every panel tile of a row of right-hand sides that
    // is final has been published, and so have the tiles it was solved with;
    // the ring starts once the chain's own last tiles have left the buffers
    if (!flag_wait(C, S, &C.F->pdone, nblk) || !flag_wait(C, S, &C.tdone[nblk], nblk)) return;
    bar_wait(C, S, &S.xdone, 0);
    if (*reinterpret_cast<volatile int *>(&S.abort)) return;
    fence_async();
    uint32_t q = 0;  // position in the ring
    uint32_t used[kBufs];
#pragma unroll
    for (int b = 0; b < kBufs; ++b) used[b] = (b == kBufX || b == kBufD) && nblk > 1 ? (uint32_t)(nblk - 1) : 0u;
    int zb = nblk - 1;  // next block whose right-hand sides are fetched
    for (int kb = nblk - 1; kb >= 0; --kb) {
        // the right-hand sides of block kb - 1 (and, at the start, kb) join;
        // their slot's last user, block kb + 3, is done: the tiles fetched so
        // far are all of blocks > kb, so two blocks' worth of the ring's six
        // buffers, those of block kb + 2 at least, have been released
        for (; zb >= 0 && zb >= kb - 1; --zb) {
            if (zb + 4 < nblk && !flag_wait(C, S, &C.bcnt[zb], 1)) return;
            fence_async();
            bar_expect(&S.zfull[zb & 3], kRhsB);
            bulk_copy(S.z[zb & 3], C.rhs + (size_t)zb * kRhsD, kRhsB, &S.zfull[zb & 3]);
            ++S.zissued[zb & 3];
        }
        for (int w = 0; w < 4; ++w) {
            const double *src;
            if (!back_tile(C, kb, w, src)) continue;
            const int b = (int)(q % kBufs);
            // (constant indices keep `used` in registers)
            uint32_t u = 0;
#pragma unroll
            for (int k = 0; k < kBufs; ++k)
                if (k == b) u = used[k]++;
            if (!claim_buf(C, S, &S.empty[b], u)) return;
            load_buf(S, b, src, kTileB);
            ++q;
        }
    }
}

// Back substitution of one 64-row block for one right-hand side by one warp:
// D' x = b, lane l holding rows l and l + 32.  A row's update is a product
// with 0 in the lanes it does not concern, so that the chain per row is one
// shuffle, one product and one multiply-add without a select.
__device__ __forceinline__ void back_diag(const double *__restrict__ D, double &b0, double &b1)
{
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    double x0 = 0.0, x1 = 0.0;
#pragma unroll 16
    for (int j = kNB - 1; j >= 32; --j) {
        const double rd = D[j * kTP + kNB], d0 = -D[j * kTP + lane], d1 = sel(lane + 32 < j, -D[j * kTP + lane + 32], 0.0);
        const double xj = __shfl_sync(full, b1, j & 31) * rd;
        x1 = sel(lane == (j & 31), xj, x1);
        b1 = fma(d1, xj, b1);
        b0 = fma(d0, xj, b0);
    }
#pragma unroll 16
    for (int j = 31; j >= 0; --j) {
        const double rd = D[j * kTP + kNB], d0 = sel(lane < j, -D[j * kTP + lane], 0.0);
        const double xj = __shfl_sync(full, b0, j) * rd;
        x0 = sel(lane == j, xj, x0);
        b0 = fma(d0, xj, b0);
    }
    b0 = x0;
    b1 = x1;
}

// s0, s1: rows `lane` and `lane + 32` of L' x for a tile L and 64 values x in
// shared memory, summed over L's rows in order.
__device__ __forceinline__ void back_product(const double *__restrict__ L, const double *__restrict__ x, double &s0, double &s1)
{
    const int lane = threadIdx.x & 31;
    s0 = s1 = 0.0;
#pragma unroll 8
    for (int p = 0; p < kNB; p += 2) {
        const double2 xp = *reinterpret_cast<const double2 *>(x + p);
        s0 = fma(L[p * kTP + lane], xp.x, s0);
        s1 = fma(L[p * kTP + lane + 32], xp.x, s1);
        s0 = fma(L[(p + 1) * kTP + lane], xp.y, s0);
        s1 = fma(L[(p + 1) * kTP + lane + 32], xp.y, s1);
    }
}

__device__ __forceinline__ void chain_compute(const Ctl &C, Smem &S)
{
    const int t = threadIdx.x, warp = warp_index(), lane = t & 31, wr = row_block();
    const int nblk = C.nblk;
    double *W = S.buf[kBufW], *Xs = S.buf[kBufOut];
    for (int k = 0; k < nblk; ++k) {
        if (k == 0) {
            const double *src = tile_ptr(C, 0, 0);
            for (int e = t; e < kTileD / 2; e += kCompute)
                reinterpret_cast<double2 *>(W)[e] = reinterpret_cast<const double2 *>(src)[e];
        } else {
            const uint32_t n = (uint32_t)(k - 1);
            Frags a, acc;
            bar_wait(C, S, &S.full[kBufX], n);
            load_frags(S.buf[kBufX], wr, a);
            __syncwarp();
            bar_arrive_lane0(&S.empty[kBufX]);
            tile_solve(a, W);
            bar_wait_free(C, S, &S.freed[0], n);  // the previous panel tile has been stored
            store_frags(Xs, wr, a);
            sync_compute();  // (and every warp has read W)
            post(S, 0, Xs, tile_ptr(C, k, k - 1), kTileB, &C.tdone[k], k);
            tile_product<true>(Xs, Xs, wr, acc);
            bar_wait(C, S, &S.full[kBufD], n);
            load_frags(S.buf[kBufD], wr, a);
            __syncwarp();
            bar_arrive_lane0(&S.empty[kBufD]);
#pragma unroll
            for (int f = 0; f < 8; ++f) {
                a[f][0] -= acc[f][0];
                a[f][1] -= acc[f][1];
            }
            bar_wait(C, S, &S.freed[1], n);  // the previous diagonal tile has been stored
            store_frags(W, wr, a);           // (what is above the diagonal is not read)
        }
        sync_compute();
        tile_potrf(C, S, W, (uint32_t)k);
        post(S, 1, W, tile_ptr(C, k, k), kTileB, &C.F->pdone, k + 1);
    }
    // back substitution: the fetching warp may overwrite every buffer once
    // the last two results have been stored
    bar_wait(C, S, &S.freed[1], (uint32_t)(nblk - 1));
    if (nblk > 1) bar_wait(C, S, &S.freed[0], (uint32_t)(nblk - 2));
    sync_compute();
    if (t == 0) bar_arrive(&S.xdone);
    const int c = warp & 3;         // right-hand side
    const bool head = warp < 4;     // the chain itself; the others look ahead
    uint32_t q = 0;
    uint32_t used[kBufs];
#pragma unroll
    for (int b = 0; b < kBufs; ++b) used[b] = (b == kBufX || b == kBufD) && nblk > 1 ? (uint32_t)(nblk - 1) : 0u;
    for (int kb = nblk - 1; kb >= 0; --kb) {
        double s0, s1, b0 = 0, b1 = 0;
        if (head) {
            bar_wait(C, S, &S.zfull[kb & 3], (uint32_t)((nblk - 1 - kb) >> 2));
            b0 = S.z[kb & 3][c * kTP + lane];
            b1 = S.z[kb & 3][c * kTP + lane + 32];
        } else if (kb >= 1) {
            bar_wait(C, S, &S.zfull[(kb - 1) & 3], (uint32_t)((nblk - kb) >> 2));
            b0 = S.z[(kb - 1) & 3][c * kTP + lane];
            b1 = S.z[(kb - 1) & 3][c * kTP + lane + 32];
        }
#pragma unroll 1
        for (int w = 0; w < 4; ++w) {
            const double *src;
            if (!back_tile(C, kb, w, src)) continue;
            const int b = (int)(q % kBufs);
            uint32_t u = 0;
#pragma unroll
            for (int k = 0; k < kBufs; ++k)
                if (k == b) u = used[k]++;
            ++q;
            if (head == (w < 2)) {
                bar_wait(C, S, &S.full[b], u);
                if (w == 1) {
                    back_diag(S.buf[b], b0, b1);
                } else {
                    back_product(S.buf[b], S.xs[(w == 2 ? kb + 2 : kb + 1) & 3] + c * kTP, s0, s1);
                    b0 -= s0;
                    b1 -= s1;
                }
            }
            __syncwarp();
            bar_arrive_lane0(&S.empty[b]);
        }
        if (head) {
            S.xs[kb & 3][c * kTP + lane] = b0;
            S.xs[kb & 3][c * kTP + lane + 32] = b1;
            const int r = kb * kNB + lane;
            if (r < C.m) C.x[(size_t)r * 4 + c] = b0;
            if (r + 32 < C.m) C.x[(size_t)(r + 32) * 4 + c] = b1;
        } else if (kb >= 1) {
            S.z[(kb - 1) & 3][c * kTP + lane] = b0;
            S.z[(kb - 1) & 3][c * kTP + lane + 32] = b1;
        }
        // the previous block's mail has been read (mailbox 0 carried nblk - 1 panel tiles before)
        bar_wait_free(C, S, &S.freed[0], (uint32_t)(nblk - 1 + nblk - 1 - kb));
        post(S, 0, nullptr, nullptr, 0, &C.F->ddone, nblk - kb);
        sync_compute();
    }
}

__device__ void chain_publish(const Ctl &C, Smem &S)
{
    uint32_t n0 = 0;
    if (!publish(C, S, 1, 0)) return;
    for (int k = 1; k < C.nblk; ++k) {
        if (!publish(C, S, 0, n0++)) return;
        if (!publish(C, S, 1, (uint32_t)k)) return;
    }
    for (int kb = C.nblk - 1; kb >= 0; --kb)
        if (!publish(C, S, 0, n0++)) return;
}

// ---------------------------------------------------------------- helpers

// Task t: tiles column by column, rows j .. nblk (nblk: the right-hand
// sides), then the right-hand-side blocks nblk - 5 .. 0 of the back
// substitution.  kind 0: none left.
struct Task {
    int kind;  // 1 tile, 2 right-hand sides of a column, 3 back substitution
    int i, j;
};

__device__ Task task_of(int t, int nblk)
{
    for (int j = 0; j < nblk; ++j) {
        const int n = nblk + 1 - j;
        if (t < n) return {t == n - 1 ? 2 : 1, j + t, j};
        t -= n;
    }
    if (t < nblk - 4) return {3, nblk - 5 - t, 0};
    return {0, 0, 0};
}

// Ring of the helpers: two stages of two buffers (0, 1 and 2, 3); buffer 4 the
// factored diagonal tile, 5 the result.
constexpr int kBufL = 4;

__device__ void helper_fetch(const Ctl &C, Smem &S, const Task &T, uint32_t &stage, uint32_t &diags)
{
    const int nblk = C.nblk;
    if (T.kind == 3) {
        // L(kb, i) needs no wait of its own: once x(kb) is asked for, the
        // factorisation is over; the first wait covers them all
        for (int kb = nblk - 1; kb >= T.i + 4; --kb) {
            const int b = 2 * (int)(stage & 1u);
            if (kb == nblk - 1 && (!flag_wait(C, S, &C.F->pdone, nblk) || !flag_wait(C, S, &C.tdone[nblk], nblk))) return;
            if (!claim_buf(C, S, &S.empty[b], stage >> 1)) return;
            fence_async();
            load_buf(S, b, tile_ptr(C, kb, T.i), kTileB);
            ++stage;
        }
        return;
    }
    const int kn = T.kind == 1 && T.i == T.j ? T.j - 1 : T.j;
    int ready = 0;  // panels known to be final
    for (int k = 0; k < kn; ++k, ++stage) {
        const int b = 2 * (int)(stage & 1u);
        if (ready <= k) {
            if (!flag_wait(C, S, &C.tdone[T.j], k + 1) || !flag_wait(C, S, &C.tdone[T.kind == 2 ? nblk : T.i], k + 1)) return;
            ready = min(ld_acquire(&C.tdone[T.j]), ld_acquire(&C.tdone[T.kind == 2 ? nblk : T.i]));
        }
        if (!claim_buf(C, S, &S.empty[b], stage >> 1)) return;
        fence_async();
        const bool two = T.kind == 2 || T.i != T.j;
        // both operands count on the first buffer's barrier
        ++S.issued[b];
        bar_expect(&S.full[b], T.kind == 2 ? kTileB + kRhsB : two ? 2 * kTileB : kTileB);
        bulk_copy(S.buf[b], tile_ptr(C, T.j, k), kTileB, &S.full[b]);
        if (T.kind == 2) bulk_copy(S.buf[b + 1], C.rhs + (size_t)k * kRhsD, kRhsB, &S.full[b]);
        else if (two) bulk_copy(S.buf[b + 1], tile_ptr(C, T.i, k), kTileB, &S.full[b]);
    }
    if (T.kind == 2 || T.i > T.j + 1) {
        if (!flag_wait(C, S, &C.F->pdone, T.j + 1)) return;
        if (!claim_buf(C, S, &S.empty[kBufL], diags)) return;
        fence_async();
        load_buf(S, kBufL, tile_ptr(C, T.j, T.j), kTileB);
        ++diags;
    }
}

__device__ __forceinline__ void helper_compute(const Ctl &C, Smem &S, const Task &T, uint32_t &stage, uint32_t &diags, uint32_t &posts)
{
    const int t = threadIdx.x, lane = t & 31, wr = row_block();
    const int nblk = C.nblk;
    double *Xs = S.buf[kBufOut];
    if (T.kind == 1) {
        const bool diag = T.i == T.j;
        const int kn = diag ? T.j - 1 : T.j;
        if (kn <= 0 && T.i <= T.j + 1) return;  // the chain reads the tile as it is
        double *A = tile_ptr(C, T.i, T.j);
        Frags a, acc;
        load_frags(A, wr, a);
        for (int k = 0; k < kn; ++k, ++stage) {
            const int b = 2 * (int)(stage & 1u);
            bar_wait(C, S, &S.full[b], stage >> 1);
            if (diag) tile_product<true>(S.buf[b], S.buf[b], wr, acc);
            else tile_product<false>(S.buf[b + 1], S.buf[b], wr, acc);
            __syncwarp();
            bar_arrive_lane0(&S.empty[b]);
#pragma unroll
            for (int f = 0; f < 8; ++f) {
                a[f][0] -= acc[f][0];
                a[f][1] -= acc[f][1];
            }
        }
        const bool solved = T.i > T.j + 1;
        if (solved) {
            bar_wait(C, S, &S.full[kBufL], diags++);
            tile_solve(a, S.buf[kBufL]);
            __syncwarp();
            bar_arrive_lane0(&S.empty[kBufL]);
        }
        bar_wait_free(C, S, &S.freed[0], posts);
        store_frags(Xs, wr, a);
        post(S, 0, Xs, A, kTileB, solved ? &C.tdone[T.i] : diag ? &C.pre_d[T.j] : &C.pre_s[T.j], solved ? T.j + 1 : 1);
        ++posts;
        return;
    }
    // four right-hand sides: thread (c, r), r = t / 64 the side, c = t % 64
    const int r = t >> 6, c = t & 63;
    if (T.kind == 2) {
        double *A = C.rhs + (size_t)T.j * kRhsD;
        double a = A[r * kTP + c];
        for (int k = 0; k < T.j; ++k, ++stage) {
            const int b = 2 * (int)(stage & 1u);
            bar_wait(C, S, &S.full[b], stage >> 1);
            const double *Li = S.buf[b + 1] + r * kTP, *Lj = S.buf[b] + c * kTP;
            double s = 0.0;
#pragma unroll 8
            for (int p = 0; p < kNB; p += 2) {
                const double2 x = *reinterpret_cast<const double2 *>(Li + p), y = *reinterpret_cast<const double2 *>(Lj + p);
                s = fma(x.y, y.y, fma(x.x, y.x, s));
            }
            __syncwarp();
            bar_arrive_lane0(&S.empty[b]);
            a -= s;
        }
        bar_wait_free(C, S, &S.freed[0], posts);
        bar_wait(C, S, &S.full[kBufL], diags++);
        const double *L = S.buf[kBufL];
        for (int c0 = 0; c0 < kNB; c0 += 16) {
            if (c >= c0 && c < c0 + 16) Xs[r * kTP + c] = a;
            sync_compute();
            if (t < 4) solve_row16(Xs + t * kTP + c0, L + c0 * kTP + c0, L + c0 * kTP + kNB);
            sync_compute();
            if (c >= c0 + 16)
#pragma unroll
                for (int p = c0; p < c0 + 16; p += 2) {
                    const double2 x = *reinterpret_cast<const double2 *>(Xs + r * kTP + p);
                    const double2 l = *reinterpret_cast<const double2 *>(L + c * kTP + p);
                    a = fma(-x.y, l.y, fma(-x.x, l.x, a));
                }
        }
        if (t < 16) Xs[(t >> 2) * kTP + kNB + (t & 3)] = 0.0;  // the pitch's spare columns
        __syncwarp();
        bar_arrive_lane0(&S.empty[kBufL]);
        post(S, 0, Xs, A, kRhsB, &C.tdone[nblk], T.j + 1);
        ++posts;
        return;
    }
    // back substitution of block i by the blocks nblk - 1 .. i + 4
    double *A = C.rhs + (size_t)T.i * kRhsD;
    bool first = true;
    double a = 0.0;
    for (int kb = nblk - 1; kb >= T.i + 4; --kb, ++stage) {
        const int b = 2 * (int)(stage & 1u);
        if (t == 0) flag_wait(C, S, &C.F->ddone, nblk - kb);
        sync_compute();
        if (first) a = __ldcg(&A[r * kTP + c]);
        first = false;
        S.small[r * kTP + c] = kb * kNB + c < C.m ? __ldcg(&C.x[(size_t)(kb * kNB + c) * 4 + r]) : 0.0;
        sync_compute();
        bar_wait(C, S, &S.full[b], stage >> 1);
        const double *L = S.buf[b] + c, *x = S.small + r * kTP;
        double s = 0.0;
#pragma unroll 8
        for (int p = 0; p < kNB; p += 2) {
            const double2 xp = *reinterpret_cast<const double2 *>(x + p);
            s = fma(L[p * kTP], xp.x, s);
            s = fma(L[(p + 1) * kTP], xp.y, s);
        }
        __syncwarp();
        bar_arrive_lane0(&S.empty[b]);
        a -= s;
    }
    bar_wait_free(C, S, &S.freed[0], posts);
    Xs[r * kTP + c] = a;
    if (t < 16) Xs[(t >> 2) * kTP + kNB + (t & 3)] = 0.0;
    post(S, 0, Xs, A, kRhsB, &C.bcnt[T.i], 1);
    ++posts;
}

// Waits (bounded) for the last of `n` copies counted on barrier b.
__device__ void drain(unsigned long long *b, uint32_t n)
{
    if (n == 0) return;
    const unsigned long long t0 = now_ns();
    while (!bar_try(b, (n - 1) & 1u))
        if (now_ns() - t0 > 2000000000ull) return;
}

__global__ void __launch_bounds__(kThreads, 1) k_chol_solve(const __grid_constant__ Ctl C)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem &S = *reinterpret_cast<Smem *>(smem_raw);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int b = 0; b < kBufs; ++b) {
            bar_init(&S.full[b], 1);
            bar_init(&S.empty[b], kCompute / 32);
            S.issued[b] = 0;
        }
        for (int b = 0; b < 4; ++b) {
            bar_init(&S.zfull[b], 1);
            S.zissued[b] = 0;
        }
        for (int b = 0; b < 2; ++b) {
            bar_init(&S.post[b], kCompute / 32);
            bar_init(&S.freed[b], 1);
        }
        bar_init(&S.xdone, 1);
        for (int b = 0; b < kPotBars; ++b) bar_init(&S.pot[b], 1);
        S.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (blockIdx.x == 0) {  // (the fetching and publishing warps' lanes meet again at the __syncwarp below)
        if (warp < kFetchWarp) chain_compute(C, S);
        else if (lane == 0) {
            if (warp == kFetchWarp) chain_fetch(C, S);
            else chain_publish(C, S);
        }
    } else {
        uint32_t stage = 0, diags = 0, posts = 0;
        bool live = true;  // the publishing warp: its mailbox is still in use
        for (;;) {
            if (threadIdx.x == 0)
                S.task = *reinterpret_cast<volatile int *>(&S.abort) ? 0x7fffffff : atomicAdd(&C.F->next, 1);
            __syncthreads();
            const Task T = task_of(S.task, C.nblk);
            __syncthreads();  // every thread has read the task
            if (T.kind == 0) break;
            if (warp < kFetchWarp) helper_compute(C, S, T, stage, diags, posts);
            else if (lane == 0) {
                if (warp == kFetchWarp) {
                    helper_fetch(C, S, T, stage, diags);
                } else {
                    const int kn = T.kind == 1 ? (T.i == T.j ? T.j - 1 : T.j) : 1;
                    const bool posted = !(T.kind == 1 && kn <= 0 && T.i <= T.j + 1);
                    if (posted && live) live = publish(C, S, 0, posts++);
                }
            }
            __syncwarp();
        }
    }
    // no copy may still be writing this CTA's shared memory when it exits: on
    // the normal path every copy has been waited for; after a time-out the
    // thread that began them waits here (bounded)
    if (warp == kFetchWarp && lane == 0) {
        for (int b = 0; b < kBufs; ++b) drain(&S.full[b], S.issued[b]);
        for (int b = 0; b < 4; ++b) drain(&S.zfull[b], S.zissued[b]);
    }
    __syncwarp();
    __syncthreads();
}

// Tile (i, j), i >= j, of (Q'KQ)(4:,4:) + lambda I (lower triangle; rows and
// columns past m zero, with ones on the diagonal), or the right-hand-side tile
// j, z(4:)'.  kFillParts CTAs per tile, 256 threads: a thread keeps its
// column's landmark and vectors in registers and takes a few rows, whose own
// come from shared memory.
constexpr int kFillParts = 4;
__global__ void __launch_bounds__(256) k_fill_tiles(const double *__restrict__ ctr, int n, const double *__restrict__ V,
                                                    const double *__restrict__ W, const double *__restrict__ Z,
                                                    double lambda, Ctl C)
{
    constexpr int ROWS = kNB / kFillParts;
    __shared__ double row[ROWS][11];
    const int m = C.m, nblk = C.nblk;
    const int ntri = nblk * (nblk + 1) / 2;
    int t = (int)blockIdx.x / kFillParts;
    const int part = (int)blockIdx.x % kFillParts;
    if (t >= ntri) {
        const int j = t - ntri;
        double *R = C.rhs + (size_t)j * kRhsD;
        if (part == 0)
            for (int e = threadIdx.x; e < kRhsD; e += blockDim.x) {
                const int r = e / kTP, c = j * kNB + e % kTP;
                R[e] = e % kTP < kNB && c < m ? Z[(size_t)(c + 4) * 4 + r] : 0.0;
            }
        return;
    }
    int j = 0;
    while (t >= nblk - j) {
        t -= nblk - j;
        ++j;
    }
    const int i = j + t, r0 = part * ROWS;
    for (int e = threadIdx.x; e < ROWS * 11; e += blockDim.x) {
        const int q = e % 11, g = min(i * kNB + r0 + e / 11, m - 1) + 4;
        row[e / 11][q] = q < 3 ? ctr[3 * g + q] : q < 7 ? V[4 * g + q - 3] : W[4 * g + q - 7];
    }
    const int c = threadIdx.x & (kNB - 1), cj = j * kNB + c, gj = min(cj, m - 1) + 4;
    const double x = ctr[3 * gj], y = ctr[3 * gj + 1], z = ctr[3 * gj + 2];
    double vj[4], wj[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        vj[k] = V[gj * 4 + k];
        wj[k] = W[gj * 4 + k];
    }
    __syncthreads();
    double *T = tile_ptr(C, i, j);
    for (int r = threadIdx.x / kNB; r < ROWS; r += 256 / kNB) {
        const int ri = i * kNB + r0 + r;
        const double *q = row[r];
        double v = 0.0;
        if (ri < m && cj < m && ri >= cj) {
            v = kdist(q[0], q[1], q[2], x, y, z);
#pragma unroll
            for (int k = 0; k < 4; ++k) v -= q[3 + k] * wj[k] + q[7 + k] * vj[k];
            if (ri == cj) v += lambda;
        } else if (ri == cj) {
            v = 1.0;
        }
        T[(r0 + r) * kTP + c] = v;
        if (c < kTP - kNB) T[(r0 + r) * kTP + kNB + c] = 0.0;
    }
}

int blocks_of(int m) { return (m + kNB - 1) / kNB; }
size_t flag_ints(int nblk) { return 4 + (size_t)(nblk + 1) + 3 * (size_t)nblk; }
size_t tri_tiles(int nblk) { return (size_t)nblk * (nblk + 1) / 2; }

}  // namespace

size_t chol_work_bytes(int m)
{
    const int nblk = blocks_of(m);
    return tri_tiles(nblk) * kTileB + (size_t)nblk * kRhsB + ((flag_ints(nblk) * sizeof(int) + 15) / 16) * 16;
}

cudaError_t launch_chol_solve(const double *ctr, int n, const double *V, const double *W, double *Z, double lambda,
                              void *work, int *status, unsigned long long limit_ns, int sm_count, cudaStream_t st)
{
    Ctl C;
    C.m = n - 4;
    C.nblk = blocks_of(C.m);
    C.tiles = static_cast<double *>(work);
    C.rhs = C.tiles + tri_tiles(C.nblk) * kTileD;
    int *flags = reinterpret_cast<int *>(C.rhs + (size_t)C.nblk * kRhsD);
    C.F = reinterpret_cast<Flags *>(flags);
    C.tdone = flags + 4;
    C.pre_d = C.tdone + C.nblk + 1;
    C.pre_s = C.pre_d + C.nblk;
    C.bcnt = C.pre_s + C.nblk;
    C.x = Z + 16;
    C.status = status;
    C.limit_ns = limit_ns;
    cudaError_t e = cudaMemsetAsync(flags, 0, flag_ints(C.nblk) * sizeof(int), st);
    if (e != cudaSuccess) return e;
    const size_t fill = tri_tiles(C.nblk) + (size_t)C.nblk;
    k_fill_tiles<<<(unsigned)(fill * kFillParts), 256, 0, st>>>(ctr, n, V, W, Z, lambda, C);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_chol_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
    if (e != cudaSuccess) return e;
    // the chain and at most one helper per task: a small system leaves the
    // other SMs to other work
    const size_t want = 1 + fill;
    const int grid = want < (size_t)sm_count ? (int)want : sm_count;
    void *args[] = {(void *)&C};
    return cudaLaunchCooperativeKernel((const void *)k_chol_solve, dim3(grid), dim3(kThreads), args, sizeof(Smem), st);
}

}  // namespace tw
