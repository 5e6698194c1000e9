// tw_jobs.cu -- resample job construction and launch, sample-hull kernels for
// footprint planning, the parameter-surface matrices, and the slab pipeline
// that streams host volumes through HBM with H2D / compute / D2H overlapped.
#include "tw_host.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <deque>

namespace tw {

RJob tps_job(const void *src, const int64_t src_sz[3], void *dst, const int64_t dst_sz[3], const float4 *nodes, int g,
             int dtype, int interp)
{
    RJob j;
    std::memset(&j, 0, sizeof(j));
    j.src = src;
    j.dst = dst;
    j.nodes = nodes;
    j.src_py = src_sz[0];
    j.src_pz = src_sz[0] * src_sz[1];
    j.dst_py = dst_sz[0];
    j.dst_pz = dst_sz[0] * dst_sz[1];
    for (int a = 0; a < 3; ++a) {
        j.src_o[a] = 0;
        j.src_n[a] = src_sz[a];
        j.glob[a] = src_sz[a];
        j.out_o[a] = 0;
        j.out_n[a] = dst_sz[a];
        j.gsz[a] = grid_size(dst_sz[a], g);
    }
    j.g = g;
    j.dtype = dtype;
    j.kind = 1;
    j.interp = interp;
    return j;
}

RJob affine_job(const void *src, const int64_t src_sz[3], void *dst, const int64_t dst_sz[3], const double M[16],
                int dtype, int interp)
{
    RJob j;
    std::memset(&j, 0, sizeof(j));
    j.src = src;
    j.dst = dst;
    j.src_py = src_sz[0];
    j.src_pz = src_sz[0] * src_sz[1];
    j.dst_py = dst_sz[0];
    j.dst_pz = dst_sz[0] * dst_sz[1];
    for (int a = 0; a < 3; ++a) {
        j.src_o[a] = 0;
        j.src_n[a] = src_sz[a];
        j.glob[a] = src_sz[a];
        j.out_o[a] = 0;
        j.out_n[a] = dst_sz[a];
    }
    for (int i = 0; i < 12; ++i) j.M[i] = M[i];
    j.g = 0;
    j.dtype = dtype;
    j.kind = 0;
    j.interp = interp;
    return j;
}

namespace {

// A stream-ordered pool block returned on its stream when the scope ends.
struct StreamBlock {
    tw_ctx *ctx = nullptr;
    cudaStream_t st = nullptr;
    void *p = nullptr;
    size_t bytes = 0;
    ~StreamBlock() { if (p) dfree_on(ctx, p, bytes, st); }
};

// A small block of the context's pool outside its budget.
struct PoolBlock {
    cudaStream_t st = nullptr;
    void *p = nullptr;
    ~PoolBlock() { if (p) cudaFreeAsync(p, st); }
};

}  // namespace

namespace {

tw_status run_group(tw_ctx *ctx, RJob *jobs, int njobs, uint32_t affine_box, cudaStream_t st);

// Copies the sources of those jobs of [first, end) that gain by it into rows
// padded to 16 bytes (one block, `copy`), moves these jobs to the front and
// returns their end.  A small launch gathers in the same or less time (517 x
// 389 x 203 uint16: 367 us gathered, 370 copied and staged; 801 x 601 x 301:
// 1091 and 850), and the copies are held to 256 MiB, which the context's pool
// then keeps, and to what the budget has left.
RJob *pad_sources(tw_ctx *ctx, RJob *first, RJob *end, StreamBlock &copy, cudaStream_t st, size_t most)
{
    constexpr int64_t kMinVoxels = 48 << 20;
    const size_t most_bytes = std::min((size_t)256 << 20, most);
    int64_t vox = 0;
    size_t bytes = 0;
    const auto row_bytes = [](const RJob &j) { return (size_t)((j.src_n[0] * (j.dtype == TW_U8 ? 1 : 2) + 15) / 16 * 16); };
    const auto size = [&](const RJob &j) { return (row_bytes(j) * (size_t)(j.src_n[1] * j.src_n[2]) + 255) / 256 * 256; };
    RJob *const last = std::stable_partition(first, end, [&](const RJob &j) {
        const int64_t out = j.out_n[0] * j.out_n[1] * j.out_n[2];
        if (j.arriving) return false;  // (the copy would read all of it)
        if (j.src_n[0] < kStageBoxW || j.src_n[1] < kStageBoxH || j.src_n[2] < 2 || bytes + size(j) > most_bytes) return false;
        if (2 * out < j.src_n[0] * j.src_n[1] * j.src_n[2]) return false;  // (a slab: the copy takes the whole source)
        bytes += size(j);
        vox += out;
        return true;
    });
    if (last == first || vox < kMinVoxels) return first;
    ErrorText text(ctx);
    if (dmalloc_on(ctx, &copy.p, bytes, st) != TW_OK) {
        text.put_back();
        return first;
    }
    copy.bytes = bytes;
    unsigned char *to = static_cast<unsigned char *>(copy.p);
    for (RJob *j = first; j < last; ++j) {
        RJob padded = *j;
        padded.src = to;
        padded.src_py = (int64_t)row_bytes(*j) / (j->dtype == TW_U8 ? 1 : 2);
        padded.src_pz = padded.src_py * j->src_n[1];
        padded.ragged = 1;
        if (!encode_source_map(padded) || launch_repitch(*j, to, (int64_t)row_bytes(*j), st, ctx->sm_count) != cudaSuccess) {
            cudaGetLastError();  // (a descriptor the driver refuses: it and the rest gather)
            return j;
        }
        to += size(*j);
        *j = padded;
        count_launch(ctx);
    }
    return last;
}

}  // namespace

tw_status run_jobs(tw_ctx *ctx, RJob *jobs, int njobs, cudaStream_t st, size_t copy_limit, size_t *copied)
{
    if (copied) *copied = 0;
    if (njobs <= 0) return TW_OK;
    const int staging = ctx->resample_staging.load();
    if (jobs[0].kind == 1) {
        // TPS jobs: those whose source TMA can describe, trilinear ones that
        // are resampled from a padded copy, and the rest, which gather
        // (below 16 M voxels a nearest-neighbour launch gathers: one launch
        // instead of five; 208 x 144 x 131 uint8, call: 81 us gathered, 91
        // staged; 256 x 256 x 128: 97 and 104; 400 x 224 x 128: 116 and 114)
        const bool nearest = jobs[0].interp != 0;
        int64_t vox = 0;
        for (int i = 0; i < njobs; ++i) vox += jobs[i].out_n[0] * jobs[i].out_n[1] * jobs[i].out_n[2];
        if (!staging || (nearest && vox < (int64_t)16 << 20)) return run_group(ctx, jobs, njobs, 0, st);
        RJob *const end = jobs + njobs;
        RJob *const mid = std::stable_partition(jobs, end, [](RJob &j) { return encode_source_map(j); });
        const auto run_tps = [&](RJob *b, RJob *e, bool gathers) -> tw_status {
            if (e == b) return TW_OK;
            ErrorText text(ctx);
            tw_status s = run_group(ctx, b, (int)(e - b), 0, st);
            if (s == TW_ERR_OOM && gathers) {  // no room for the plans: gathering needs none
                text.put_back();
                for (RJob *j = b; j < e; ++j) j->tma_ok = 0;
                s = run_group(ctx, b, (int)(e - b), 0, st);
            }
            return s;
        };
        TW_TRY(run_tps(jobs, mid, nearest));
        StreamBlock copy{ctx, st};
        RJob *const last = jobs[0].interp == 0 ? pad_sources(ctx, mid, end, copy, st, copy_limit) : mid;
        if (copied) *copied = copy.bytes;
        TW_TRY(run_tps(mid, last, true));
        if (end > last) TW_TRY(run_group(ctx, last, (int)(end - last), 0, st));
        return TW_OK;
    }
    // affine jobs whose tiles can be staged first, the others gather
    uint32_t box = 0;
    RJob *const mid = std::stable_partition(jobs, jobs + njobs, [&](RJob &j) {
        const uint32_t b = staging ? encode_affine_box(j, staging == 2) : 0u;
        box = std::max(box, b);
        return b != 0;
    });
    const int ns = (int)(mid - jobs);
    if (ns > 0) TW_TRY(run_group(ctx, jobs, ns, box, st));
    if (ns < njobs) TW_TRY(run_group(ctx, mid, njobs - ns, 0, st));
    return TW_OK;
}

// TPS units walk 64 output planes (several cell layers: the staged source
// window is loaded once per walk); when a launch has too few units to
// balance, they get shorter.  Staged ones down to 16 planes -- below that the
// windows and the per-layer set-up cost more than an even last wave gives (256 x
// 256 x 128 uint8: 109 us at 4 planes, 91 at 16; 512^3 uint16: 573 at 64, 513 at
// 16; 1024 x 1024 x 256 uint8, spacing 4: 2114 at 64, 2011 at 32).  Gathered units
// keep no window: they need fewer to balance, and a small launch is better off
// with many short ones (64^3 uint8, call: 61 us at 16 planes, 53 at 1).
int tps_unit_planes(const RJob *jobs, int njobs, bool staged, int sm_count)
{
    int64_t bd[3];
    brick_dims(1, jobs[0].g, bd);
    int zs = std::max(64, jobs[0].g);
    for (; zs > (staged ? 16 : 1); zs /= 2) {
        int64_t total = 0;
        for (int i = 0; i < njobs; ++i) {
            const int64_t *n = jobs[i].out_n;
            total += (n[0] + bd[0] - 1) / bd[0] * ((n[1] + bd[1] - 1) / bd[1]) * ((n[2] + zs - 1) / zs);
        }
        if (total >= (staged ? 32 : 8) * (int64_t)sm_count) break;
    }
    return zs;
}

namespace {

// One launch over jobs that share (dtype, kind, g, interp); affine_box: bytes
// of the largest staged box when the jobs are staged affine jobs, else 0.
tw_status run_group(tw_ctx *ctx, RJob *jobs, int njobs, uint32_t affine_box, cudaStream_t st)
{
    int64_t total = 0;
    auto count = [&](int zs) {
        total = 0;
        for (int i = 0; i < njobs; ++i) {
            int64_t bd[3];
            brick_dims(jobs[i].kind, jobs[i].g, bd);
            if (jobs[i].kind == 1) bd[2] = zs;
            else if (affine_box)
                for (int a = 0; a < 3; ++a) bd[a] = kAffineTile[a];
            jobs[i].zs = zs;
            for (int a = 0; a < 3; ++a) jobs[i].bricks[a] = (jobs[i].out_n[a] + bd[a] - 1) / bd[a];
            jobs[i].brick_begin = total;
            total += jobs[i].bricks[0] * jobs[i].bricks[1] * jobs[i].bricks[2];
        }
    };
    const bool staged = jobs[0].kind == 1 && jobs[0].tma_ok != 0, ragged = staged && jobs[0].ragged;
    count(jobs[0].kind == 1 ? tps_unit_planes(jobs, njobs, staged, ctx->sm_count) : 8);
    if (total == 0) return TW_OK;
    // the units' staging plans and the list of units left to the gather kernel
    StreamBlock fb{ctx, st};
    if (staged) {
        fb.bytes = tps_stage_ws_bytes(total);
        TW_TRY(dmalloc_on(ctx, &fb.p, fb.bytes, st));
        TW_CUDA_TRY(cudaMemsetAsync(fb.p, 0, sizeof(int64_t), st));
    }
    void *d_fb = fb.p;
    // plan, walk lists, staged (interior walks), staged (other walks), gather
    const uint64_t launches = staged ? 5 : 1;
    const auto launch = [&](const RJob *d) {
        return affine_box ? launch_affine_staged(d, njobs, total, jobs[0].dtype, affine_box, st, ctx->sm_count, ctx->err_word)
                          : launch_resample(d, njobs, total, jobs[0].dtype, jobs[0].kind, jobs[0].g, jobs[0].interp, st,
                                            ctx->sm_count, ctx->err_word, d_fb, ragged);
    };
    const size_t bytes = sizeof(RJob) * (size_t)njobs;
    if (njobs <= tw_ctx::kJobsPerSlot && ctx->job_d) {
        // descriptors through the context's slot ring: an asynchronous copy
        // from pinned memory, so the host never waits for earlier work here
        std::lock_guard<std::mutex> lk(ctx->job_mu);
        const int s = ctx->job_next;
        ctx->job_next = (s + 1) % tw_ctx::kJobSlots;
        TW_CUDA_TRY(cudaEventSynchronize(ctx->job_ev[s]));  // the slot's previous launch has finished
        RJob *h = ctx->job_h + (size_t)s * tw_ctx::kJobsPerSlot;
        RJob *d = ctx->job_d + (size_t)s * tw_ctx::kJobsPerSlot;
        std::memcpy(h, jobs, bytes);
        TW_CUDA_TRY(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st));
        cudaError_t e = launch(d);
        if (e != cudaSuccess) return fail(ctx, TW_ERR_CUDA, std::string("resample launch: ") + cudaGetErrorString(e));
        TW_CUDA_TRY(cudaEventRecord(ctx->job_ev[s], st));
        count_launch(ctx, launches);
        return TW_OK;
    }
    RJob *d_jobs = nullptr;
    TW_CUDA_TRY(cudaMallocFromPoolAsync((void **)&d_jobs, bytes, ctx->pool, st));
    TW_CUDA_TRY(cudaMemcpyAsync(d_jobs, jobs, bytes, cudaMemcpyHostToDevice, st));
    cudaError_t e = launch(d_jobs);
    cudaFreeAsync(d_jobs, st);
    if (e != cudaSuccess) return fail(ctx, TW_ERR_CUDA, std::string("resample launch: ") + cudaGetErrorString(e));
    count_launch(ctx, launches);
    return TW_OK;
}

}  // namespace

// ------------------------------------------------------- TMA descriptors

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library does not link the driver API); null when the driver lacks it.
EncodeTiled encode_fn()
{
    static EncodeTiled fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return (EncodeTiled) nullptr;
        }
        return reinterpret_cast<EncodeTiled>(f);
    }();
    return fn;
}

}  // namespace

bool encode_source_map(RJob &j)
{
    j.tma_ok = 0;
    const EncodeTiled fn = encode_fn();
    if (!fn || !j.src) return false;
    const uint64_t es = j.dtype == TW_U8 ? 1 : 2;
    // TMA rules: 16-byte aligned base and row / plane pitches; a box (one
    // staged plane: kStageBoxW x kStageBoxH elements) no larger than the tensor
    if (reinterpret_cast<uintptr_t>(j.src) % 16 != 0) return false;
    if ((j.src_py * es) % 16 != 0 || (j.src_pz * es) % 16 != 0) return false;
    if (j.src_n[0] < kStageBoxW || j.src_n[1] < kStageBoxH || j.src_n[2] < 1) return false;
    if (j.src_n[0] > 0xffffffffLL || j.src_n[1] > 0xffffffffLL || j.src_n[2] > 0xffffffffLL) return false;
    if ((uint64_t)j.src_pz * es >= (1ull << 40)) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)j.src_n[0], (cuuint64_t)j.src_n[1], (cuuint64_t)j.src_n[2]};
    const cuuint64_t strides[2] = {(cuuint64_t)j.src_py * es, (cuuint64_t)j.src_pz * es};
    const cuuint32_t box[3] = {(cuuint32_t)kStageBoxW, (cuuint32_t)kStageBoxH, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(&j.tmap, es == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3,
                          const_cast<void *>(j.src), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return false;
    j.tma_ok = 1;
    return true;
}

namespace {

// floor of a position for the estimates below, |q| < 8192 (no call of floor: these
// run on every call, and 600 of them took 2 us)
int low_int(double q) { return (int)(q + 8192.0) - 8192; }

// How a warp's tap loads of a staged affine tile meet the 32 banks: floors of
// the positions of a few of its rows (two rows of 16 lanes, a voxel pair
// each).
struct TapRows {
    static constexpr int kRows = 4;
    int q[kRows][32][3];
    explicit TapRows(const double M[12])
    {
        const double at[kRows][5] = {{0, 0, .31, .62, .13}, {6, 5, .77, .05, .48}, {10, 9, .52, .89, .95}, {14, 15, .16, .4, .7}};
        for (int r = 0; r < kRows; ++r)
            for (int l = 0; l < 32; ++l) {
                const double p[3] = {2.0 * (l & 15), at[r][0] + (l >> 4), at[r][1]};
                for (int a = 0; a < 3; ++a)
                    q[r][l][a] = low_int(M[a * 4] * p[0] + M[a * 4 + 1] * p[1] + M[a * 4 + 2] * p[2] + at[r][2 + a]);
            }
    }
    // shared-memory passes per load, summed over the rows: the most distinct
    // words any bank is asked for (at least `limit` once the sum reaches it)
    int passes(int pr, int pp, int es, int limit) const
    {
        int sum = 0;
        for (int r = 0; r < kRows && sum < limit; ++r) {
            int word[32], depth[32] = {0}, chain[32], head[32], worst = 1;
            for (int k = 0; k < 32; ++k) head[k] = -1;
            for (int l = 0; l < 32; ++l) {
                const int w = (q[r][l][2] * pp + q[r][l][1] * pr + q[r][l][0] * es) >> 2, bank = w & 31;
                int k = head[bank];
                while (k >= 0 && word[k] != w) k = chain[k];
                if (k >= 0) continue;
                word[l] = w;
                chain[l] = head[bank];
                head[bank] = l;
                worst = std::max(worst, ++depth[bank]);
            }
            sum += worst;
        }
        return sum;
    }
};

// The part of an affine job's output tiles that have a sample inside the subject
// volume, from 6 x 6 x 6 of them.
double inside_part(const RJob &j)
{
    constexpr int N = 6;
    // per axis of the source: the part of a position each axis of the output
    // gives, and the limits of a tile's centre
    double part[3][3][N], lo[3], hi[3];
    for (int r = 0; r < 3; ++r) {
        const double *m = j.M + 4 * r;
        double h = 0.0;
        for (int a = 0; a < 3; ++a) {
            h += 0.5 * std::fabs(m[a]) * (kAffineTile[a] - 1);
            for (int i = 0; i < N; ++i)
                part[r][a][i] = m[a] * ((double)j.out_o[a] + (i + 0.5) / N * (double)j.out_n[a]) + (a == 0 ? m[3] : 0.0);
        }
        lo[r] = -h;
        hi[r] = (double)(j.glob[r] - 1) + h;
    }
    int n = 0;
    for (int z = 0; z < N; ++z)
        for (int y = 0; y < N; ++y) {
            double yz[3];
            for (int r = 0; r < 3; ++r) yz[r] = part[r][1][y] + part[r][2][z];
            for (int x = 0; x < N; ++x) {
                bool in = true;
                for (int r = 0; r < 3; ++r) {
                    const double q = yz[r] + part[r][0][x];
                    in = in & (q >= lo[r]) & (q <= hi[r]);
                }
                n += in;
            }
        }
    return (double)n / (N * N * N);
}

// Is an affine job faster staged than gathered?  Both are estimated in cycles per
// 64 voxels and SM, fitted to 2,200 timings: scales of 0.3 to 4 along some or all
// axes, rotations, both, uint8 and uint16, rows of whole 16 bytes or not, sources
// of 4 M to 0.5 G elements, 5 to 100 % of the output inside.  Gathered, a sample
// costs by the 32-byte sectors of a row's tap loads, more where rows run along
// source planes, and by the source bytes it consumes; one outside the source
// costs the same whatever the matrix.  Staged, a sample costs by the bytes of the
// box, dearer by granules, and with two or more stages also by its bank passes.
// us gathered and staged at 1021 x 1019 x 509, by granules: reduction by 2 of
// uint16 399 and 939, by 2.25 of uint8 249 and 567, no rotation, uint16, 2255 and
// 2682, 15 degrees about each axis, uint16, 4980 and 3643; at 1024 x 1024 x 512,
// by TMA: 396 and 366, 246 and 303, 2217 and 1500, 4967 and 1544; 512 x 512 x 256
// uint16, a quarter turn about y and a reduction by 2, an eighth of the output
// inside: 626 and 1205.  The factors lean towards staging where the estimates
// meet.  Over the timings the choice costs 0.4 % over the faster one (staged
// always: 7 %, up to 2.5 times).
bool staging_pays(const RJob &j, bool tma, bool one_stage, double bytes, double passes)
{
    const int es = j.dtype == TW_U8 ? 1 : 2;
    const double *M = j.M;
    const double at[3][3] = {{.3, .6, .1}, {.7, .1, .5}, {.5, .9, .95}};
    int sectors = 0;  // of three rows' loads, where a lane's is not the one before its
    for (const auto &o : at) {
        int64_t last = INT64_MIN;
        for (int l = 0; l < 32; ++l) {
            const int64_t q[3] = {low_int(M[0] * 2 * l + o[0]), low_int(M[4] * 2 * l + o[1]), low_int(M[8] * 2 * l + o[2])};
            const int64_t s = ((q[2] * j.src_pz + q[1] * j.src_py + q[0]) * es) >> 5;
            sectors += s != last;
            last = s;
        }
    }
    const double S = sectors / 3.0;
    const double det = std::fabs(M[0] * (M[5] * M[10] - M[6] * M[9]) - M[1] * (M[4] * M[10] - M[6] * M[8]) +
                                 M[2] * (M[4] * M[9] - M[5] * M[8]));
    const double yz = std::fabs(M[9]) / (std::fabs(M[5]) + std::fabs(M[9]) + 1e-9);
    const double xz = std::fabs(M[8]) / (std::fabs(M[0]) + std::fabs(M[4]) + std::fabs(M[8]) + 1e-9);
    // (a sector per lane: 150 to 1160 cycles)
    const double inside = S > 28.0 ? 400.0
                                   : 54 + 2.8 * std::min(S, 16.0) + 7 * std::max(S - 16, 0.0) + 26 * yz + 100 * xz +
                                         .037 * 64 * es * det;
    const double f = inside_part(j), gathered = f * inside + (1 - f) * 115;
    if (!tma) {  // (granules from a source that stays in L2 cost less)
        const bool in_l2 = (double)j.src_pz * (double)j.src_n[2] * es < 100e6;
        return 50 + .122 * bytes * (.3 + .7 * f) <= (in_l2 ? 1.2 : 1.1) * gathered;
    }
    const double staged = one_stage ? (es == 1 ? 70 : 62) + .0345 * bytes * (.8 + .2 * f) + 15 * std::max(passes - 3, 0.0)
                                    : 33 + 10.3 * passes + .009 * bytes;
    return staged <= 1.05 * gathered;
}

}  // namespace

uint32_t plan_affine_box(RJob &j, bool can_tma, bool always)
{
    j.tma_ok = 0;
    const int es = j.dtype == TW_U8 ? 1 : 2;
    // a nearest-neighbour sample reads one element: gathered it takes less
    // than its share of a staged box (406 against 1050 us, 700 x 600 x 300 u16)
    if (j.interp == 1 || reinterpret_cast<uintptr_t>(j.src) % 16 != 0) return 0;
    // extents of a tile's samples, their +1 taps, and a margin for rounding
    int box[3];
    double reach[3];  // largest positions relative to their brick's origin
    for (int r = 0; r < 3; ++r) {
        double ext = 0.0, far = 0.0;
        const int brick[3] = {256, 8, 8};
        for (int a = 0; a < 3; ++a) {
            const double m = std::fabs(j.M[r * 4 + a]);
            ext += m * (kAffineTile[a] - 1);
            far += m * brick[a];
        }
        if (!(ext < 240.0) || !(std::fabs(j.M[r * 4 + 3]) < 1e9)) return 0;  // (NaN and infinity included)
        box[r] = (int)std::floor(ext + 2.0 / 64.0) + 4;
        reach[r] = far + box[r];
    }
    for (int a = 0; a < 3; ++a) {
        const int64_t lim = (int64_t)1 << 28;  // TMA coordinates are int32
        if (j.out_o[a] < -lim || j.out_o[a] + j.out_n[a] > lim || j.src_o[a] < -lim || j.src_o[a] > lim || j.glob[a] > lim) return 0;
    }
    double tiles = 1.0;
    for (int a = 0; a < 3; ++a) tiles *= (double)((j.out_n[a] + kAffineTile[a] - 1) / kAffineTile[a]);
    if (tiles >= 2147483648.0) return 0;
    // The box's pitches: the smallest that copies allow, padded (planes by up
    // to seven steps, then rows by one) until a tap load takes close to its two
    // passes -- unpadded, some matrices put most lanes in a few banks (8.8
    // passes at 10 degrees about each axis with rows of 1034 bytes, 16 at a
    // quarter turn about z).
    const int A = 16 / es, w1 = (box[0] + A - 1 + A - 1) / A * A;  // starts on a 16-byte boundary
    const bool tma = can_tma && (j.src_py * es) % 16 == 0 && (j.src_pz * es) % 16 == 0 && w1 + A <= std::min<int64_t>(256, j.src_n[0]) &&
                     box[1] + 7 <= j.src_n[1] && box[2] <= j.src_n[2] && (uint64_t)j.src_pz * es < (1ull << 40);
    const int dy = (int)((j.src_py * es) & 15), dz = (int)((j.src_pz * es) & 15);
    const TapRows rows(j.M);
    const int good = 9 * TapRows::kRows / 4;  // 2.25 passes
    int best = 1 << 30;
    int64_t bytes = 0;
    for (int pad = 0; pad < 16 && best > good; ++pad) {
        const int i = pad >> 3, k = pad & 7;
        int pr, pp;
        if (tma) {
            pr = (w1 + A * i) * es;
            pp = pr * (box[1] + k);
        } else {
            // congruent to the source's pitches modulo 16, rows at least 30
            // bytes apart: each is copied in whole 16-byte granules
            pr = ((box[0] * es + 30 - dy + 15) & ~15) + dy + 16 * i;
            pp = ((pr * box[1] - dz + 15) & ~15) + dz + 16 * k;
        }
        const int64_t need = ((int64_t)pp * box[2] + 32 + 127) / 128 * 128;
        if (need > kAffineSmem) continue;
        if (bytes && 2 * bytes <= kAffineSmem && 2 * need > kAffineSmem) continue;  // two stages are worth more
        const int p = rows.passes(pr, pp, es, best);
        if (p >= best) continue;
        best = p;
        bytes = need;
        j.st_w = tma ? w1 + A * i : box[0];
        j.st_h = tma ? box[1] + k : box[1];
        j.st_pr = pr;
        j.st_pp = pp;
    }
    j.st_d = box[2];
    // the box fits, and tap offsets and their partial sums (floating point,
    // exact below 2^22) stay small
    if (!bytes || reach[2] * j.st_pp + reach[1] * j.st_pr + reach[0] * es > 2097152.0) return 0;
    const double copied = (double)(tma ? j.st_pp : (box[0] * es + 30) / 16 * 16 * box[1]) * box[2];
    const double passes = (double)best / TapRows::kRows;
    const double voxels64 = kAffineTile[0] * kAffineTile[1] * kAffineTile[2] / 64;
    if (!always && !staging_pays(j, tma, 2 * bytes > kAffineSmem, copied / voxels64, passes)) return 0;
    j.tma_ok = tma ? 1 : 2;
    return (uint32_t)bytes;
}

uint32_t encode_affine_box(RJob &j, bool always)
{
    const EncodeTiled fn = encode_fn();
    const uint32_t bytes = plan_affine_box(j, fn != nullptr, always);
    if (j.tma_ok == 1) {
        const int es = j.dtype == TW_U8 ? 1 : 2;
        const cuuint64_t dims[3] = {(cuuint64_t)j.src_n[0], (cuuint64_t)j.src_n[1], (cuuint64_t)j.src_n[2]};
        const cuuint64_t strides[2] = {(cuuint64_t)j.src_py * es, (cuuint64_t)j.src_pz * es};
        const cuuint32_t b[3] = {(cuuint32_t)j.st_w, (cuuint32_t)j.st_h, (cuuint32_t)j.st_d};
        const cuuint32_t estr[3] = {1, 1, 1};
        if (fn(&j.tmap, es == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void *>(j.src),
               dims, strides, b, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
            j.tma_ok = 0;
            return 0;
        }
    }
    return bytes;
}

// ------------------------------------------------------------ sample hulls

namespace {

__device__ __forceinline__ void warp_minmax(float &mn, float &mx)
{
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
}

// One CTA per output cell-layer cz: min/max of q_z = DF_z + (k-1)g over node
// planes k = cz..cz+3 (convex-hull bound of the cubic B-spline).
__global__ void k_layer_zhull(const float4 *nodes, int64_t gx, int64_t gy, int g, float *zmin, float *zmax)
{
    __shared__ float smn[32], smx[32];
    const int cz = blockIdx.x;
    float mn = 3.4e38f, mx = -3.4e38f;
    const int64_t plane = gx * gy;
    for (int k = 0; k < 4; ++k) {
        const float zpos = (float)((int64_t)(cz + k - 1) * g);
        const float4 *p = nodes + (int64_t)(cz + k) * plane;
        for (int64_t i = threadIdx.x; i < plane; i += blockDim.x) {
            float q = p[i].z + zpos;
            mn = fminf(mn, q);
            mx = fmaxf(mx, q);
        }
    }
    warp_minmax(mn, mx);
    if ((threadIdx.x & 31) == 0) { smn[threadIdx.x >> 5] = mn; smx[threadIdx.x >> 5] = mx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { mn = fminf(mn, smn[w]); mx = fmaxf(mx, smx[w]); }
        zmin[cz] = fminf(mn, smn[0]);
        zmax[cz] = fmaxf(mx, smx[0]);
    }
}

// One CTA per box: min/max of q = DF + node position over nodes
// [c0, c1 + 3) on each axis (clamped to the grid).
__global__ void k_box_hull(const float4 *nodes, int64_t gx, int64_t gy, int64_t gz, int g, const int64_t *boxes,
                           float *lo, float *hi)
{
    __shared__ float sm[6][32];
    const int64_t *b = boxes + 6 * blockIdx.x;
    int64_t n0[3], n1[3];
    const int64_t gs[3] = {gx, gy, gz};
    for (int a = 0; a < 3; ++a) {
        n0[a] = b[a];
        n1[a] = b[3 + a] + 3;
        if (n1[a] > gs[a]) n1[a] = gs[a];
    }
    const int64_t ex = n1[0] - n0[0], ey = n1[1] - n0[1], ez = n1[2] - n0[2];
    const int64_t tot = ex * ey * ez;
    float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (int64_t i = threadIdx.x; i < tot; i += blockDim.x) {
        int64_t x = n0[0] + i % ex, t = i / ex;
        int64_t y = n0[1] + t % ey, z = n0[2] + t / ey;
        float4 d = nodes[(z * gy + y) * gx + x];
        float q[3] = {d.x + (float)((x - 1) * g), d.y + (float)((y - 1) * g), d.z + (float)((z - 1) * g)};
        for (int a = 0; a < 3; ++a) { mn[a] = fminf(mn[a], q[a]); mx[a] = fmaxf(mx[a], q[a]); }
    }
    for (int a = 0; a < 3; ++a) warp_minmax(mn[a], mx[a]);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int a = 0; a < 3; ++a) { sm[a][w] = mn[a]; sm[3 + a][w] = mx[a]; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int a = 0; a < 3; ++a) {
            float m0 = sm[a][0], m1 = sm[3 + a][0];
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) { m0 = fminf(m0, sm[a][k]); m1 = fmaxf(m1, sm[3 + a][k]); }
            lo[3 * blockIdx.x + a] = m0;
            hi[3 * blockIdx.x + a] = m1;
        }
    }
}

}  // namespace

tw_status tps_layer_zhull(tw_ctx *ctx, const float4 *nodes, const int64_t gsz[3], int g, cudaStream_t st,
                          std::vector<float> &zmin, std::vector<float> &zmax)
{
    const int64_t layers = gsz[2] - 3;
    zmin.assign(layers, 0.f);
    zmax.assign(layers, 0.f);
    if (layers <= 0) return TW_OK;
    // from the context's pool, which keeps its blocks: the device's default
    // pool gives its memory back at every synchronisation, so a block of it
    // cost milliseconds of mapping per call
    PoolBlock b{st};
    TW_CUDA_TRY(cudaMallocFromPoolAsync(&b.p, sizeof(float) * 2 * (size_t)layers, ctx->pool, st));
    float *d = static_cast<float *>(b.p);
    k_layer_zhull<<<(unsigned)layers, 256, 0, st>>>(nodes, gsz[0], gsz[1], g, d, d + layers);
    TW_CUDA_TRY(cudaGetLastError());
    count_launch(ctx);
    TW_CUDA_TRY(cudaMemcpyAsync(zmin.data(), d, sizeof(float) * layers, cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaMemcpyAsync(zmax.data(), d + layers, sizeof(float) * layers, cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaStreamSynchronize(st));
    return TW_OK;
}

tw_status tps_box_hull(tw_ctx *ctx, const float4 *nodes, const int64_t gsz[3], int g,
                       const std::vector<CellBox> &boxes, cudaStream_t st, std::vector<float> &lo,
                       std::vector<float> &hi)
{
    const size_t nb = boxes.size();
    lo.assign(3 * nb, 0.f);
    hi.assign(3 * nb, 0.f);
    if (nb == 0) return TW_OK;
    std::vector<int64_t> hb(6 * nb);
    for (size_t i = 0; i < nb; ++i)
        for (int a = 0; a < 3; ++a) {
            hb[6 * i + a] = boxes[i].c0[a];
            hb[6 * i + 3 + a] = boxes[i].c1[a];
        }
    PoolBlock b{st};
    TW_CUDA_TRY(cudaMallocFromPoolAsync(&b.p, (sizeof(int64_t) + sizeof(float)) * 6 * nb, ctx->pool, st));
    int64_t *db = static_cast<int64_t *>(b.p);
    float *dh = reinterpret_cast<float *>(db + 6 * nb);
    TW_CUDA_TRY(cudaMemcpyAsync(db, hb.data(), sizeof(int64_t) * 6 * nb, cudaMemcpyHostToDevice, st));
    k_box_hull<<<(unsigned)nb, 256, 0, st>>>(nodes, gsz[0], gsz[1], gsz[2], g, db, dh, dh + 3 * nb);
    TW_CUDA_TRY(cudaGetLastError());
    count_launch(ctx);
    TW_CUDA_TRY(cudaMemcpyAsync(lo.data(), dh, sizeof(float) * 3 * nb, cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaMemcpyAsync(hi.data(), dh + 3 * nb, sizeof(float) * 3 * nb, cudaMemcpyDeviceToHost, st));
    TW_CUDA_TRY(cudaStreamSynchronize(st));
    return TW_OK;
}

// ------------------------------------------------------- parameter surface

namespace {
void mat_mul4(const double *a, const double *b, double *c)
{
    double t[16];
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) {
            double s = 0;
            for (int k = 0; k < 4; ++k) s += a[i * 4 + k] * b[k * 4 + j];
            t[i * 4 + j] = s;
        }
    std::memcpy(c, t, sizeof(t));
}
void ident4(double *m)
{
    for (int i = 0; i < 16; ++i) m[i] = (i % 5 == 0) ? 1.0 : 0.0;
}
}  // namespace

tw_status make_param_affine(int warp_mode, int deformation_mode, const double para[3], const int64_t in_sz[3],
                            const int64_t out_sz[3], double M[16])
{
    ident4(M);
    if (warp_mode == 0 && deformation_mode == 2) {
        // scaling about the origin voxel: out(p) = in(p / s)
        for (int a = 0; a < 3; ++a) {
            if (!(para[a] > 0.0)) return TW_ERR_ARG;
            M[a * 5] = 1.0 / para[a];
        }
        return TW_OK;
    }
    if (warp_mode == 1 && deformation_mode == 1) {
        // translation: out(p) = in(p - t)
        for (int a = 0; a < 3; ++a) M[a * 4 + 3] = -para[a];
        return TW_OK;
    }
    if (warp_mode == 1 && deformation_mode == 0) {
        // rotation by angles (degrees) about x, then y, then z, about the
        // input centre, which lands on the output centre:
        //   forward  p_out = c_out + Rz Ry Rx (p_in - c_in)
        //   pull-back p_in = c_in + (Rz Ry Rx)^T (p_out - c_out)
        const double d2r = std::acos(-1.0) / 180.0;
        const double ax = para[0] * d2r, ay = para[1] * d2r, az = para[2] * d2r;
        double Rx[16], Ry[16], Rz[16], R[16];
        ident4(Rx); ident4(Ry); ident4(Rz);
        Rx[5] = std::cos(ax); Rx[6] = -std::sin(ax); Rx[9] = std::sin(ax); Rx[10] = std::cos(ax);
        Ry[0] = std::cos(ay); Ry[2] = std::sin(ay); Ry[8] = -std::sin(ay); Ry[10] = std::cos(ay);
        Rz[0] = std::cos(az); Rz[1] = -std::sin(az); Rz[4] = std::sin(az); Rz[5] = std::cos(az);
        mat_mul4(Ry, Rx, R);
        mat_mul4(Rz, R, R);
        double ci[3], co[3];
        for (int a = 0; a < 3; ++a) {
            ci[a] = 0.5 * (double)(in_sz[a] - 1);
            co[a] = 0.5 * (double)(out_sz[a] - 1);
        }
        for (int r = 0; r < 3; ++r) {
            double t = ci[r];
            for (int c = 0; c < 3; ++c) {
                M[r * 4 + c] = R[c * 4 + r];  // transpose
                t -= R[c * 4 + r] * co[c];
            }
            M[r * 4 + 3] = t;
        }
        return TW_OK;
    }
    return TW_ERR_ARG;
}

// ---------------------------------------------------------- slab pipeline

namespace {

struct Pinned {
    void *p = nullptr;
    size_t bytes = 0;
    ~Pinned() { if (p) cudaFreeHost(p); }
};

struct Events {
    std::vector<cudaEvent_t> ev;
    ~Events() { for (auto e : ev) cudaEventDestroy(e); }
    cudaError_t make(size_t n)
    {
        ev.resize(n, nullptr);
        for (auto &e : ev) {
            cudaError_t r = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
            if (r != cudaSuccess) return r;
        }
        return cudaSuccess;
    }
};

}  // namespace

tw_status stream_slabs(tw_ctx *ctx, const SlabIO &io,
                       const std::function<void(int64_t, int64_t, int64_t &, int64_t &)> &need,
                       const std::function<tw_status(int64_t, int64_t, const void *, void *, cudaStream_t)> &compute)
{
    const bool src_dev = is_device_ptr(io.src), dst_dev = is_device_ptr(io.dst);
    if (src_dev && dst_dev) {
        // nothing to stream: the whole volume in one launch; in slabs only
        // when its workspace does not fit the budget
        ErrorText text(ctx);
        const tw_status s = compute(0, io.dst_planes, io.src, io.dst, ctx->stream);
        if (s == TW_OK) return check_kernel_errors(ctx);
        if (s != TW_ERR_OOM) return s;
        text.put_back();
    }
    const bool src_pin = !src_dev && is_pinned_ptr(io.src), dst_pin = !dst_dev && is_pinned_ptr(io.dst);
    const size_t src_bytes = io.src_plane_bytes * (size_t)io.src_planes;
    const size_t dst_bytes = io.dst_plane_bytes * (size_t)io.dst_planes;
    void *d_src = src_dev ? const_cast<void *>(io.src) : nullptr;
    void *d_dst = dst_dev ? io.dst : nullptr;
    struct Guard {
        tw_ctx *c; void *p; size_t b;
        ~Guard() { if (p) dfree(c, p, b); }
    } gs{ctx, nullptr, 0}, gd{ctx, nullptr, 0};
    if (!src_dev) {
        TW_TRY(dmalloc(ctx, &d_src, src_bytes));
        gs.p = d_src; gs.b = src_bytes;
    }
    if (!dst_dev) {
        TW_TRY(dmalloc(ctx, &d_dst, dst_bytes));
        gd.p = d_dst; gd.b = dst_bytes;
    }
    // source chunks of ~16 MiB (whole planes): 0.3 ms of the link each
    int64_t chunk = std::max<int64_t>(1, (int64_t)((16ull << 20) / std::max<size_t>(io.src_plane_bytes, 1)));
    chunk = std::min(chunk, io.src_planes);
    const int64_t nchunks = (io.src_planes + chunk - 1) / chunk;
    const int64_t nslabs = (io.dst_planes + io.slab - 1) / io.slab;
    Events ev_up, ev_comp, ev_down;
    TW_CUDA_TRY(ev_up.make(nchunks));
    TW_CUDA_TRY(ev_comp.make(nslabs));
    TW_CUDA_TRY(ev_down.make(nslabs));
    // pageable host memory goes through pinned staging rings
    const int kRing = 3;
    Pinned up_ring[kRing], down_ring[kRing];
    const size_t up_slot = io.src_plane_bytes * (size_t)chunk;
    const size_t down_slot = io.dst_plane_bytes * (size_t)io.slab;
    if (!src_dev && !src_pin)
        for (auto &r : up_ring) {
            TW_CUDA_TRY(cudaHostAlloc(&r.p, up_slot, cudaHostAllocDefault));
            r.bytes = up_slot;
        }
    if (!dst_dev && !dst_pin)
        for (auto &r : down_ring) {
            TW_CUDA_TRY(cudaHostAlloc(&r.p, down_slot, cudaHostAllocDefault));
            r.bytes = down_slot;
        }
    std::vector<int64_t> up_slot_owner(kRing, -1), down_slot_owner(kRing, -1);
    int64_t uploaded = 0;  // chunks issued
    std::deque<int64_t> pending_down;  // slabs whose D2H into a staging slot must be copied out

    auto drain_one = [&](void) -> tw_status {
        const int64_t s = pending_down.front();
        pending_down.pop_front();
        TW_CUDA_TRY(cudaEventSynchronize(ev_down.ev[s]));
        const int64_t z0 = s * io.slab, z1 = std::min(io.dst_planes, z0 + io.slab);
        std::memcpy(static_cast<char *>(io.dst) + (size_t)z0 * io.dst_plane_bytes, down_ring[s % kRing].p,
                    (size_t)(z1 - z0) * io.dst_plane_bytes);
        return TW_OK;
    };

    auto upload_until = [&](int64_t zhi) -> tw_status {
        const int64_t need_chunk = src_dev ? -1 : std::min(nchunks - 1, zhi / chunk);
        while (uploaded <= need_chunk) {
            const int64_t k = uploaded;
            const int64_t z0 = k * chunk, z1 = std::min(io.src_planes, z0 + chunk);
            const size_t bytes = (size_t)(z1 - z0) * io.src_plane_bytes;
            char *dptr = static_cast<char *>(d_src) + (size_t)z0 * io.src_plane_bytes;
            const char *hptr = static_cast<const char *>(io.src) + (size_t)z0 * io.src_plane_bytes;
            if (src_pin) {
                TW_CUDA_TRY(cudaMemcpyAsync(dptr, hptr, bytes, cudaMemcpyHostToDevice, ctx->h2d));
            } else {
                const int slot = (int)(k % kRing);
                if (up_slot_owner[slot] >= 0) TW_CUDA_TRY(cudaEventSynchronize(ev_up.ev[up_slot_owner[slot]]));
                std::memcpy(up_ring[slot].p, hptr, bytes);
                TW_CUDA_TRY(cudaMemcpyAsync(dptr, up_ring[slot].p, bytes, cudaMemcpyHostToDevice, ctx->h2d));
                up_slot_owner[slot] = k;
            }
            TW_CUDA_TRY(cudaEventRecord(ev_up.ev[k], ctx->h2d));
            ctx->h2d_bytes += bytes;
            ++uploaded;
        }
        if (need_chunk >= 0) TW_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ev_up.ev[need_chunk], 0));
        return TW_OK;
    };

    for (int64_t s = 0; s < nslabs; ++s) {
        const int64_t z0 = s * io.slab, z1 = std::min(io.dst_planes, z0 + io.slab);
        int64_t lo = 0, hi = io.src_planes - 1;
        if (!src_dev) need(z0, z1, lo, hi);
        hi = std::max<int64_t>(0, std::min(hi, io.src_planes - 1));
        TW_TRY(upload_until(hi));
        TW_TRY(compute(z0, z1, d_src, d_dst, ctx->stream));
        TW_CUDA_TRY(cudaEventRecord(ev_comp.ev[s], ctx->stream));
        if (!dst_dev) {
            TW_CUDA_TRY(cudaStreamWaitEvent(ctx->d2h, ev_comp.ev[s], 0));
            const size_t bytes = (size_t)(z1 - z0) * io.dst_plane_bytes;
            const char *dptr = static_cast<const char *>(d_dst) + (size_t)z0 * io.dst_plane_bytes;
            if (dst_pin) {
                TW_CUDA_TRY(cudaMemcpyAsync(static_cast<char *>(io.dst) + (size_t)z0 * io.dst_plane_bytes, dptr, bytes,
                                            cudaMemcpyDeviceToHost, ctx->d2h));
            } else {
                const int slot = (int)(s % kRing);
                while (!pending_down.empty() && pending_down.front() <= s - kRing) TW_TRY(drain_one());
                TW_CUDA_TRY(cudaMemcpyAsync(down_ring[slot].p, dptr, bytes, cudaMemcpyDeviceToHost, ctx->d2h));
                pending_down.push_back(s);
            }
            TW_CUDA_TRY(cudaEventRecord(ev_down.ev[s], ctx->d2h));
            ctx->d2h_bytes += (size_t)(z1 - z0) * io.dst_plane_bytes;
        }
    }
    while (!pending_down.empty()) TW_TRY(drain_one());
    TW_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    TW_CUDA_TRY(cudaStreamSynchronize(ctx->d2h));
    TW_CUDA_TRY(cudaStreamSynchronize(ctx->h2d));
    return check_kernel_errors(ctx);
}

}  // namespace tw
