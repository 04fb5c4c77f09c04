// gizmo_b200/csrc/noalloc.cu -- density sums for callers that cannot allocate
// device memory (gz_density_sums_noalloc in include/gizmo_hydro.h).
//
// Some callers own all device memory themselves -- a host code whose memory
// pool has reserved the device, or a loop that cannot accept the device-wide
// synchronisation a cudaMalloc/cudaFree implies -- and so cannot use a
// gz_context, which allocates its buffers. This entry point computes the same
// fixed-h density sums as gz_density_sums for a particle set that the caller
// already holds in device memory, and allocates nothing: its only scratch is
// the static Scratch below (2.1 MiB of device memory) that every GPU loading this
// library holds until the process exits.
//
// The particles are put in Morton order first, so that runs of 32 have small
// bounding boxes; a run of 32 targets then tests every other run's box and only
// scans the particles of the runs it can reach. Each pair of those is screened in
// FP32, with a margin that bounds the FP32 rounding, and only the pairs near or
// inside the support take the exact FP64 test and the sums, whose arithmetic is
// the one of k_density_sums in FP64 (this file is built with -fmad=false like
// passes_fp64.cu), so the sums agree with gz_density_sums up to summation order.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/gizmo_hydro.h"
#include "state.cuh"

using namespace gz;

namespace {

constexpr int kMaxParticles = GZ_NOALLOC_MAX_PARTICLES;
constexpr int kRun = 32;      // particles of a run: the targets of a block, and the unit of the box tests
constexpr int kSlices = 8;    // warps of a block, each taking its share of the candidates for the block's targets
constexpr int kShare = kRun / kSlices;  // candidates a warp takes from each run
constexpr int kHits = 32;     // screened candidates a lane holds before the warp evaluates them
constexpr int kFewHits = 8;   // up to as many of a target are evaluated by its own lane
constexpr int kDigits = 256;  // Morton key, 8 bits an axis: three 8-bit radix passes
constexpr int kSortBlocks = 8, kSortWarps = 32;  // the cluster that sorts
constexpr int kSortRounds = kMaxParticles / (kSortBlocks * kSortWarps * 32);  // most particles a lane holds
constexpr int kMaxDevices = 128;
static_assert(kMaxParticles <= 65536, "a hit is a 16-bit particle index");

// Bounding box of a run, rounded outward to FP32: lo.w the largest coordinate
// magnitude, hi.w the largest |h|. A run that holds a NaN is given the whole space.
// All lengths of the screen are in units of the box, so that their squares stay in
// FP32's range whatever the unit of length is (unscaled, the squares of a box below
// ~1e-19 are denormal, and the screen's slack no longer covers their rounding).
struct RunBox {
    float4 lo, hi;
};

// The only scratch of the entry point. Shared by every call on a device; what a
// call reads it has written itself, so nothing in it needs clearing.
struct Scratch {
    unsigned key[2][kMaxParticles];
    int order[2][kMaxParticles];              // sorted -> caller's index: [0] after the sort
    float4 pos[kMaxParticles];                // sorted FP32 positions in units of the box; w: the caller's index
    RunBox box[kMaxParticles / kRun];
};
static_assert(sizeof(Scratch) <= 2162688, "the documented size (2.1 MiB) is out of date");
static __device__ __align__(256) Scratch g_scratch;

std::mutex g_setup_mutex;
Scratch *g_scratch_ptr[kMaxDevices] = {};  // device address of g_scratch, per device

// A particle index read from the scratch. It lies in [0, n) unless another call overlaps this one and rewrites the
// scratch: the results are undefined then, but no access leaves the caller's arrays.
__device__ __forceinline__ int own_index(int i, int n) { return (int)min((unsigned)i, (unsigned)(n - 1)); }

// What the sums read of the scratch.
struct SumsWork {
    const int *order;
    const float4 *pos;
    const RunBox *box;
};

__device__ unsigned spread8(unsigned x)
{
    x = (x | (x << 8)) & 0x00f00fu;
    x = (x | (x << 4)) & 0x0c30c3u;
    return (x | (x << 2)) & 0x249249u;
}

// Morton key of caller's particle i (the order only has to be good: coordinates outside the box are clamped)
__device__ unsigned key_of(const double *__restrict__ pos, int i, double box)
{
    unsigned k = 0;
    for (int c = 0; c < 3; c++) {
        const double v = pos[3 * (size_t)i + c] / box * 256.0;
        k |= spread8(v > 0.0 ? (v < 255.0 ? (unsigned)v : 255u) : 0u) << c;
    }
    return k;
}

// The caller's particles in the order of their Morton keys, equal keys in the caller's order: a stable radix sort of
// three 8-bit digits by one cluster. Each warp owns a run of consecutive places and holds its particles in registers
// from their count to their scatter; the warps' counts become offsets in shared memory, the blocks' in distributed
// shared memory, and the cluster's barrier separates the passes.
//
// The sort is this file's own, and one launch whatever n is, for what the entry point promises: a library's sort picks
// its kernels by n, so that the first larger call loads new ones (which can need device memory and a synchronisation
// when the caller has neither to give), and its blocks wait on flags in the scratch, which a second, overlapping call
// rewrites. Here a place is computed from registers and shared memory alone and always lies in [0, n).
// It is bound by the latency of its three passes' barriers and loads, on eight multiprocessors: whole call 29, 66, 105,
// 171, 248 and 533 us at 100, 1,000, 4,000, 10,000, 20,000 and 65,536 particles, with a library's sort 27, 64, 103, 198,
// 268 and 529.
__global__ void __cluster_dims__(kSortBlocks, 1, 1) __launch_bounds__(32 * kSortWarps)
    k_noalloc_sort(int n, const double *__restrict__ pos, double box, Scratch *g)
{
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    __shared__ unsigned short s_cnt[kSortWarps][kDigits];  // a warp's particles of each digit, then those of the warps before it
    __shared__ int s_total[kDigits];                       // the block's particles of each digit
    __shared__ int s_base[kDigits];                        // places before the block's particles of each digit
    __shared__ int s_sum[kDigits / 32];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = (int)cluster.block_rank();
    // places of a warp: a multiple of 32, the same for every warp
    const int per = ((n + kSortBlocks * kSortWarps - 1) / (kSortBlocks * kSortWarps) + 31) / 32 * 32;
    const int first = (rank * kSortWarps + warp) * per + lane;
    for (int pass = 0; pass < 3; pass++) {
        const int src = pass == 1 ? 0 : 1, dst = 1 - src;  // the keys' way: -> 0 -> 1 -> 0
        unsigned key[kSortRounds];
        int idx[kSortRounds];
        unsigned short at[kSortRounds];  // place among the warp's particles of the digit
#pragma unroll
        for (int r = 0; r < kSortRounds; r++) {
            const int e = first + 32 * r;
            key[r] = 0;
            idx[r] = e;
            if (32 * r < per && e < n) {
                if (pass == 0) {
                    key[r] = key_of(pos, e, box);
                } else {
                    key[r] = __ldcg(&g->key[src][e]);
                    idx[r] = __ldcg(&g->order[src][e]);
                }
            }
        }
        for (int k = threadIdx.x; k < kSortWarps * kDigits; k += 32 * kSortWarps) (&s_cnt[0][0])[k] = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortRounds; r++) {
            if (32 * r >= per) break;
            const int d = (key[r] >> (8 * pass)) & (kDigits - 1);
            const bool have = first + 32 * r < n;
            const unsigned same = __match_any_sync(full, have ? d : kDigits);
            const int before = have ? s_cnt[warp][d] : 0;
            __syncwarp();
            at[r] = (unsigned short)(before + __popc(same & ((1u << lane) - 1u)));
            if (have && lane == __ffs(same) - 1) s_cnt[warp][d] = (unsigned short)(before + __popc(same));
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < kDigits) {
            int run = 0;
            for (int w = 0; w < kSortWarps; w += 16) {
                int c[16];
#pragma unroll
                for (int k = 0; k < 16; k++) c[k] = s_cnt[w + k][threadIdx.x];
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    s_cnt[w + k][threadIdx.x] = (unsigned short)run;
                    run += c[k];
                }
            }
            s_total[threadIdx.x] = run;
        }
        cluster.sync();
        int all = 0, before = 0, incl = 0;
        if (threadIdx.x < kDigits) {
#pragma unroll
            for (int b = 0; b < kSortBlocks; b++) {
                const int c = *cluster.map_shared_rank(&s_total[threadIdx.x], b);
                if (b < rank) before += c;
                all += c;
            }
            incl = all;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(full, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) s_sum[warp] = incl;
        }
        __syncthreads();
        if (threadIdx.x < kDigits) {
            for (int w = 0; w < warp; w++) before += s_sum[w];
            s_base[threadIdx.x] = before + incl - all;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortRounds; r++) {
            if (32 * r >= per || first + 32 * r >= n) break;
            const int d = (key[r] >> (8 * pass)) & (kDigits - 1);
            const int to = s_base[d] + s_cnt[warp][d] + at[r];
            if (pass < 2) __stcg(&g->key[dst][to], key[r]);
            __stcg(&g->order[dst][to], idx[r]);
        }
        __threadfence();
        cluster.sync();  // the places are written, and every block's totals read
    }
}

__global__ void __launch_bounds__(128) k_noalloc_runs(int n, const double *__restrict__ pos,
                                                      const double *__restrict__ hs, double unit,
                                                      const int *__restrict__ order, float4 *out, RunBox *box)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const float inf = __int_as_float(0x7f800000);
    float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf}, mag = 0.0f, h = 0.0f;
    bool nan = false;
    if (s < n) {
        const size_t o = (size_t)own_index(order[s], n);
        const double hv = fabs(hs[o]) / unit;
        float f[3];
        for (int c = 0; c < 3; c++) {
            const double v = pos[3 * o + c] / unit;
            f[c] = __double2float_rn(v);
            lo[c] = __double2float_rd(v);
            hi[c] = __double2float_ru(v);
            mag = fmaxf(mag, __double2float_ru(fabs(v)));
            nan |= v != v;
        }
        nan |= hv != hv;
        h = __double2float_ru(hv);
        out[s] = make_float4(f[0], f[1], f[2], __int_as_float((int)o));
    }
    for (int d = 16; d > 0; d >>= 1) {
        for (int c = 0; c < 3; c++) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], d));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], d));
        }
        mag = fmaxf(mag, __shfl_xor_sync(0xffffffffu, mag, d));
        h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, d));
    }
    nan = __any_sync(0xffffffffu, nan);
    if ((threadIdx.x & 31) == 0 && s < n) {
        box[s / kRun] = nan ? RunBox{make_float4(-inf, -inf, -inf, mag), make_float4(inf, inf, inf, inf)}
                            : RunBox{make_float4(lo[0], lo[1], lo[2], mag), make_float4(hi[0], hi[1], hi[2], h)};
    }
}

// The most by which an FP32 separation can differ from the FP64 one, for
// coordinates of magnitude up to m (units of the box): each axis divides two
// coordinates by the box (2^-53 m each), rounds them (2^-24 m each), their difference
// (2^-24 2m) and the wrap (2^-24 (2m + 1)), in all less than 2^-24 (8m + 2) an axis
// and, over three axes and the rounding of the squares, less than 2^-24 (16m + 8).
__device__ __forceinline__ float screen_margin(float m) { return 5.9604645e-8f * (16.0f * m + 8.0f); }

// distance of the interval [a, b] of coordinate differences to the nearest of 0 and +-1 (the box), where a
// pair's minimum image on one axis is measured from
__device__ __forceinline__ float axis_distance(float a, float b)
{
    const float d0 = fmaxf(a, -b), dp = fmaxf(a - 1.0f, 1.0f - b), dm = fmaxf(a + 1.0f, -1.0f - b);
    return fmaxf(fminf(d0, fminf(dp, dm)), 0.0f);
}

struct Target {
    double x, y, z, vx, vy, vz, h2, hinv;
};

struct SumsInput {
    const double *pos, *vel, *mass;
};

// one neighbour's contribution: DensitySpec::pair_kernel (density_loop.h:1140-1385)
__device__ __forceinline__ void add_pair(const PassParams &p, const SumsInput &in, const Target &t, size_t j, double *a)
{
    const double mj = in.mass[j], xj = in.pos[3 * j], yj = in.pos[3 * j + 1], zj = in.pos[3 * j + 2];
    const double vjx = in.vel[3 * j], vjy = in.vel[3 * j + 1], vjz = in.vel[3 * j + 2];  // all in flight together
    if (mj <= 0) return;
    double dx, dy, dz;
    const double r2 = sep2(t.x, t.y, t.z, xj, yj, zj, p.box, p.half, dx, dy, dz);
    if (r2 >= t.h2) return;
    const int mfv = p.method == 1;
    const double hinv3 = t.hinv * t.hinv * t.hinv, hinv4 = hinv3 * t.hinv;  // as k_hinv
    const double r = sqrt(r2);
    const double u = r * t.hinv;
    double wk, dwk;
    k_main(p.kernel, u, hinv3, hinv4, wk, dwk);
    const double mj_wk = mj * wk;
    a[0] += wk;
    a[1] += mj_wk;
    if (mfv && r == 0.0) {
        a[14] += mj_wk * vjx;
        a[15] += mj_wk * vjy;
        a[16] += mj_wk * vjz;
    }
    a[2] += -(3.0 * t.hinv * wk + u * dwk);
    if (r > 0.0) {
        a[4] += dx * dx * wk;
        a[5] += dy * dy * wk;
        a[6] += dz * dz * wk;
        a[7] += dx * dy * wk;
        a[8] += dy * dz * wk;
        a[9] += dx * dz * wk;
        a[10] += wk * dx;
        a[11] += wk * dy;
        a[12] += wk * dz;
        const double dvx = t.vx - vjx, dvy = t.vy - vjy, dvz = t.vz - vjz;
        if (mfv) {
            a[14] += mj_wk * (t.vx - dvx);
            a[15] += mj_wk * (t.vy - dvy);
            a[16] += mj_wk * (t.vz - dvz);
        }
        a[3] -= dwk * (dx * dvx + dy * dvy + dz * dvz) / r;
    }
}

// One target per lane: a block holds the 32 targets of a run. Its warps first test
// the boxes of all runs and list the ones the targets can reach; then each warp
// takes kShare candidates of every listed run (so the work, which is concentrated
// in the few nearest runs, is spread over the warps) and screens 32 candidates at
// a time: a broadcast shared-memory read and ~14 FP32 instructions a pair, no
// branch, the outcomes the bits of a mask. The candidates that pass are collected
// in shared memory and evaluated together, so the FP64 arithmetic runs with most
// lanes busy although few of the scanned pairs need it; the warps' sums are added
// at the end in a fixed order. A pair is rejected only when its FP32 separation is
// beyond |h| by more than the margin; NaNs are never rejected.
//
// What bounds it: the latency of a block's chain (run list, screen, evaluation),
// not throughput. Measured on a clustered MFV set (whole call, sort included): 66,
// 248 and 533 us at 1,000, 20,000 and 65,536 particles, against 473, 5,945 and
// 18,300 us with one thread per target testing every pair in FP64 (157 blocks of
// 128 at 20,000: four warps per multiprocessor, each taking the sums for one or two
// of its lanes at a time). The alternatives were compared on another such set, at
// 57, 250 and 459 us for this form: four warps a block 82, 332 and 544 us; eight at
// three blocks per multiprocessor (80 registers, spills) 66, 292 and 514; all pairs
// screened, without the order and the boxes, 27, 404 and 2,803.
__global__ void __launch_bounds__(32 * kSlices, 2) k_noalloc_density_sums(PassParams p, int n,
                                                                          const double *__restrict__ pos,
                                                                          const double *__restrict__ vel,
                                                                          const double *__restrict__ mass,
                                                                          const double *__restrict__ hs, SumsWork w,
                                                                          double *acc, double *pv)
{
    constexpr int kThreads = 32 * kSlices;
    // the scan's tiles and hits, then (in the same place) the slices' sums
    struct Scan {
        float4 tile[kSlices][32];
        unsigned short hit[kHits][kThreads];
    };
    __shared__ union {
        Scan scan;
        double sum[kSlices][17][32];
    } sh;
    __shared__ unsigned short s_run[kMaxParticles / kRun];  // the reached runs, ascending
    __shared__ int s_cnt[kSlices];
    __shared__ unsigned s_top;  // largest coordinate magnitude among them
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int s = blockIdx.x * kRun + lane;
    const bool valid = s < n;
    const int sv = valid ? s : n - 1;  // a lane past the end follows the last target and stores nothing
    const size_t i = (size_t)own_index(w.order[sv], n);
    Target me;
    me.x = pos[3 * i]; me.y = pos[3 * i + 1]; me.z = pos[3 * i + 2];
    me.vx = vel[3 * i]; me.vy = vel[3 * i + 1]; me.vz = vel[3 * i + 2];
    const double hd = hs[i];
    me.h2 = hd * hd;
    double hinv3, hinv4;
    k_hinv(hd, me.hinv, hinv3, hinv4);
    double a[17];
#pragma unroll
    for (int k = 0; k < 17; k++) a[k] = 0;

    // The collected candidates. Usually every lane evaluates its own; a target
    // that holds far more than the others (a long kernel that reaches into a
    // clump) would keep one lane busy and the rest idle, so the warp evaluates
    // its candidates together, one per lane, and adds the sums across the lanes.
    int hits = 0;
    const SumsInput in{pos, vel, mass};
    auto evaluate = [&]() {
        unsigned many = __ballot_sync(full, hits > kFewHits);
        // (in units of a lane's own evaluation: a shared one costs about three with its cross-lane sums)
        if (__popc(many) * 3 > __reduce_max_sync(full, hits) - kFewHits) many = 0u;
        for (; many; many &= many - 1u) {
            const int tl = __ffs(many) - 1;
            Target t;
            t.x = __shfl_sync(full, me.x, tl); t.y = __shfl_sync(full, me.y, tl); t.z = __shfl_sync(full, me.z, tl);
            t.vx = __shfl_sync(full, me.vx, tl); t.vy = __shfl_sync(full, me.vy, tl); t.vz = __shfl_sync(full, me.vz, tl);
            t.h2 = __shfl_sync(full, me.h2, tl); t.hinv = __shfl_sync(full, me.hinv, tl);
            double b[17];
#pragma unroll
            for (int k = 0; k < 17; k++) b[k] = 0;
            if (lane < __shfl_sync(full, hits, tl)) add_pair(p, in, t, sh.scan.hit[lane][(threadIdx.x & ~31) + tl], b);
#pragma unroll
            for (int k = 0; k < 17; k++) {
                const double v = warp_sum(b[k], full, 32);
                if (lane == tl) a[k] += v;
            }
            if (lane == tl) hits = 0;
        }
        const int most = __reduce_max_sync(full, hits);
        for (int k = 0; k < most; k++)
            if (k < hits) add_pair(p, in, me, sh.scan.hit[k][threadIdx.x], a);
        hits = 0;
        __syncwarp();
    };

    const float4 mf = w.pos[sv];
    const RunBox mine = w.box[blockIdx.x];
    const float hf = __double2float_ru(fabs(hd) / p.box);
    const int runs = (n + kRun - 1) / kRun;
    // the runs the targets can reach
    if (threadIdx.x == 0) s_top = 0u;
    int reached = 0;
    for (int q0 = 0; q0 < runs; q0 += kThreads) {
        const int q = q0 + (int)threadIdx.x;
        bool in = false;
        float top = 0.0f;
        if (q < runs) {
            const RunBox b = w.box[q];
            top = b.lo.w;
            const float R = mine.hi.w + screen_margin(fmaxf(mine.lo.w, top));
            const float gx = axis_distance(mine.lo.x - b.hi.x, mine.hi.x - b.lo.x);
            const float gy = axis_distance(mine.lo.y - b.hi.y, mine.hi.y - b.lo.y);
            const float gz = axis_distance(mine.lo.z - b.hi.z, mine.hi.z - b.lo.z);
            in = !(gx * gx + gy * gy + gz * gz > R * R * 1.000001f);
        }
        const unsigned bal = __ballot_sync(full, in);
        const unsigned tmax = __reduce_max_sync(full, in ? __float_as_uint(top) : 0u);
        __syncthreads();  // s_cnt of the last round has been read
        if (lane == 0) {
            s_cnt[slice] = __popc(bal);
            if (bal) atomicMax(&s_top, tmax);  // (magnitudes are not negative: their bits order like them)
        }
        __syncthreads();
        int at = reached;
#pragma unroll
        for (int k = 0; k < kSlices; k++) {
            if (k < slice) at += s_cnt[k];
            reached += s_cnt[k];
        }
        if (in) s_run[at + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)q;
    }
    __syncthreads();
    const float hi = hf + screen_margin(fmaxf(__uint_as_float(s_top), mine.lo.w));
    const float hi2 = hi * hi * 1.000001f;
    for (int q0 = 0; q0 < reached; q0 += kSlices) {
        const int ql = q0 + lane / kShare;
        int c = n;
        if (ql < reached) c = s_run[ql] * kRun + slice * kShare + lane % kShare;
        const unsigned have = __ballot_sync(full, c < n);
        if (c < n) sh.scan.tile[slice][lane] = w.pos[c];
        __syncwarp();
        unsigned pass = 0;
#pragma unroll
        for (int k = 0; k < 32; k++) {
            const float4 q = sh.scan.tile[slice][k];
            // the minimum image's magnitude: |d|, or 1 - |d| beyond half the box (squared below)
            float dx = fabsf(mf.x - q.x), dy = fabsf(mf.y - q.y), dz = fabsf(mf.z - q.z);
            dx = fminf(dx, 1.0f - dx);
            dy = fminf(dy, 1.0f - dy);
            dz = fminf(dz, 1.0f - dz);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (!(r2 > hi2)) pass |= 1u << k;
        }
        pass &= have;
        while (__any_sync(full, pass != 0u)) {
            if (pass) {
                const int k = __ffs(pass) - 1;
                sh.scan.hit[hits++][threadIdx.x] = (unsigned short)own_index(__float_as_int(sh.scan.tile[slice][k].w), n);
                pass &= pass - 1u;
            }
            __syncwarp();
            if (__any_sync(full, hits == kHits)) evaluate();
        }
        __syncwarp();  // the tile has been read
    }
    evaluate();

    // the slices' sums, added in slice order, one sum at a time per warp
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 17; k++) sh.sum[slice][k][lane] = a[k];
    __syncthreads();
    for (int k = slice; k < 17; k += kSlices) {
        double v = sh.sum[0][k][lane];
#pragma unroll
        for (int q = 1; q < kSlices; q++) v += sh.sum[q][k][lane];
        if (!valid) continue;
        if (k < 13) acc[14 * i + k] = v;
        else if (k == 13) acc[14 * i + 13] = 0.0;
        else if (pv) pv[3 * i + (k - 14)] = v;
    }
}

// Device address of g_scratch on the current device, looked up once per device
// (host code must not pass the symbol itself: on the host it names a stand-in,
// not device memory).
int scratch_address(Scratch **out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return GZ_ERR_NO_DEVICE;
    if (dev < 0 || dev >= kMaxDevices) return GZ_ERR_ARG;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_ptr[dev]) {
        void *q = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&q, g_scratch);
        if (e != cudaSuccess || !q) return GZ_ERR_CUDA;
        g_scratch_ptr[dev] = (Scratch *)q;
    }
    *out = g_scratch_ptr[dev];
    return GZ_OK;
}

}  // namespace

extern "C" int gz_density_sums_noalloc(const gz_params *params, int n, const double *pos, const double *vel,
                                       const double *mass, const double *h, double *acc, double *pv, void *stream)
{
    if (!params || n < 0) return GZ_ERR_ARG;
    if (params->kernel != GZ_KERNEL_CUBIC && params->kernel != GZ_KERNEL_WENDLAND_C2) return GZ_ERR_ARG;
    if (params->method != GZ_METHOD_MFM && params->method != GZ_METHOD_MFV) return GZ_ERR_ARG;
    if (!(params->box_size > 0)) return GZ_ERR_ARG;
    if (n > kMaxParticles) return GZ_ERR_CAPACITY;
    if (n == 0) return GZ_OK;
    if (!pos || !vel || !mass || !h || !acc) return GZ_ERR_ARG;
    Scratch *g = nullptr;
    const int rc = scratch_address(&g);
    if (rc) return rc;
    PassParams p{};
    p.kernel = params->kernel;
    p.method = params->method;
    p.first_step = params->first_step;
    p.selfgravity_off = params->selfgravity_off;
    p.box = params->box_size;
    p.half = 0.5 * params->box_size;
    p.gamma = params->gamma;
    p.des_num_ngb = params->des_num_ngb;
    p.max_num_ngb_dev = params->max_num_ngb_dev;
    p.min_kernel_radius = params->min_kernel_radius;
    p.max_kernel_radius = params->max_kernel_radius;
    cudaStream_t s = (cudaStream_t)stream;
    k_noalloc_sort<<<kSortBlocks, 32 * kSortWarps, 0, s>>>(n, pos, p.box, g);
    k_noalloc_runs<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(n, pos, h, p.box, g->order[0], g->pos, g->box);
    const SumsWork w{g->order[0], g->pos, g->box};
    k_noalloc_density_sums<<<(unsigned)((n + kRun - 1) / kRun), 32 * kSlices, 0, s>>>(p, n, pos, vel, mass, h, w, acc,
                                                                                     pv);
    return cudaGetLastError() == cudaSuccess ? GZ_OK : GZ_ERR_CUDA;
}
