// tis_pair_lists_noalloc: the cell binning and SR/LR pair-list build of
// populate_lists (E:1461-1694 of src/16SCD_Mg_Cl_K_COPY_fast.cpp) for one
// configuration held in caller-owned device memory, without allocating.
//
// Why it exists: some callers cannot allocate device memory at the point they
// need a list.  A host whose CUDA work is being captured into a graph cannot
// call cudaMalloc (it is not a capturable operation), cudaFree synchronises the
// whole device, and engines that embed this library in their own time step often
// run under a fixed memory budget with every buffer reserved up front.  This
// entry point therefore takes only caller buffers and keeps its scratch (cell
// counts, offsets and the cell-sorted particle list) in a file-scope __device__
// array that every GPU loading the library holds until the process exits.
//
// Limits: at most kNaMaxParticles particles and kNaMaxCells cells.  All calls
// share the one scratch array, so calls that overlap on the GPU (different
// streams, or different host threads on one device) race and must be ordered
// by the caller.  The first call on a device looks up the array's device
// address (cudaGetSymbolAddress) with that device current; make that first call
// before any stream capture begins.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "tis_device.cuh"
#include "tis_host.h"

namespace {

constexpr int kNaMaxParticles = 65536;
constexpr int kNaMaxCells = 32768;
constexpr int kNaThreads = 128;
// scratch layout (ints): count[kNaMaxCells] | start[kNaMaxCells] | unused[kNaMaxCells] |
//                        where[kNaMaxParticles] | sorted[kNaMaxParticles]
// where: a particle's cell and its rank among the cell's particles (na_where)
constexpr size_t kNaScratchInts = 3 * (size_t)kNaMaxCells + 2 * (size_t)kNaMaxParticles;  // 896 KiB

static __device__ __align__(256) int g_na_scratch[kNaScratchInts];

struct NaArgs {
    const double *x, *y, *z;
    const int *kind;
    int n;
    double box[3], hbox[3], lcell[3];
    int mc[3], nc;
    double r2sr, r2lr;
    float boxf[3], hboxf[3], r2f[4];  // FP32 box; r2f: below [0] SR, above [1] not SR, below [2] within LR, above [3] not
    int half;                         // three or more cells per axis: each pair of cells met once
    int *sr, *lr;
    long long sr_cap, lr_cap;
    unsigned long long *counts;  // caller's device [SR pairs, LR pairs, particles outside the grid]
    int *scratch;
};

__device__ inline int na_axis(double v, double side, double l)
{
    double t = v;
    if (t < 0) t = __dadd_rn(t, side);
    else if (t > side) t = __dsub_rn(t, side);
    return (int)ceil(__ddiv_rn(t, l));
}

// cell (15 bits) and rank (16 bits) of a particle in one int; -1: outside the grid
static_assert(kNaMaxCells <= 1 << 15 && kNaMaxParticles <= 1 << 16, "na_where");
__device__ inline int na_where(int cell, int rank) { return cell | (rank << 15); }

__global__ void k_na_clear(NaArgs a)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nc; i += gridDim.x * blockDim.x) a.scratch[i] = 0;
    if (blockIdx.x == 0 && threadIdx.x < 3) a.counts[threadIdx.x] = 0ull;
}

__global__ void k_na_assign(NaArgs a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    int *count = a.scratch, *where = a.scratch + 3 * kNaMaxCells;
    const int i1 = na_axis(a.x[p], a.box[0], a.lcell[0]);
    const int i2 = na_axis(a.y[p], a.box[1], a.lcell[1]);
    const int i3 = na_axis(a.z[p], a.box[2], a.lcell[2]);
    if (i1 < 1 || i1 > a.mc[0] || i2 < 1 || i2 > a.mc[1] || i3 < 1 || i3 > a.mc[2]) {
        where[p] = -1;  // beyond the single periodic wrap of separate_in_cells: left out, and counted
        atomicAdd(a.counts + 2, 1ull);
        return;
    }
    const int c = (i1 - 1) * a.mc[1] * a.mc[2] + (i2 - 1) * a.mc[2] + (i3 - 1);
    where[p] = na_where(c, atomicAdd(count + c, 1));
}

constexpr int kNaScanThreads = 1024;

// one block: exclusive scan of the cell counts, a run of consecutive cells per thread
__global__ void __launch_bounds__(kNaScanThreads) k_na_scan(NaArgs a)
{
    const int *count = a.scratch;
    int *start = a.scratch + kNaMaxCells;
    __shared__ int s_warp[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int per = (a.nc + kNaScanThreads - 1) / kNaScanThreads, c0 = tid * per, c1 = min(a.nc, c0 + per);
    int sum = 0;
    for (int c = c0; c < c1; ++c) sum += count[c];
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        int t = s_warp[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        s_warp[lane] = t;
    }
    __syncthreads();
    int at = (w > 0 ? s_warp[w - 1] : 0) + incl - sum;
    for (int c = c0; c < c1; ++c) {
        start[c] = at;
        at += count[c];
    }
}

__global__ void k_na_fill(NaArgs a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const int *start = a.scratch + kNaMaxCells, *where = a.scratch + 3 * kNaMaxCells;
    int *sorted = a.scratch + 3 * kNaMaxCells + kNaMaxParticles;
    const int w = where[p];
    if (w >= 0) sorted[start[w & (kNaMaxCells - 1)] + (w >> 15)] = p;
}

__device__ inline double na_r2(const NaArgs &a, int i, int j)  // CC_vector + r^2 (E:674-683)
{
    double v[3] = {__dsub_rn(a.x[i], a.x[j]), __dsub_rn(a.y[i], a.y[j]), __dsub_rn(a.z[i], a.z[j])};
    for (int k = 0; k < 3; ++k) {
        if (v[k] > a.hbox[k]) v[k] = __dsub_rn(v[k], a.box[k]);
        if (v[k] < -a.hbox[k]) v[k] = __dadd_rn(v[k], a.box[k]);
    }
    return __dadd_rn(__dadd_rn(__dmul_rn(v[0], v[0]), __dmul_rn(v[1], v[1])), __dmul_rn(v[2], v[2]));
}

constexpr int kNaWarps = 4, kNaBuf = 64;

// x as a float, its significand cut to 24 bits, by integers (0 below 2^-126; coordinates are below 2^128)
__device__ __forceinline__ float na_float(double x)
{
    const int hi = __double2hiint(x), m = hi & 0x7fffffff;
    const int f = __funnelshift_l((unsigned)__double2loint(x), (unsigned)(m - 0x38000000), 3);
    return __int_as_float((m < 0x38100000 ? 0 : f & 0x7fffffff) | (hi & 0x80000000));
}

// pairs found by a warp, written out 32 at a time: one atomic on the pair count and one
// coalesced store per 32 pairs
struct NaBuf {
    int2 pair[kNaBuf];
};

__device__ __forceinline__ void na_flush(NaBuf &b, int &held, int n, unsigned long long *count, int *out, long long cap,
                                         int lane)
{
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(count, (unsigned long long)n);
    at = __shfl_sync(0xffffffffu, at, 0);
    __syncwarp();  // the warp's pairs are in the buffer
    if (lane < n) {
        const long long s = (long long)at + lane;
        if (s < cap) {  // the caller's array is aligned to its ints only
            out[2 * s] = b.pair[lane].x;
            out[2 * s + 1] = b.pair[lane].y;
        }
    }
    __syncwarp();
    const int2 rest = lane + n < held ? b.pair[lane + n] : make_int2(0, 0);
    __syncwarp();
    if (lane + n < held) b.pair[lane] = rest;
    held -= n;
}

__device__ __forceinline__ void na_add(NaBuf &b, int &held, bool hit, int p, int j, unsigned long long *count, int *out,
                                       long long cap, int lane)
{
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (!m) return;
    if (hit) b.pair[held + __popc(m & ((1u << lane) - 1u))] = make_int2(min(p, j), max(p, j));
    held += __popc(m);  // at most 31 + 32
    if (held >= 32) na_flush(b, held, 32, count, out, cap, lane);
}

// Every unordered pair once: SR when r^2 <= r2sr, else LR when r^2 <= r2lr and neither bead
// is a sugar or a base (E:1626-1644).  A warp per particle, in cell order so that the
// warps of a block read the same candidates; its neighbour cells (a lane each; the later
// half of them and the particles behind it in its own where the grid has three or more
// cells per axis) are scanned end to end, 32 candidates at a time.  FP32 distances decide
// outside a band around the radii, FP64 ones with the reference's rounding inside it: the
// FP64 pipe bound the former version, a thread per particle over all 27 cells, at 3.0 ms
// for 45,922 particles; this one takes 0.09 ms.
__global__ void __launch_bounds__(32 * kNaWarps) k_na_pairs(NaArgs a)
{
    __shared__ NaBuf s_buf[kNaWarps][2];
    __shared__ int s_seg[kNaWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned le = (2u << lane) - 1u;
    const int *count = a.scratch, *start = a.scratch + kNaMaxCells;
    const int *where = a.scratch + 3 * kNaMaxCells, *sorted = where + kNaMaxParticles;
    const int m1 = a.mc[0], m2 = a.mc[1], m3 = a.mc[2], n = a.n - (int)a.counts[2];
    int sr = 0, lr = 0;
    for (int s0 = blockIdx.x * kNaWarps + w; s0 < n; s0 += gridDim.x * kNaWarps) {
        const int p = sorted[s0], c = where[p] & (kNaMaxCells - 1);
        const float xf = na_float(a.x[p]), yf = na_float(a.y[p]), zf = na_float(a.z[p]);
        const int kp = a.kind[p];
        const bool chp = kp != 1 && kp != 2;
        int cnt = 0, at = 0;
        if (lane < 27 && (!a.half || lane >= 13)) {
            const int d1 = lane / 9 - 1, d2 = (lane / 3) % 3 - 1, d3 = lane % 3 - 1;
            if (d1 <= min(m1, 3) - 2 && d2 <= min(m2, 3) - 2 && d3 <= min(m3, 3) - 2) {  // each cell of a small grid once
                int u = c / (m2 * m3) + d1, v = (c / m3) % m2 + d2, e = c % m3 + d3;
                u += u < 0 ? m1 : u >= m1 ? -m1 : 0;
                v += v < 0 ? m2 : v >= m2 ? -m2 : 0;
                e += e < 0 ? m3 : e >= m3 ? -m3 : 0;
                const int cc = (u * m2 + v) * m3 + e;
                at = start[cc];
                cnt = count[cc];
                if (a.half && lane == 13) {  // its own cell: those behind it
                    cnt -= s0 + 1 - at;
                    at = s0 + 1;
                }
            }
        }
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31), first = incl - cnt;
        const unsigned has = __ballot_sync(0xffffffffu, cnt > 0);
        __syncwarp();
        if (cnt > 0) s_seg[w][__popc(has & (le >> 1))] = at - first;
        __syncwarp();
        int before = 0;
        for (int t0 = 0; t0 < total; t0 += 32) {
            const unsigned rel = (unsigned)(first - t0);
            const unsigned begins = __reduce_or_sync(0xffffffffu, cnt > 0 && rel < 32u ? 1u << rel : 0u);
            const int t = t0 + lane;
            int j = -1, cls = 0;
            if (t < total) {
                j = sorted[s_seg[w][before + __popc(begins & le) - 1] + t];
                if (a.half || j > p) {
                    const int kj = a.kind[j];
                    float v[3] = {xf - na_float(a.x[j]), yf - na_float(a.y[j]), zf - na_float(a.z[j])};
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        v[k] = v[k] > a.hboxf[k] ? v[k] - a.boxf[k] : v[k];
                        v[k] = v[k] < -a.hboxf[k] ? v[k] + a.boxf[k] : v[k];
                    }
                    const float r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
                    const bool ch = chp && kj != 1 && kj != 2;
                    if (r2 < a.r2f[0]) cls = 1;
                    else if (r2 > a.r2f[1] && (!ch || r2 > a.r2f[3])) cls = 0;
                    else if (r2 > a.r2f[1] && r2 < a.r2f[2]) cls = 2;
                    else {
                        const double e2 = na_r2(a, p, j);
                        cls = e2 <= a.r2sr ? 1 : ch && e2 <= a.r2lr ? 2 : 0;
                    }
                }
            }
            before += __popc(begins);
            na_add(s_buf[w][0], sr, cls == 1, p, j, a.counts, a.sr, a.sr_cap, lane);
            na_add(s_buf[w][1], lr, cls == 2, p, j, a.counts + 1, a.lr, a.lr_cap, lane);
        }
    }
    if (sr) na_flush(s_buf[w][0], sr, sr, a.counts, a.sr, a.sr_cap, lane);
    if (lr) na_flush(s_buf[w][1], lr, lr, a.counts + 1, a.lr, a.lr_cap, lane);
}

std::mutex g_na_mutex;
int *g_na_ptr[64] = {nullptr};

}  // namespace

extern "C" int tis_pair_lists_noalloc(const double *d_x, const double *d_y, const double *d_z, const int32_t *d_kind,
                                      int32_t n, const double *box, double sr_radius, double lr_radius,
                                      int32_t *d_sr_pairs, int64_t sr_cap, int32_t *d_lr_pairs, int64_t lr_cap,
                                      uint64_t *d_counts, void *stream)
{
    using tis::fail;
    if (!d_x || !d_y || !d_z || !d_kind || !box || !d_counts || n < 0 || sr_cap < 0 || lr_cap < 0 ||
        (sr_cap > 0 && !d_sr_pairs) || (lr_cap > 0 && !d_lr_pairs))
        return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: bad argument");
    if (!(sr_radius > 0) || !(lr_radius >= sr_radius))
        return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: need 0 < sr_radius <= lr_radius");
    if (n > kNaMaxParticles)
        return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: %d particles exceed the fixed limit of %d", n, kNaMaxParticles);
    NaArgs a;
    memset(&a, 0, sizeof a);
    a.nc = 1;
    for (int k = 0; k < 3; ++k) {
        if (!(box[k] > 0)) return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: box side %d not positive", k);
        a.box[k] = box[k];
        a.hbox[k] = 0.5 * box[k];
        a.mc[k] = (int)(box[k] / lr_radius);  // E:1484-1490
        if (a.mc[k] < 1) return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: box side %d below the LR radius", k);
        a.lcell[k] = box[k] / a.mc[k];
        if ((long long)a.nc * a.mc[k] > kNaMaxCells)
            return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: more than %d cells; use a larger LR radius or smaller box",
                        kNaMaxCells);
        a.nc *= a.mc[k];
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(TIS_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return fail(TIS_ERR_ARG, "tis_pair_lists_noalloc: device %d out of range", dev);
    {
        std::lock_guard<std::mutex> lk(g_na_mutex);
        if (!g_na_ptr[dev]) {  // set-up, once per device, with that device current
            void *ptr = nullptr;
            e = cudaGetSymbolAddress(&ptr, g_na_scratch);
            if (e != cudaSuccess) return fail(TIS_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
            g_na_ptr[dev] = (int *)ptr;
        }
    }
    a.scratch = g_na_ptr[dev];
    a.x = d_x;
    a.y = d_y;
    a.z = d_z;
    a.kind = d_kind;
    a.n = n;
    a.r2sr = sr_radius * sr_radius;
    a.r2lr = lr_radius * lr_radius;
    a.sr = d_sr_pairs;
    a.lr = d_lr_pairs;
    a.sr_cap = sr_cap;
    a.lr_cap = lr_cap;
    a.counts = (unsigned long long *)d_counts;
    cudaStream_t s = (cudaStream_t)stream;
    // FP32 thresholds: a coordinate difference formed from cut FP32 coordinates of magnitude
    // up to 2 L, imaged with a rounded box, is off by at most e = 4 L 2^-22, and by twice that
    // where it lies so near L / 2 that the other image is taken; r^2 is then off by at most
    // 4 sqrt(3) r e + 12 e^2 and a few roundings (1e-6 r^2)
    double longest = 0;
    for (int k = 0; k < 3; ++k) {
        a.boxf[k] = (float)a.box[k];
        a.hboxf[k] = (float)a.hbox[k];
        longest = std::max(longest, a.box[k]);
        a.half = (k == 0 || a.half) && a.mc[k] >= 3;
    }
    const double off = 4.0 * longest * std::ldexp(1.0, -22);
    auto band = [&](double r2) { return 8.0 * sqrt(r2) * off + 12.0 * off * off + 1.0e-6 * r2; };
    a.r2f[0] = (float)((a.r2sr - band(a.r2sr)) * (1.0 - 1.0e-6));
    a.r2f[1] = (float)((a.r2sr + band(a.r2sr)) * (1.0 + 1.0e-6));
    a.r2f[2] = (float)((a.r2lr - band(a.r2lr)) * (1.0 - 1.0e-6));
    a.r2f[3] = (float)((a.r2lr + band(a.r2lr)) * (1.0 + 1.0e-6));
    // the shared scratch keeps the last call's contents: the counters that must start at zero are cleared
    k_na_clear<<<std::min(64, (a.nc + 255) / 256), 256, 0, s>>>(a);
    if (n > 0) {
        const int nb = (n + kNaThreads - 1) / kNaThreads;
        k_na_assign<<<nb, kNaThreads, 0, s>>>(a);
        k_na_scan<<<1, kNaScanThreads, 0, s>>>(a);
        k_na_fill<<<nb, kNaThreads, 0, s>>>(a);
        // two particles per warp, at most
        k_na_pairs<<<std::max(1, std::min(4096, (n + 2 * kNaWarps - 1) / (2 * kNaWarps))), 32 * kNaWarps, 0, s>>>(a);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TIS_ERR_CUDA, "tis_pair_lists_noalloc launch: %s", cudaGetErrorString(e));
    return TIS_OK;
}
