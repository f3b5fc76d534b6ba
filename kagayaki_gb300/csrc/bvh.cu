// bvh.cu - GPU binned-SAH BVH build and collapse into 8-wide compressed
// nodes.  Replaces the host build construct_BVH / Divide_AABB
// (ConstructBVH.cuh:13-207) and the per-node cudaMalloc upload
// (struct_BVH_node.cuh:72-83).
//
// Pipeline (all on the device stream; the host only orders the launches):
//   1. primitive boxes + scene bounds;
//   2. large tasks (> kSmall primitives): one level at a time, many blocks per
//      task: 32-bin centroid binning per axis (shared-memory atomics merged
//      into per-task global bins), one warp evaluates SAH over the 3 x 31
//      planes, a stable partition by chunks (warp ballots over the bin codes)
//      reorders the refs;
//   3. small tasks (<= kSmall): one block builds the whole subtree in shared
//      memory, a warp per node, nodes of at most 32 primitives one primitive
//      per lane; a split's place among the refs names its children's node
//      slots, so the tree is deterministic;
//   4. collapse: a bottom-up pass fills the SAH cost table of the optimal
//      collapse (k_dp_*); then breadth first, every wide node takes the 8
//      children that table chose; children with at most 1 (large scenes) or 3
//      (small ones) triangles are leaf children; slots are ordered by octant so traversal visits near
//      children first; child boxes are quantised to 8 bits against the parent
//      box (conservative rounding).
// Every kernel bounds-checks its writes and raises an error flag instead of
// writing out of range.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <utility>
#include <vector>

#include <cooperative_groups.h>

#include "kgk_device.cuh"
#include "kgk_internal.h"

namespace cg = cooperative_groups;

namespace kgk {
namespace {

constexpr int kBins = 32;
// Primitives per block in the large-task path: enough blocks for the chip on
// small scenes, fewer merges of block bins into task bins on large ones
// (build at 1024 / 4096 per block: 2.28 / 2.43 ms for 82k triangles, 13.0 /
// 12.2 ms for 5.2M; the line is where 4096 still fills the chip).
constexpr int kChunkSmall = 1024, kChunkLarge = 4096;
constexpr int kLargeChunkTris = 1 << 20;
constexpr int kSmall = 2048;   // tasks up to this size build inside one block
// Triangles per leaf child of a wide node, chosen per scene (bvh_build).
// One for large scenes: a wide node's leaf children then hold a triangle
// each, so its quantised child box culls that triangle alone, and a node
// yields at most 8 triangle tests.  Measured on the C2 frame (5.2M
// triangles): 3089 Mrays/s at 1, 2978 at 2, 2799 at 3 (extend 43.5 / 46.0 /
// 50.3 ms), for 1.72M / 1.00M / 0.71M wide nodes.  Three for small scenes, whose nodes and triangles stay in cache:
// the 36-triangle Cornell box (C1) runs 1509 Mrays/s at 3, 1156 at 1.
constexpr int kMaxLeaf = 3;                // the largest leaf the node format holds (8 x 3 = 24 bits)
constexpr int kLeafLarge = 1;
constexpr int kLargeSceneTris = 1 << 16;   // scenes above this use kLeafLarge
constexpr int kThreads = 256;
constexpr int kBinInts = 13;   // count, box lo/hi, centroid lo/hi (ordered ints)

enum BuildError : int {
    kErrNone = 0,
    kErrSmallTooBig = 1,
    kErrNodeOverflow = 2,
    kErrStackOverflow = 3,
    kErrWideOverflow = 4,
    kErrTriOverflow = 5,
    kErrBadChild = 6,
};

struct Task {
    int node, begin, count;
    int buf;  // which of the two ref buffers holds its refs
    float clo[3], chi[3];
    int first_chunk, pad;  // a large task's chunks follow each other
};

struct Split {
    int axis;   // -1: split by position
    int bin;
    int nleft;
    int pad;
    float lo[2][3], hi[2][3];    // child boxes (0 = left, 1 = right)
    float clo[2][3], chi[2][3];  // child centroid bounds
};

__device__ __forceinline__ void raise_err(int *err, int code) { atomicCAS(err, 0, code); }

__device__ __forceinline__ int bin_of(float c, float lo, float scale) {
    int b = (int)((c - lo) * scale);
    return b < 0 ? 0 : (b >= kBins ? kBins - 1 : b);
}

// Bin scale of one axis: kBins / extent, 0 for a flat axis.
__device__ __forceinline__ float bin_scale(float lo, float hi) {
    float e = hi - lo;
    return e > 0.0f ? (float)kBins / e : 0.0f;
}

__device__ __forceinline__ float3 centroid(float4 lo, float4 hi) {
    return f3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
}

__device__ __forceinline__ float3 warp_min3(float3 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmin3(v, f3(__shfl_xor_sync(~0u, v.x, o), __shfl_xor_sync(~0u, v.y, o), __shfl_xor_sync(~0u, v.z, o)));
    return v;
}
__device__ __forceinline__ float3 warp_max3(float3 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmax3(v, f3(__shfl_xor_sync(~0u, v.x, o), __shfl_xor_sync(~0u, v.y, o), __shfl_xor_sync(~0u, v.z, o)));
    return v;
}

// ---------------------------------------------------------------------------
// 1. primitive boxes
// ---------------------------------------------------------------------------
__global__ void k_init_bounds(int *g) {
    int i = threadIdx.x;
    if (i < 12) g[i] = (i % 6) < 3 ? f2o(INFINITY) : f2o(-INFINITY);
}

// A few resident blocks, each walking the triangles and adding its bounds to
// the scene's once.  With twelve atomics per warp on the same twelve words the
// kernel took 1.37 ms at 5.2M triangles; now it reads and writes at the memory's
// rate (0.066 ms for 437 MB).
__global__ void __launch_bounds__(256) k_prim_bounds(const float4 *__restrict__ verts, int n, float4 *plo,
                                                     float4 *phi, int *ref, int *gbounds) {
    __shared__ int sb[12];
    if (threadIdx.x < 12) sb[threadIdx.x] = threadIdx.x % 6 < 3 ? f2o(INFINITY) : f2o(-INFINITY);
    __syncthreads();
    float3 slo = f3(INFINITY, INFINITY, INFINITY), shi = f3(-INFINITY, -INFINITY, -INFINITY);
    float3 clo = slo, chi = shi;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 a = f3(verts[3 * (size_t)i]), b = f3(verts[3 * (size_t)i + 1]), c = f3(verts[3 * (size_t)i + 2]);
        const float3 lo = fmin3(a, fmin3(b, c)), hi = fmax3(a, fmax3(b, c));
        plo[i] = f4(lo, 0.0f);
        phi[i] = f4(hi, 0.0f);
        ref[i] = i;
        const float3 q = f3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
        slo = fmin3(slo, lo);
        shi = fmax3(shi, hi);
        clo = fmin3(clo, q);
        chi = fmax3(chi, q);
    }
    const float3 lo[2] = {warp_min3(slo), warp_min3(clo)}, hi[2] = {warp_max3(shi), warp_max3(chi)};
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            atomicMin(&sb[6 * k], f2o(lo[k].x)); atomicMin(&sb[6 * k + 1], f2o(lo[k].y));
            atomicMin(&sb[6 * k + 2], f2o(lo[k].z));
            atomicMax(&sb[6 * k + 3], f2o(hi[k].x)); atomicMax(&sb[6 * k + 4], f2o(hi[k].y));
            atomicMax(&sb[6 * k + 5], f2o(hi[k].z));
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        if (threadIdx.x % 6 < 3) atomicMin(&gbounds[threadIdx.x], sb[threadIdx.x]);
        else atomicMax(&gbounds[threadIdx.x], sb[threadIdx.x]);
    }
}

// ---------------------------------------------------------------------------
// Split evaluation by one warp over bins[3][kBins][kBinInts].
// ---------------------------------------------------------------------------
struct WarpSplit {
    int axis, bin;
    float cost;
};

__device__ __forceinline__ float3 shfl_up3(float3 v, int o) {
    return f3(__shfl_up_sync(~0u, v.x, o), __shfl_up_sync(~0u, v.y, o), __shfl_up_sync(~0u, v.z, o));
}
__device__ __forceinline__ float3 shfl_down3(float3 v, int o) {
    return f3(__shfl_down_sync(~0u, v.x, o), __shfl_down_sync(~0u, v.y, o), __shfl_down_sync(~0u, v.z, o));
}

// Scans one axis: on return lane b holds left (bins 0..b) and right
// (bins b+1..31) counts/boxes/centroid boxes.
struct AxisScan {
    int lc, rc;
    float3 llo, lhi, rlo, rhi, lclo, lchi, rclo, rchi;
};

__device__ AxisScan scan_axis(const int *bins, int axis) {
    const int lane = threadIdx.x & 31;
    const int *B = bins + (axis * kBins + lane) * kBinInts;
    int cnt = B[0];
    float3 lo = f3(o2f(B[1]), o2f(B[2]), o2f(B[3])), hi = f3(o2f(B[4]), o2f(B[5]), o2f(B[6]));
    float3 clo = f3(o2f(B[7]), o2f(B[8]), o2f(B[9])), chi = f3(o2f(B[10]), o2f(B[11]), o2f(B[12]));
    int pc = cnt, sc = cnt;
    float3 plo = lo, phi = hi, pclo = clo, pchi = chi;
    float3 slo = lo, shi = hi, sclo = clo, schi = chi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int a = __shfl_up_sync(~0u, pc, o);
        float3 alo = shfl_up3(plo, o), ahi = shfl_up3(phi, o), aclo = shfl_up3(pclo, o), achi = shfl_up3(pchi, o);
        int b = __shfl_down_sync(~0u, sc, o);
        float3 blo = shfl_down3(slo, o), bhi = shfl_down3(shi, o), bclo = shfl_down3(sclo, o), bchi = shfl_down3(schi, o);
        if (lane >= o) {
            pc += a; plo = fmin3(plo, alo); phi = fmax3(phi, ahi); pclo = fmin3(pclo, aclo); pchi = fmax3(pchi, achi);
        }
        if (lane + o < 32) {
            sc += b; slo = fmin3(slo, blo); shi = fmax3(shi, bhi); sclo = fmin3(sclo, bclo); schi = fmax3(schi, bchi);
        }
    }
    AxisScan r;
    r.lc = pc; r.llo = plo; r.lhi = phi; r.lclo = pclo; r.lchi = pchi;
    r.rc = __shfl_down_sync(~0u, sc, 1);
    r.rlo = shfl_down3(slo, 1); r.rhi = shfl_down3(shi, 1);
    r.rclo = shfl_down3(sclo, 1); r.rchi = shfl_down3(schi, 1);
    if (lane == 31) r.rc = 0;
    return r;
}

// Best plane over all axes (lowest cost, ties -> lowest axis, then lowest bin).
__device__ WarpSplit warp_best_split(const int *bins) {
    const int lane = threadIdx.x & 31;
    WarpSplit best{-1, -1, INFINITY};
    for (int a = 0; a < 3; ++a) {
        AxisScan s = scan_axis(bins, a);
        float cost = INFINITY;
        if (lane < 31 && s.lc > 0 && s.rc > 0)
            cost = surface_area(s.llo, s.lhi) * (float)s.lc + surface_area(s.rlo, s.rhi) * (float)s.rc;
        float c = cost;
        int l = lane;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            float c2 = __shfl_xor_sync(~0u, c, o);
            int l2 = __shfl_xor_sync(~0u, l, o);
            if (c2 < c || (c2 == c && l2 < l)) { c = c2; l = l2; }
        }
        if (c < best.cost) { best.cost = c; best.axis = a; best.bin = l; }
    }
    return best;
}

__device__ void init_bins(int *bins) {
    for (int i = threadIdx.x; i < 3 * kBins * kBinInts; i += blockDim.x) {
        int k = i % kBinInts;
        bins[i] = k == 0 ? 0 : ((k - 1) % 6 < 3 ? f2o(INFINITY) : f2o(-INFINITY));
    }
}

// Lowers / raises a bound of a bin in shared memory.  Most primitives lie
// inside what their bin holds already, so the word is read first: reads of one
// word by many lanes are free, atomics on it are not.  A stale read only costs
// an atomic that changes nothing.  k_bin_large, per level of 5.2M triangles: 87 us
// for 140.  The small builder's bins hold a few primitives each: there the reads
// cost more than they save (3.66 ms for 3.56), so it adds without looking.
__device__ __forceinline__ void bin_min(int *w, int v) {
    if (v < *(volatile int *)w) atomicMin(w, v);
}
__device__ __forceinline__ void bin_max(int *w, int v) {
    if (v > *(volatile int *)w) atomicMax(w, v);
}

// ---------------------------------------------------------------------------
// 2. large tasks
// ---------------------------------------------------------------------------
struct Chunk {
    int task, begin, end, pad;
};

__global__ void k_init_global_bins(int *gbins, int ntasks) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntasks * 3 * kBins * kBinInts) return;
    int k = i % kBinInts;
    gbins[i] = k == 0 ? 0 : ((k - 1) % 6 < 3 ? f2o(INFINITY) : f2o(-INFINITY));
}

// One block per chunk.  Besides the task's bins it leaves what the partition
// needs, so that no later kernel of the level gathers the boxes again: each
// position's three bins (five bits an axis) and the chunk's counts, summed
// along the bins.
constexpr int kHist = 3 * kBins;

__global__ void __launch_bounds__(kThreads) k_bin_large(const Chunk *chunks, const Task *tasks, const int *ref,
                                                        const float4 *plo, const float4 *phi, int *gbins,
                                                        unsigned short *codes, int *hist) {
    __shared__ int bins[3 * kBins * kBinInts];
    const Chunk ch = chunks[blockIdx.x];
    const Task tk = tasks[ch.task];
    float sc[3];
    for (int a = 0; a < 3; ++a) sc[a] = bin_scale(tk.clo[a], tk.chi[a]);
    init_bins(bins);
    __syncthreads();
    for (int i = ch.begin + threadIdx.x; i < ch.end; i += blockDim.x) {
        const int p = ref[i];
        const float4 lo = plo[p], hi = phi[p];
        const float3 c = centroid(lo, hi);
        const int l[3] = {f2o(lo.x), f2o(lo.y), f2o(lo.z)}, h[3] = {f2o(hi.x), f2o(hi.y), f2o(hi.z)};
        const int m[3] = {f2o(c.x), f2o(c.y), f2o(c.z)};
        unsigned code = 0u;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int b = bin_of(comp(c, a), tk.clo[a], sc[a]);
            code |= (unsigned)b << (5 * a);
            int *B = bins + (a * kBins + b) * kBinInts;
            atomicAdd(&B[0], 1);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                bin_min(&B[1 + k], l[k]);
                bin_max(&B[4 + k], h[k]);
                bin_min(&B[7 + k], m[k]);
                bin_max(&B[10 + k], m[k]);
            }
        }
        codes[i] = (unsigned short)code;
    }
    __syncthreads();
    if (threadIdx.x < kHist)  // an axis per warp
        hist[(size_t)blockIdx.x * kHist + threadIdx.x] = warp_incl_scan(bins[threadIdx.x * kBinInts]);
    int *G = gbins + (size_t)ch.task * 3 * kBins * kBinInts;
    for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
        const int *B = bins + i * kBinInts;
        if (B[0] == 0) continue;
        int *D = G + i * kBinInts;
        atomicAdd(&D[0], B[0]);
        for (int k = 1; k <= 3; ++k) atomicMin(&D[k], B[k]);
        for (int k = 4; k <= 6; ++k) atomicMax(&D[k], B[k]);
        for (int k = 7; k <= 9; ++k) atomicMin(&D[k], B[k]);
        for (int k = 10; k <= 12; ++k) atomicMax(&D[k], B[k]);
    }
}

// The lefts of the task's chunks before each of its chunks, by one warp.
__device__ void chunk_lefts(const Task &tk, int chunk, int axis, int bin, int nleft, const int *hist, int *before,
                            int *err) {
    const int lane = threadIdx.x & 31, n_chunks = (tk.count + chunk - 1) / chunk;
    int run = 0;
    for (int base = 0; base < n_chunks; base += 32) {
        const int c = base + lane;
        int v = 0;
        if (c < n_chunks)
            v = axis < 0 ? min(max(nleft - c * chunk, 0), min(chunk, tk.count - c * chunk))
                         : hist[(size_t)(tk.first_chunk + c) * kHist + axis * kBins + bin];
        const int incl = warp_incl_scan(v);
        if (c < n_chunks) before[tk.first_chunk + c] = run + incl - v;
        run += __shfl_sync(~0u, incl, 31);
    }
    if (run != nleft && lane == 0) raise_err(err, kErrBadChild);  // the chunks disagree with the bins
}

// One warp per task: SAH split, child boxes, the chunks' places.
__global__ void k_split_large(const Task *tasks, int ntasks, const int *gbins, Split *out, int chunk,
                              const int *hist, int *before, int *err) {
    const int t = blockIdx.x;
    if (t >= ntasks) return;
    const int lane = threadIdx.x & 31;
    const int *bins = gbins + (size_t)t * 3 * kBins * kBinInts;
    WarpSplit best = warp_best_split(bins);
    Split s;
    memset(&s, 0, sizeof s);
    if (best.axis < 0) {
        // Every centroid in one bin on every axis: split by position, both
        // children conservatively take the parent's boxes.
        AxisScan a = scan_axis(bins, 0);
        // lane 31 holds the full box in its prefix
        float3 lo = f3(__shfl_sync(~0u, a.llo.x, 31), __shfl_sync(~0u, a.llo.y, 31), __shfl_sync(~0u, a.llo.z, 31));
        float3 hi = f3(__shfl_sync(~0u, a.lhi.x, 31), __shfl_sync(~0u, a.lhi.y, 31), __shfl_sync(~0u, a.lhi.z, 31));
        float3 clo = f3(__shfl_sync(~0u, a.lclo.x, 31), __shfl_sync(~0u, a.lclo.y, 31), __shfl_sync(~0u, a.lclo.z, 31));
        float3 chi = f3(__shfl_sync(~0u, a.lchi.x, 31), __shfl_sync(~0u, a.lchi.y, 31), __shfl_sync(~0u, a.lchi.z, 31));
        if (lane == 0) {
            s.axis = -1;
            s.bin = -1;
            s.nleft = tasks[t].count / 2;
            for (int c = 0; c < 2; ++c) {
                s.lo[c][0] = lo.x; s.lo[c][1] = lo.y; s.lo[c][2] = lo.z;
                s.hi[c][0] = hi.x; s.hi[c][1] = hi.y; s.hi[c][2] = hi.z;
                s.clo[c][0] = clo.x; s.clo[c][1] = clo.y; s.clo[c][2] = clo.z;
                s.chi[c][0] = chi.x; s.chi[c][1] = chi.y; s.chi[c][2] = chi.z;
            }
            out[t] = s;
        }
        chunk_lefts(tasks[t], chunk, -1, 0, tasks[t].count / 2, hist, before, err);
        return;
    }
    AxisScan a = scan_axis(bins, best.axis);
    chunk_lefts(tasks[t], chunk, best.axis, best.bin, __shfl_sync(~0u, a.lc, best.bin), hist, before, err);
    if (lane == best.bin) {
        s.axis = best.axis;
        s.bin = best.bin;
        s.nleft = a.lc;
        s.lo[0][0] = a.llo.x; s.lo[0][1] = a.llo.y; s.lo[0][2] = a.llo.z;
        s.hi[0][0] = a.lhi.x; s.hi[0][1] = a.lhi.y; s.hi[0][2] = a.lhi.z;
        s.lo[1][0] = a.rlo.x; s.lo[1][1] = a.rlo.y; s.lo[1][2] = a.rlo.z;
        s.hi[1][0] = a.rhi.x; s.hi[1][1] = a.rhi.y; s.hi[1][2] = a.rhi.z;
        s.clo[0][0] = a.lclo.x; s.clo[0][1] = a.lclo.y; s.clo[0][2] = a.lclo.z;
        s.chi[0][0] = a.lchi.x; s.chi[0][1] = a.lchi.y; s.chi[0][2] = a.lchi.z;
        s.clo[1][0] = a.rclo.x; s.clo[1][1] = a.rclo.y; s.clo[1][2] = a.rclo.z;
        s.chi[1][0] = a.rchi.x; s.chi[1][1] = a.rchi.y; s.chi[1][2] = a.rchi.z;
        out[t] = s;
    }
}

// Stable partition of a chunk: each warp moves kWarpRuns x 32 consecutive refs,
// held in registers while the warps add up their lefts.
// A level of 5.2M triangles (bins, split, partition) takes 125 us; with centroid
// atomics unconditional, a counting pass over the boxes and a third gather here
// it took 252.
template <int kWarpRuns>
__global__ void __launch_bounds__(kThreads) k_part_scatter(const Chunk *chunks, const Task *tasks,
                                                           const Split *splits, const int *before,
                                                           const int *ref, const unsigned short *codes,
                                                           int *ref_out, int n, int *err) {
    __shared__ int warp_lefts[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Chunk ch = chunks[blockIdx.x];
    const int tb = tasks[ch.task].begin, tc = tasks[ch.task].count;
    const int axis = splits[ch.task].axis, bin = splits[ch.task].bin, nleft = splits[ch.task].nleft;
    const int first = ch.begin + warp * kWarpRuns * 32 + lane;
    int p[kWarpRuns], lefts = 0;
    unsigned left = 0u;
#pragma unroll
    for (int k = 0; k < kWarpRuns; ++k) {
        const int i = first + 32 * k;
        const bool valid = i < ch.end;
        p[k] = valid ? ref[i] : 0;
        const int code = valid ? codes[i] : 0;
        if (valid && (axis < 0 ? i - tb < nleft : ((code >> (5 * axis)) & (kBins - 1)) <= bin)) left |= 1u << k;
        lefts += __popc(__ballot_sync(~0u, (left >> k) & 1u));
    }
    if (lane == 0) warp_lefts[warp] = lefts;
    __syncthreads();
    int lb = before[blockIdx.x];  // lefts of the task before this warp's next run
    for (int w = 0; w < warp; ++w) lb += warp_lefts[w];
#pragma unroll
    for (int k = 0; k < kWarpRuns; ++k) {
        const int i = first + 32 * k;
        const bool l = (left >> k) & 1u;
        const unsigned m = __ballot_sync(~0u, l);
        const int before_me = lb + __popc(m & ((1u << lane) - 1u));
        if (i < ch.end) {
            const int dst = l ? tb + before_me : tb + nleft + ((i - tb) - before_me);
            if (dst < tb || dst >= tb + tc || dst >= n) raise_err(err, kErrBadChild);
            else ref_out[dst] = p[k];
        }
        lb += __popc(m);
    }
}

__global__ void k_write_nodes(const int *ids, const BinNode *vals, const int *firsts,
                              const int *counts, int m, BinNode *nodes, int *bfirst, int *bcount,
                              int cap, int *err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    int id = ids[i];
    if (id < 0 || id >= cap) { raise_err(err, kErrNodeOverflow); return; }
    nodes[id] = vals[i];
    bfirst[id] = firsts[i];
    bcount[id] = counts[i];
}

// ---------------------------------------------------------------------------
// 3. small tasks: one block builds a whole subtree
//
// The block holds its task's primitive boxes in shared memory and permutes
// 16-bit local indices.  Nodes of more than 32 primitives go level by level,
// a warp (or, while a level has fewer nodes than the block has warps, a group
// of warps) binning each; nodes of at most 32 are finished by one warp with a
// primitive per lane (tiny_build).  A split at position m of the task (its
// right child begins there) owns the node slots slot_base + 2 (m - 1) + {0, 1}:
// every split of a task has its own m, so no counter orders the warps and the
// tree is the same on every run.
//
// What bounds it: the binary tree down to one triangle has as many inner
// nodes as triangles, half of them with two or three primitives.  One block
// of 256 threads per node (its bins cleared, filled and scanned, eight
// barriers, for two primitives) took 126.5 ms of the 142 ms build of 5.2M
// triangles; this takes 3.55 ms (82k triangles: 10.2 -> 0.23 ms), the same
// tree.  Shared-memory atomics bound the levels above 32 primitives, shuffles
// and min / max the rest; boxes in shared memory (108 KB) allow two blocks of
// 12 warps per SM, whose levels overlap.
// ---------------------------------------------------------------------------
constexpr int kSbWarps = 12, kSbThreads = 32 * kSbWarps;  // two blocks per SM (shared memory)
constexpr int kTiny = 32;       // nodes up to this size: one primitive per lane
constexpr int kSbBinInts = 7;   // count, box lo / hi (ordered ints)
constexpr int kSbBins = 3 * kBins * kSbBinInts;
constexpr int kSbNodes = kSmall / (kTiny + 1) + 1;  // nodes above kTiny primitives on one level

struct SbNode {
    int node, b, c;
    float clo[3], chi[3];
};

struct SbShared {
    float box[6][kSmall];          // lo xyz, hi xyz by local index
    int prim[kSmall];              // primitive of a local index
    unsigned short idx[kSmall], tmp[kSmall];
    int bins[kSbWarps][kSbBins];
    SbNode list[2][kSbNodes];      // this level's and the next level's nodes
    int2 tiny[kSmall / 2];         // (node, b | c << 16)
    unsigned char perm[kSbWarps][32];
    int n_list[2], n_tiny;
};
static_assert(2 * (sizeof(SbShared) + 1024) <= 227 * 1024, "two blocks per SM");

// What the build writes of a node when it is made: its box and its range of
// refs; a leaf's mark, or links that its own split fills in.
__device__ __forceinline__ void put_node(BinNode *nodes, int *bfirst, int *bcount, int id, float3 lo, float3 hi,
                                         int first, int count, bool leaf) {
    nodes[id].lo = make_float4(lo.x, lo.y, lo.z, leaf ? __int_as_float(first) : 0.0f);
    nodes[id].hi = make_float4(hi.x, hi.y, hi.z, leaf ? __int_as_float(-count) : 0.0f);
    bfirst[id] = first;
    bcount[id] = count;
}

__device__ __forceinline__ float3 shfl3(float3 v, int src) {
    return f3(__shfl_sync(~0u, v.x, src), __shfl_sync(~0u, v.y, src), __shfl_sync(~0u, v.z, src));
}

// warp_best_split over a warp's bins of kSbBinInts ints (no centroid boxes);
// also the number of primitives left of the plane.
__device__ WarpSplit sb_best_split(const int *bins, int *n_left) {
    const int lane = threadIdx.x & 31;
    WarpSplit best{-1, -1, INFINITY};
    int nl = 0;
    for (int a = 0; a < 3; ++a) {
        const int *B = bins + (a * kBins + lane) * kSbBinInts;
        int pc = B[0], sc = pc;
        float3 plo = f3(o2f(B[1]), o2f(B[2]), o2f(B[3])), phi = f3(o2f(B[4]), o2f(B[5]), o2f(B[6]));
        float3 slo = plo, shi = phi;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(~0u, pc, o), d = __shfl_down_sync(~0u, sc, o);
            const float3 ulo = shfl_up3(plo, o), uhi = shfl_up3(phi, o);
            const float3 dlo = shfl_down3(slo, o), dhi = shfl_down3(shi, o);
            if (lane >= o) { pc += u; plo = fmin3(plo, ulo); phi = fmax3(phi, uhi); }
            if (lane + o < 32) { sc += d; slo = fmin3(slo, dlo); shi = fmax3(shi, dhi); }
        }
        const int rc = __shfl_down_sync(~0u, sc, 1);
        const float3 rlo = shfl_down3(slo, 1), rhi = shfl_down3(shi, 1);
        float c = INFINITY;
        if (lane < 31 && pc > 0 && rc > 0)
            c = surface_area(plo, phi) * (float)pc + surface_area(rlo, rhi) * (float)rc;
        int l = lane;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float c2 = __shfl_xor_sync(~0u, c, o);
            const int l2 = __shfl_xor_sync(~0u, l, o);
            if (c2 < c || (c2 == c && l2 < l)) { c = c2; l = l2; }
        }
        const int lc = __shfl_sync(~0u, pc, l);
        if (c < best.cost) { best.cost = c; best.axis = a; best.bin = l; nl = lc; }
    }
    *n_left = nl;
    return best;
}

// Inclusive minimum / maximum over a lane's segment [sb, ..], up to its lane; the
// longest segment of the warp has `longest` lanes.
__device__ __forceinline__ void seg_scan_box(float3 &lo, float3 &hi, int sb, int longest) {
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < longest; o <<= 1) {
        const float3 l = shfl_up3(lo, o), h = shfl_up3(hi, o);
        if (lane - o >= sb) {
            lo = fmin3(lo, l);
            hi = fmax3(hi, h);
        }
    }
}

// Finishes the subtree of at most 32 primitives at refs [b, b + c) of the
// task: lane i holds primitive i, the nodes of one level are segments of
// lanes, and all of them are split at once.  A segment's candidate planes are
// its primitives' own bins (an empty bin's plane makes the same partition as
// the occupied bin before it, at a larger index).  The lanes take their segment
// in the order of an axis's bins (ranks counted for the three axes at once, a
// byte each) and the boxes left and right of every plane are scans from both
// ends; the choice (least cost, then lowest axis, then lowest bin) is that of
// the 32-bin scan.  Instruction issue bounds the small builder, most of it here;
// with every lane walking its segment for the sums instead of scans, 5.2M
// triangles took 3.48 for 3.10 ms in it (walking only segments of up to 4
// or 8 lanes: no difference).
__device__ void tiny_build(SbShared &sh, int root, int b, int c, int begin, int slot_base, int max_leaf,
                           BinNode *nodes, int *bfirst, int *bcount) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const bool mine = lane < c;
    int local = mine ? sh.idx[b + lane] : 0;
    float3 lo = f3(sh.box[0][local], sh.box[1][local], sh.box[2][local]);
    float3 hi = f3(sh.box[3][local], sh.box[4][local], sh.box[5][local]);
    int sb = mine ? 0 : lane, se = mine ? c : lane + 1;  // this lane's segment
    int node = root;
    while (true) {
        const int s = se - sb;
        const bool act = mine && s > max_leaf;
        const int longest = __reduce_max_sync(~0u, act ? s : 0);
        if (longest == 0) break;
        const float3 cen = f3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
        float3 clo = cen, chi = cen;
        seg_scan_box(clo, chi, sb, longest);
        clo = shfl3(clo, se - 1);
        chi = shfl3(chi, se - 1);
        unsigned bin[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
            bin[a] = (unsigned)bin_of(comp(cen, a), comp(clo, a), bin_scale(comp(clo, a), comp(chi, a)));
        const unsigned packed = bin[0] | bin[1] << 8 | bin[2] << 16;
        float cost = INFINITY;
        int key = 0x7fffffff;  // axis, bin
        // each lane's rank in its segment by (bin, lane), per axis: a byte of
        // d has its top bit set where the other's bin, or in a tie its lane,
        // is the lower one
        const unsigned mine2 = 2u * packed, base = 0x7f7f7fu + mine2;
        unsigned rank = 0u;
        for (int k = 0; k < longest; ++k) {
            const int src = sb + k;
            const unsigned other = __shfl_sync(~0u, mine2, src);
            const unsigned d = base + (src < lane ? 0x010101u : 0u) - other;
            if (k < s) rank += (d >> 7) & 0x010101u;
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            sh.perm[warp][sb + ((rank >> (8 * a)) & 0xffu)] = (unsigned char)lane;
            __syncwarp();
            const int src = sh.perm[warp][lane];
            __syncwarp();
            float3 llo = shfl3(lo, src), lhi = shfl3(hi, src), rlo = llo, rhi = lhi;
            const unsigned b = (__shfl_sync(~0u, packed, src) >> (8 * a)) & 0xffu;
            for (int o = 1; o < longest; o <<= 1) {
                const float3 ul = shfl_up3(llo, o), uh = shfl_up3(lhi, o);
                const float3 dl = shfl_down3(rlo, o), dh = shfl_down3(rhi, o);
                if (lane - o >= sb) { llo = fmin3(llo, ul); lhi = fmax3(lhi, uh); }
                if (lane + o < se) { rlo = fmin3(rlo, dl); rhi = fmax3(rhi, dh); }
            }
            rlo = shfl_down3(rlo, 1);
            rhi = shfl_down3(rhi, 1);
            const unsigned nb = __shfl_down_sync(~0u, b, 1);
            if (lane + 1 < se && nb != b) {  // the last primitive of its bin: a plane
                const int lc = lane - sb + 1, rc = se - lane - 1;
                const float ca = surface_area(llo, lhi) * (float)lc + surface_area(rlo, rhi) * (float)rc;
                if (ca < cost) { cost = ca; key = a * kBins + (int)b; }
            }
        }
        float best = cost;
        int bkey = key;
        for (int o = 1; o < longest; o <<= 1) {
            const float q = __shfl_up_sync(~0u, best, o);
            const int qk = __shfl_up_sync(~0u, bkey, o);
            if (lane - o >= sb && (q < best || (q == best && qk < bkey))) { best = q; bkey = qk; }
        }
        best = __shfl_sync(~0u, best, se - 1);
        bkey = __shfl_sync(~0u, bkey, se - 1);
        // no plane (all centroids in one bin on every axis): by position
        bool left = lane - sb < s / 2;
        if (best < INFINITY) {
            const int a = bkey / kBins;
            left = (a == 0 ? bin[0] : a == 1 ? bin[1] : bin[2]) <= (unsigned)(bkey % kBins);
        }
        const unsigned lefts = __ballot_sync(~0u, act && left);
        const unsigned seg = (unsigned)((1ull << se) - (1ull << sb));
        const int nl = __popc(lefts & seg);
        const int dst = !act ? lane
                        : left ? sb + __popc(lefts & seg & below) : sb + nl + __popc(~lefts & seg & below);
        sh.perm[warp][dst] = (unsigned char)lane;
        __syncwarp();
        const int src = sh.perm[warp][lane];
        __syncwarp();
        lo = shfl3(lo, src);
        hi = shfl3(hi, src);
        local = __shfl_sync(~0u, local, src);
        // the children's segments, boxes and records
        const int mid = sb + nl, id = slot_base + 2 * (b + mid - 1);
        const bool right = lane >= mid;
        if (act) {
            if (lane == sb) {
                nodes[node].lo.w = __int_as_float(id);
                nodes[node].hi.w = __int_as_float(id + 1);
            }
            node = right ? id + 1 : id;
            sb = right ? mid : sb;
            se = right ? se : mid;
        }
        float3 nlo = lo, nhi = hi;
        seg_scan_box(nlo, nhi, sb, __reduce_max_sync(~0u, act ? se - sb : 0));
        if (act && lane == se - 1)
            put_node(nodes, bfirst, bcount, node, nlo, nhi, begin + b + sb, se - sb, se - sb <= max_leaf);
    }
    if (mine) sh.idx[b + lane] = (unsigned short)local;
}

// Splits node e by its bins, one warp: the stable partition of its indices,
// the children's boxes and centroid bounds, their records, and their places
// in the next level's list or the tiny list.
__device__ void sb_split(SbShared &sh, const SbNode &e, const int *bins, int next, int begin, int slot_base,
                         int max_leaf, BinNode *nodes, int *bfirst, int *bcount, int *err) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    int nl;
    const WarpSplit w = sb_best_split(bins, &nl);
    if (w.axis < 0) nl = e.c / 2;
    const int ax = w.axis < 0 ? 0 : w.axis;
    const float sc = bin_scale(e.clo[ax], e.chi[ax]);
    const float3 inf = f3(INFINITY, INFINITY, INFINITY), ninf = f3(-INFINITY, -INFINITY, -INFINITY);
    float3 lo[2] = {inf, inf}, hi[2] = {ninf, ninf}, clo[2] = {inf, inf}, chi[2] = {ninf, ninf};
    int nls = 0, nrs = 0;
    for (int base = 0; base < e.c; base += 32) {
        const int i = base + lane;
        const bool valid = i < e.c;
        const int local = valid ? sh.idx[e.b + i] : 0;
        const float3 l = f3(sh.box[0][local], sh.box[1][local], sh.box[2][local]);
        const float3 h = f3(sh.box[3][local], sh.box[4][local], sh.box[5][local]);
        const float3 c = f3(0.5f * (l.x + h.x), 0.5f * (l.y + h.y), 0.5f * (l.z + h.z));
        const bool left = w.axis < 0 ? i < e.c / 2 : bin_of(comp(c, ax), e.clo[ax], sc) <= w.bin;
        const unsigned lm = __ballot_sync(~0u, valid && left), rm = __ballot_sync(~0u, valid && !left);
        if (valid) {
            const int dst = left ? nls + __popc(lm & below) : nl + nrs + __popc(rm & below);
            if (dst < e.c) sh.tmp[e.b + dst] = (unsigned short)local;
            else raise_err(err, kErrBadChild);
            if (left) {
                lo[0] = fmin3(lo[0], l); hi[0] = fmax3(hi[0], h);
                clo[0] = fmin3(clo[0], c); chi[0] = fmax3(chi[0], c);
            } else {
                lo[1] = fmin3(lo[1], l); hi[1] = fmax3(hi[1], h);
                clo[1] = fmin3(clo[1], c); chi[1] = fmax3(chi[1], c);
            }
        }
        nls += __popc(lm);
        nrs += __popc(rm);
    }
    if (nls != nl) {  // the partition disagrees with the bins: no children
        if (lane == 0) raise_err(err, kErrBadChild);
        return;
    }
    __syncwarp();
    for (int i = lane; i < e.c; i += 32) sh.idx[e.b + i] = sh.tmp[e.b + i];
    const int id = slot_base + 2 * (e.b + nl - 1);
    if (lane == 0) {
        nodes[e.node].lo.w = __int_as_float(id);
        nodes[e.node].hi.w = __int_as_float(id + 1);
    }
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const float3 l = warp_min3(lo[side]), h = warp_max3(hi[side]);
        const float3 cl = warp_min3(clo[side]), ch = warp_max3(chi[side]);
        if (lane != 0) continue;
        const int b = side ? e.b + nl : e.b, c = side ? e.c - nl : nl;
        put_node(nodes, bfirst, bcount, id + side, l, h, begin + b, c, c <= max_leaf);
        if (c <= max_leaf) continue;
        if (c <= kTiny) {
            const int k = atomicAdd(&sh.n_tiny, 1);
            if (k < kSmall / 2) sh.tiny[k] = make_int2(id + side, b | c << 16);
            else raise_err(err, kErrStackOverflow);
        } else {
            const int k = atomicAdd(&sh.n_list[next], 1);
            if (k < kSbNodes) {
                SbNode n;
                n.node = id + side; n.b = b; n.c = c;
                n.clo[0] = cl.x; n.clo[1] = cl.y; n.clo[2] = cl.z;
                n.chi[0] = ch.x; n.chi[1] = ch.y; n.chi[2] = ch.z;
                sh.list[next][k] = n;
            } else {
                raise_err(err, kErrStackOverflow);
            }
        }
    }
}

__global__ void __launch_bounds__(kSbThreads, 2) k_small_build(const Task *tasks, const int *slot_bases, int ntasks,
                                                               const float4 *__restrict__ plo,
                                                               const float4 *__restrict__ phi, int *ref,
                                                               const int *ref_b, BinNode *nodes, int *bfirst,
                                                               int *bcount, int cap, int max_leaf, int *err) {
    extern __shared__ __align__(16) unsigned char sb_raw[];
    SbShared &sh = *reinterpret_cast<SbShared *>(sb_raw);
    if (blockIdx.x >= ntasks) return;
    const Task tk = tasks[blockIdx.x];
    const int m = tk.count, slot_base = slot_bases[blockIdx.x];
    if (m > kSmall || m < 1 || tk.node < 0 || tk.node >= cap || slot_base < 0 || slot_base + 2 * (m - 1) > cap) {
        if (threadIdx.x == 0) raise_err(err, m > kSmall || m < 1 ? kErrSmallTooBig : kErrNodeOverflow);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < m; i += kSbThreads) {
        const int p = (tk.buf ? ref_b : ref)[tk.begin + i];
        const float4 l = plo[p], h = phi[p];
        sh.prim[i] = p;
        sh.idx[i] = (unsigned short)i;
        sh.box[0][i] = l.x; sh.box[1][i] = l.y; sh.box[2][i] = l.z;
        sh.box[3][i] = h.x; sh.box[4][i] = h.y; sh.box[5][i] = h.z;
    }
    if (threadIdx.x == 0) {
        sh.n_list[0] = sh.n_list[1] = sh.n_tiny = 0;
        bfirst[tk.node] = tk.begin;
        bcount[tk.node] = m;
        if (m <= max_leaf) {
            nodes[tk.node].lo.w = __int_as_float(tk.begin);
            nodes[tk.node].hi.w = __int_as_float(-m);
        } else if (m <= kTiny) {
            sh.tiny[0] = make_int2(tk.node, m << 16);
            sh.n_tiny = 1;
        } else {
            SbNode n;
            n.node = tk.node; n.b = 0; n.c = m;
            for (int a = 0; a < 3; ++a) { n.clo[a] = tk.clo[a]; n.chi[a] = tk.chi[a]; }
            sh.list[0][0] = n;
            sh.n_list[0] = 1;
        }
    }
    __syncthreads();
    for (int cur = 0;; cur ^= 1) {
        const int n = min(sh.n_list[cur], kSbNodes);  // uniform: last written before a barrier
        if (n == 0) break;
        const int wpn = max(1, kSbWarps / n), groups = kSbWarps / wpn;
        const int g = warp / wpn, wi = warp % wpn;
        for (int base = 0; base < n; base += groups) {
            const bool act = g < groups && base + g < n;
            int *bins = sh.bins[g < groups ? g : 0];
            if (act)
                for (int i = wi * 32 + lane; i < kSbBins; i += wpn * 32) {
                    const int k = i % kSbBinInts;
                    bins[i] = k == 0 ? 0 : (k <= 3 ? f2o(INFINITY) : f2o(-INFINITY));
                }
            __syncthreads();
            if (act) {
                const SbNode e = sh.list[cur][base + g];
                float sc[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) sc[a] = bin_scale(e.clo[a], e.chi[a]);
                for (int i = wi * 32 + lane; i < e.c; i += wpn * 32) {
                    const int local = sh.idx[e.b + i];
                    float3 l = f3(sh.box[0][local], sh.box[1][local], sh.box[2][local]);
                    float3 h = f3(sh.box[3][local], sh.box[4][local], sh.box[5][local]);
                    const float3 c = f3(0.5f * (l.x + h.x), 0.5f * (l.y + h.y), 0.5f * (l.z + h.z));
                    const int o[6] = {f2o(l.x), f2o(l.y), f2o(l.z), f2o(h.x), f2o(h.y), f2o(h.z)};
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        int *B = bins + (a * kBins + bin_of(comp(c, a), e.clo[a], sc[a])) * kSbBinInts;
                        atomicAdd(&B[0], 1);
                        atomicMin(&B[1], o[0]); atomicMin(&B[2], o[1]); atomicMin(&B[3], o[2]);
                        atomicMax(&B[4], o[3]); atomicMax(&B[5], o[4]); atomicMax(&B[6], o[5]);
                    }
                }
            }
            __syncthreads();
            if (act && wi == 0)
                sb_split(sh, sh.list[cur][base + g], bins, cur ^ 1, tk.begin, slot_base, max_leaf, nodes, bfirst,
                         bcount, err);
            __syncthreads();
        }
        if (threadIdx.x == 0) sh.n_list[cur] = 0;
        __syncthreads();
    }
    const int nt = min(sh.n_tiny, kSmall / 2);
    for (int k = warp; k < nt; k += kSbWarps) {
        const int2 e = sh.tiny[k];
        tiny_build(sh, e.x, e.y & 0xffff, e.y >> 16, tk.begin, slot_base, max_leaf, nodes, bfirst, bcount);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += kSbThreads) ref[tk.begin + i] = sh.prim[sh.idx[i]];
}

// ---------------------------------------------------------------------------
// 4. collapse into 8-wide compressed nodes
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool bn_leaf(const BinNode &n) { return __float_as_int(n.hi.w) < 0; }

// SAH-optimal choice of each wide node's children (Ylitie, Karras and Laine,
// "Efficient incoherent ray traversal on GPUs through compressed wide BVHs",
// HPG 2017, section 3.1).  cost(n, i) is the least SAH cost of the binary
// subtree at n represented as at most i children of a wide node:
//   cost(n, 1) = leaf cost if n may be a leaf (at most max_leaf triangles:
//                c_prim A(n) count), else A(n) c_node + D(n, 8);
//   cost(n, i) = min(cost(n, i - 1), D(n, i)),
//   D(n, j)    = min over 0 < k < j of cost(left, k) + cost(right, j - k).
// The table is filled bottom up, a node by the second of its children to
// finish; dec[n] keeps the argmin k of D(n, 8) (bits 0-2) and, for j = 2..8,
// the k of D(n, j) when it beats cost(n, j - 1), else 0 (bits 3(j-1)..).
constexpr float kCostNode = 1.0f;
constexpr float kCostTri = 0.3f;
constexpr float kCostInf = 3.0e38f;

// The row of a node whose children's rows are l and r, for its decision.
__device__ __forceinline__ unsigned dp_join(const float (&l)[8], const float (&r)[8], float area, float (&row)[8]) {
    float D[9];
    int K[9];
#pragma unroll
    for (int j = 2; j <= 8; ++j) {
        float best = kCostInf;
        int bk = 1;
#pragma unroll
        for (int k = 1; k < j; ++k) {
            const float c = l[k - 1] + r[j - k - 1];
            if (c < best) { best = c; bk = k; }
        }
        D[j] = best;
        K[j] = bk;
    }
    float c = kCostNode * area + D[8];
    unsigned d = (unsigned)K[8];
    row[0] = c;
#pragma unroll
    for (int j = 2; j <= 8; ++j) {
        if (D[j] < c) {
            c = D[j];
            d |= (unsigned)K[j] << (3 * (j - 1));
        }
        row[j - 1] = c;
    }
    return d;
}
__device__ __forceinline__ float dp_leaf_cost(const BinNode &nd) {
    return kCostTri * surface_area(f3(nd.lo), f3(nd.hi)) * (float)-__float_as_int(nd.hi.w);
}
// own is the left child's row if own_left: joins it with the sibling's.
__device__ __forceinline__ unsigned dp_join_own(float (&own)[8], const float (&sib)[8], bool own_left, float area) {
    float l[8], r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        l[j] = own_left ? own[j] : sib[j];
        r[j] = own_left ? sib[j] : own[j];
    }
    return dp_join(l, r, area, own);
}
__device__ __forceinline__ void dp_get(const float4 *row, float (&c)[8]) {
    const float4 a = row[0], b = row[1];
    c[0] = a.x; c[1] = a.y; c[2] = a.z; c[3] = a.w;
    c[4] = b.x; c[5] = b.y; c[6] = b.z; c[7] = b.w;
}
__device__ __forceinline__ void dp_put(float4 *row, const float (&c)[8]) {
    row[0] = make_float4(c[0], c[1], c[2], c[3]);
    row[1] = make_float4(c[4], c[5], c[6], c[7]);
}

// The subtree of one small task, a block each, its table in shared memory.  The
// nodes are the pairs of children at slot_base + 2q, so an inner node is known
// by its children's pair.  A thread starts at each leaf and goes on up from the
// pairs it finishes second, as many steps in turn as the subtree is high.  That
// chain bounds it: 0.57 ms at 5.2M triangles and 0.035 ms at 82k, where parents,
// counters and rows of the whole tree in global memory took 1.25 and 0.064.  256
// and 1024 threads are within 1 % of the build.
constexpr int kDpThreads = 512;
struct DpShared {
    float4 row[kSmall][2];          // by pair
    int node[2 * kSmall];           // by slot: a leaf's cost, or the sign bit and an inner node's pair
    float area[kSmall];             // of pair q's parent
    unsigned short parent[kSmall];  // slot of pair q's parent + 1; 0 the task's root
    int visits[kSmall];
};

__global__ void __launch_bounds__(kDpThreads) k_dp_small(const Task *tasks, const int *slot_bases, int ntasks,
                                                         const BinNode *nodes, int cap, float4 *root_rows,
                                                         unsigned *dec, int *err) {
    extern __shared__ __align__(16) unsigned char dp_raw[];
    DpShared &sh = *reinterpret_cast<DpShared *>(dp_raw);
    constexpr unsigned short kNone = 0xffff;
    if (blockIdx.x >= ntasks) return;
    const int root = tasks[blockIdx.x].node, m = tasks[blockIdx.x].count, base = slot_bases[blockIdx.x];
    const int slots = 2 * (m - 1);
    if (m < 1 || m > kSmall || base < 0 || base + slots > cap || root < 0 || root >= cap) return;
    for (int i = threadIdx.x; i < m; i += kDpThreads) {
        sh.parent[i] = kNone;
        sh.visits[i] = 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= slots; i += kDpThreads) {  // 0: the root, i: slot i - 1
        const BinNode nd = nodes[i == 0 ? root : base + i - 1];
        int v;
        if (bn_leaf(nd)) {  // or a slot that no node took (filled with -1)
            const float c = dp_leaf_cost(nd);
            v = __float_as_int(c) & 0x7fffffff;
            if (i == 0) {
                const float row[8] = {c, c, c, c, c, c, c, c};
                dp_put(root_rows + 2 * blockIdx.x, row);
            }
        } else {
            const int l = __float_as_int(nd.lo.w) - base;
            if (l < 0 || l + 1 >= slots || (l & 1) || __float_as_int(nd.hi.w) != base + l + 1) {
                raise_err(err, kErrBadChild);
                v = 0;
            } else {
                sh.parent[l >> 1] = (unsigned short)i;
                sh.area[l >> 1] = surface_area(f3(nd.lo), f3(nd.hi));
                v = (int)(0x80000000u | (unsigned)(l >> 1));
            }
        }
        if (i > 0) sh.node[i - 1] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < slots; i += kDpThreads) {
        int s = i;
        if (sh.parent[s >> 1] == kNone || sh.node[s] < 0) continue;
        float own[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) own[j] = __int_as_float(sh.node[s]);
        for (int guard = 0; guard < kSmall; ++guard) {
            const int q = s >> 1;
            __threadfence_block();
            if (atomicAdd(&sh.visits[q], 1) == 0) break;  // the sibling's thread goes on from here
            __threadfence_block();
            const int v = sh.node[s ^ 1], p = sh.parent[q];
            float sib[8];
            if (v < 0) {
                dp_get(sh.row[v & (kSmall - 1)], sib);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) sib[j] = __int_as_float(v);
            }
            dec[p == 0 ? root : base + p - 1] = dp_join_own(own, sib, (s & 1) == 0, sh.area[q]);
            if (p == 0) {
                dp_put(root_rows + 2 * blockIdx.x, own);
                break;
            }
            dp_put(sh.row[q], own);
            s = p - 1;
        }
    }
}

// The nodes above the small tasks, from every task's root up: pair q's children
// are nodes 1 + 2q and 2 + 2q.  rows: by node.
__global__ void k_dp_top(const Task *tasks, int ntasks, const BinNode *nodes, const int *parent, int n_top,
                         const float4 *root_rows, float4 *rows, unsigned *dec, int *visits, int *err) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntasks) return;
    int node = tasks[t].node;
    if (node < 0 || node >= n_top) { raise_err(err, kErrBadChild); return; }
    float own[8], sib[8];
    dp_get(root_rows + 2 * t, own);
    while (node > 0) {  // a parent's id is below its children's
        const int q = (node - 1) >> 1, p = parent[q], other = node & 1 ? node + 1 : node - 1;
        __stcg(rows + 2 * node, make_float4(own[0], own[1], own[2], own[3]));
        __stcg(rows + 2 * node + 1, make_float4(own[4], own[5], own[6], own[7]));
        __threadfence();
        if (atomicAdd(&visits[q], 1) == 0) return;
        __threadfence();
        if (p < 0 || p >= node) { raise_err(err, kErrBadChild); return; }
        const float4 a = __ldcg(rows + 2 * other), b = __ldcg(rows + 2 * other + 1);
        sib[0] = a.x; sib[1] = a.y; sib[2] = a.z; sib[3] = a.w;
        sib[4] = b.x; sib[5] = b.y; sib[6] = b.z; sib[7] = b.w;
        const BinNode nd = nodes[p];
        dec[p] = dp_join_own(own, sib, (node & 1) != 0, surface_area(f3(nd.lo), f3(nd.hi)));
        node = p;
    }
}

// The wide children of binary node b, at most eight, as the cost table chose;
// *n_inner and *n_tris count what they add to the next level and the records.
__device__ bool collapse_choose(int b, const BinNode *nodes, const int *bcount, const unsigned *dec, int cap,
                                int max_leaf, int *children, int *n_inner, int *n_tris) {
    int C[8];
    int nc = 0;
    if (b < 0 || b >= cap) return false;
    const BinNode nb = nodes[b];
    if (bcount[b] <= max_leaf || bn_leaf(nb)) {
        C[nc++] = b;
    } else {
        // the 8 slots go to b's two children as the cost table chose, and on
        // down until each share is one slot, a leaf or a node that keeps
        // what it was given
        int sn[16], sj[16];
        int sp = 0;
        const int k8 = (int)(dec[b] & 7u);
        sn[sp] = __float_as_int(nb.lo.w); sj[sp++] = k8;
        sn[sp] = __float_as_int(nb.hi.w); sj[sp++] = 8 - k8;
        while (sp > 0) {
            --sp;
            const int c = sn[sp];
            int j = sj[sp];
            if (c < 0 || c >= cap || j < 1 || nc >= 8) return false;
            const BinNode nn = nodes[c];
            if (j > 1 && bcount[c] > max_leaf && !bn_leaf(nn)) {
                const unsigned dc = dec[c];
                while (j > 1 && ((dc >> (3 * (j - 1))) & 7u) == 0u) --j;
                if (j > 1) {
                    const int k = (int)((dc >> (3 * (j - 1))) & 7u);
                    if (sp + 2 > 16 || k < 1 || k >= j) return false;
                    sn[sp] = __float_as_int(nn.lo.w); sj[sp++] = k;
                    sn[sp] = __float_as_int(nn.hi.w); sj[sp++] = j - k;
                    continue;
                }
            }
            C[nc++] = c;
        }
    }
    int ni = 0, nt = 0;
    for (int i = 0; i < 8; ++i) {
        const int c = i < nc ? C[i] : -1;
        children[i] = c;
        if (c >= 0) {
            if (c >= cap) return false;
            const int k = bcount[c];
            if (k <= max_leaf) nt += k;
            else ni += 1;
        }
    }
    *n_inner = ni;
    *n_tris = nt;
    return true;
}

// Per-axis quantisation exponent: the smallest power of two s with
// extent / s <= 255, returned as the biased exponent byte.
__device__ __forceinline__ int quant_exponent(float extent) {
    if (!(extent > 0.0f)) return 27;  // 2^-100: a flat axis
    float r = extent / 255.0f;
    int e;
    frexpf(r, &e);  // r = m * 2^e, m in [0.5, 1)
    int k = e;      // 2^e >= r
    if (ldexpf(1.0f, k - 1) >= r) k -= 1;
    while (extent / ldexpf(1.0f, k) > 255.0f) ++k;
    if (k < -100) k = -100;
    return k + 127;
}

// OR over the eight lanes of a node.
__device__ __forceinline__ unsigned or8(unsigned gm, unsigned v) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v |= __shfl_xor_sync(gm, v, o);
    return v;
}
// The byte of one plane, conservative: rounded down (kUp false) or up and
// moved on while the decoded plane lies on the wrong side.
template <bool kUp>
__device__ __forceinline__ unsigned quant_plane(float v, float p, float s) {
    float q;
    if (kUp) {
        q = ceilf((v - p) / s);
        while (q < 255.0f && p + q * s < v) q += 1.0f;
    } else {
        q = floorf((v - p) / s);
        while (q > 0.0f && p + q * s > v) q -= 1.0f;
    }
    return (unsigned)fminf(fmaxf(q, 0.0f), 255.0f);
}

struct CollapseArgs {
    const BinNode *nodes;
    const int *bfirst, *bcount, *ref;
    const unsigned *dec;
    const float4 *verts, *attr;
    const kgk_material *mats;
    WideNode *wide;
    float4 *tri_rec;
    int *tasks[2];     // binary nodes to turn into wide ones, this level's and the next one's
    int *child_list;   // 8 per task
    int2 *counts;      // per task: inner children, triangles
    int4 *sums;        // per block: the same summed, and whether a check failed
    int *result;       // wide nodes, triangles, levels
    int *err;
    int cap, list_cap, wide_cap, n_tris, n_mats, max_leaf;
};

// Eight lanes write one wide node, a child each: slots, quantised planes and
// triangle records side by side instead of one thread looping over children,
// slots and planes with its arrays in local memory.  The triangle gather (48
// bytes in, 48 out each) bounds it.
// Task's children at list[0..8), the node's place, the first of its inner
// children among the next level's tasks and nodes, the first of its triangles.
__device__ void collapse_emit(const CollapseArgs &A, const int *list, int me, int pos0, int child_base, int tri_base,
                              int *next_tasks, int *failed) {
    const int k = threadIdx.x & 7;
    const unsigned gm = 0xffu << (threadIdx.x & 24);  // this node's lanes
    const auto bad = [&](int code) {
        raise_err(A.err, code);
        *failed = 1;
    };
    const int c = list[k];
    const bool valid = c >= 0;
    if (__any_sync(gm, c >= A.cap)) {
        if (k == 0) bad(kErrBadChild);
        return;
    }
    const int nc = __popc(__ballot_sync(gm, valid));
    float3 clo = f3(INFINITY, INFINITY, INFINITY), chi = f3(-INFINITY, -INFINITY, -INFINITY);
    int cnt = 0;
    if (valid) {
        clo = f3(A.nodes[c].lo);
        chi = f3(A.nodes[c].hi);
        cnt = A.bcount[c];
    }
    float3 plo = clo, phi = chi;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        plo = fmin3(plo, f3(__shfl_xor_sync(gm, plo.x, o), __shfl_xor_sync(gm, plo.y, o), __shfl_xor_sync(gm, plo.z, o)));
        phi = fmax3(phi, f3(__shfl_xor_sync(gm, phi.x, o), __shfl_xor_sync(gm, phi.y, o), __shfl_xor_sync(gm, phi.z, o)));
    }
    // slot assignment: child i -> slot s maximising dot(centre_i - centre, D(s)),
    // D(s) = (s&4 ? +1 : -1, s&2 ? +1 : -1, s&1 ? +1 : -1); greedy over pairs,
    // ties to the lower child, then the lower slot.
    const float3 d = 0.5f * (clo + chi) - 0.5f * (plo + phi);
    int slot = -1;
    unsigned taken = 0u;
    for (int round = 0; round < nc; ++round) {
        float v = -INFINITY;
        int sl = -1;
        if (valid && slot < 0) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const float q = ((s & 4) ? d.x : -d.x) + ((s & 2) ? d.y : -d.y) + ((s & 1) ? d.z : -d.z);
                if (!((taken >> s) & 1u) && q > v) { v = q; sl = s; }
            }
        }
        int who = k;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            const float v2 = __shfl_xor_sync(gm, v, o);
            const int w2 = __shfl_xor_sync(gm, who, o), s2 = __shfl_xor_sync(gm, sl, o);
            if (s2 >= 0 && (sl < 0 || v2 > v || (v2 == v && w2 < who))) { v = v2; who = w2; sl = s2; }
        }
        if (sl < 0) {  // boxes that are not numbers: the first child left, the first slot left
            who = __ffs((__ballot_sync(gm, valid && slot < 0) & gm) >> (threadIdx.x & 24)) - 1;
            sl = __ffs(~taken) - 1;
        }
        taken |= 1u << sl;
        if (who == k) slot = sl;
    }
    // quantisation frame
    const float3 ext = (phi - plo) * (1.0f + 1.0f / 1048576.0f);
    const int ex = quant_exponent(ext.x), ey = quant_exponent(ext.y), ez = quant_exponent(ext.z);
    const float sx = ldexpf(1.0f, ex - 127), sy = ldexpf(1.0f, ey - 127), sz = ldexpf(1.0f, ez - 127);
    const bool inner = valid && cnt > A.max_leaf, leaf = valid && !inner;
    if (__any_sync(gm, leaf && (cnt < 1 || cnt > kMaxLeaf))) {
        if (k == 0) bad(kErrTriOverflow);
        return;
    }
    unsigned own = 0u;  // leaf bits, and the inner bit above them
    if (leaf)
        for (int j = 0; j < cnt; ++j) own |= 1u << (slot + 8 * j);
    if (inner) own = 1u << (24 + slot);
    const unsigned field = or8(gm, own);
    // six plane words of four slots each: low and high per axis
    unsigned w[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) w[i] = 0u;
    if (valid) {
        const unsigned q[6] = {quant_plane<false>(clo.x, plo.x, sx), quant_plane<true>(chi.x, plo.x, sx),
                               quant_plane<false>(clo.y, plo.y, sy), quant_plane<true>(chi.y, plo.y, sy),
                               quant_plane<false>(clo.z, plo.z, sz), quant_plane<true>(chi.z, plo.z, sz)};
        const int sh = 8 * (slot & 3);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const unsigned b = q[i] << sh;
            w[2 * i] = slot < 4 ? b : 0u;
            w[2 * i + 1] = slot < 4 ? 0u : b;
        }
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) w[i] = or8(gm, w[i]);
    if (inner) {
        const int j = __popc((field >> 24) & ((1u << slot) - 1u));
        if (pos0 + j >= A.list_cap || child_base + j >= A.wide_cap) bad(kErrWideOverflow);
        else next_tasks[pos0 + j] = c;
    }
    // triangles in the order of their bits: every leaf's first, then the second ones, ...
    if (leaf) {
        const int f = A.bfirst[c];
        for (int j = 0; j < cnt; ++j) {
            const int dst = tri_base + __popc(field & ((1u << (slot + 8 * j)) - 1u));
            if (f < 0 || f + j >= A.n_tris || dst < 0 || dst >= A.n_tris) { bad(kErrTriOverflow); break; }
            const int prim = A.ref[f + j];
            if (prim < 0 || prim >= A.n_tris) { bad(kErrTriOverflow); break; }
            // The material class goes into the .w of the second record (1 =
            // Disney BRDF, 0 = any other type; the intersection test reads only
            // .xyz there), so a closest hit tells the shading queues apart
            // without a material lookup.
            const unsigned mat = __float_as_uint(A.attr[4 * (size_t)prim + 3].w) & 0x7fffffffu;
            const int cls = mat < (unsigned)A.n_mats && A.mats[mat].MATERIAL_TYPE_ID == 1 ? 1 : 0;
            const float4 a = A.verts[3 * (size_t)prim], b = A.verts[3 * (size_t)prim + 1], cc = A.verts[3 * (size_t)prim + 2];
            A.tri_rec[3 * (size_t)dst] = make_float4(a.x, a.y, a.z, __int_as_float(prim));
            A.tri_rec[3 * (size_t)dst + 1] = make_float4(b.x, b.y, b.z, __int_as_float(cls));
            A.tri_rec[3 * (size_t)dst + 2] = make_float4(cc.x, cc.y, cc.z, 0.0f);
        }
    }
    if (me >= A.wide_cap) {
        if (k == 0) bad(kErrWideOverflow);
        return;
    }
    float4 out = make_float4(plo.x, plo.y, plo.z,
                             __uint_as_float((unsigned)ex | ((unsigned)ey << 8) | ((unsigned)ez << 16)));
    if (k == 1) out = make_float4(__int_as_float(child_base), __int_as_float(tri_base), __uint_as_float(field), 0.0f);
#pragma unroll
    for (int a = 0; a < 3; ++a)  // low words of slots 0-3 and 4-7, then the high ones
        if (k == 2 + a)
            out = make_float4(__uint_as_float(w[4 * a]), __uint_as_float(w[4 * a + 1]), __uint_as_float(w[4 * a + 2]),
                              __uint_as_float(w[4 * a + 3]));
    if (k < 5) reinterpret_cast<float4 *>(A.wide + me)[k] = out;
}

// The whole collapse, breadth first, one cooperative launch: a level is a pass
// that chooses children and sums what they take, a grid barrier, a pass that
// places and writes them, a grid barrier.  Every block sums the blocks before it
// by itself, so places do not depend on timing.  With a launch per pass and scan
// and the host waiting for each level's totals, the collapse of 82k triangles
// took 0.27 ms of kernels and 0.4 ms of gaps, of 5.2M 1.23 and 0.8 ms; this takes
// 0.16 and 1.07 ms.
// All blocks decide alike whether to go on: from the sums, which carry the
// failed checks too, never from the error flag.
constexpr int kCollapseThreads = 256;

__global__ void __launch_bounds__(kCollapseThreads) k_collapse(const CollapseArgs A) {
    __shared__ int ws[32], s_inner[kCollapseThreads], s_tri[kCollapseThreads], acc[5], failed;
    cg::grid_group grid = cg::this_grid();
    const int tid = threadIdx.x;
    int ntasks = 1, level_start = 0, tri_start = 0, levels = 0;
    if (tid == 0) failed = 0;
    __syncthreads();
    for (int cur = 0; ntasks > 0; cur ^= 1) {
        ++levels;
        const int next_start = level_start + ntasks;
        const int per = (ntasks + gridDim.x - 1) / gridDim.x;
        const int t0 = min(ntasks, (int)blockIdx.x * per), t1 = min(ntasks, t0 + per);
        if (tid < 5) acc[tid] = 0;
        __syncthreads();
        int ni = 0, nt = 0;
        for (int t = t0 + tid; t < t1; t += kCollapseThreads) {
            int a = 0, b = 0;
            if (!collapse_choose(levels == 1 ? 0 : A.tasks[cur][t], A.nodes, A.bcount, A.dec, A.cap, A.max_leaf,
                                 A.child_list + 8 * (size_t)t, &a, &b)) {
                raise_err(A.err, kErrBadChild);
                failed = 1;
            }
            A.counts[t] = make_int2(a, b);
            ni += a;
            nt += b;
        }
        ni = __reduce_add_sync(~0u, ni);
        nt = __reduce_add_sync(~0u, nt);
        if ((tid & 31) == 0) {
            atomicAdd(&acc[0], ni);
            atomicAdd(&acc[1], nt);
        }
        __syncthreads();
        if (tid == 0) A.sums[blockIdx.x] = make_int4(acc[0], acc[1], failed, 0);
        grid.sync();
        if (tid < 5) acc[tid] = 0;
        __syncthreads();
        int before_i = 0, before_t = 0, all_i = 0, all_t = 0, any = 0;
        for (int b = tid; b < (int)gridDim.x; b += kCollapseThreads) {
            const int4 v = __ldcg(A.sums + b);
            all_i += v.x;
            all_t += v.y;
            any |= v.z;
            if (b < (int)blockIdx.x) {
                before_i += v.x;
                before_t += v.y;
            }
        }
        before_i = __reduce_add_sync(~0u, before_i);
        before_t = __reduce_add_sync(~0u, before_t);
        all_i = __reduce_add_sync(~0u, all_i);
        all_t = __reduce_add_sync(~0u, all_t);
        any = __reduce_or_sync(~0u, (unsigned)any);
        if ((tid & 31) == 0) {
            atomicAdd(&acc[0], before_i);
            atomicAdd(&acc[1], before_t);
            atomicAdd(&acc[2], all_i);
            atomicAdd(&acc[3], all_t);
            atomicOr(&acc[4], any);
        }
        __syncthreads();
        before_i = acc[0];
        before_t = acc[1];
        const int next_n = acc[2], level_tris = acc[3];
        if (acc[4] || next_n > A.list_cap || next_n > A.wide_cap - next_start || level_tris > A.n_tris - tri_start) {
            if (!acc[4]) raise_err(A.err, kErrWideOverflow);
            return;  // every block: the totals are the same
        }
        for (int base = t0; base < t1; base += kCollapseThreads) {
            const int t = base + tid;
            const int2 v = t < t1 ? A.counts[t] : make_int2(0, 0);
            int tot_i, tot_t;
            s_inner[tid] = before_i + block_excl_scan(v.x, ws, &tot_i);
            s_tri[tid] = before_t + block_excl_scan(v.y, ws, &tot_t);
            before_i += tot_i;
            before_t += tot_t;
            __syncthreads();
            const int m = min(kCollapseThreads, t1 - base);
            for (int j = tid >> 3; j < m; j += kCollapseThreads / 8)
                collapse_emit(A, A.child_list + 8 * (size_t)(base + j), level_start + base + j, s_inner[j],
                              next_start + s_inner[j], tri_start + s_tri[j], A.tasks[cur ^ 1], &failed);
            __syncthreads();
        }
        grid.sync();
        level_start = next_start;
        tri_start += level_tris;
        ntasks = next_n;
    }
    if (blockIdx.x == 0 && tid == 0) {
        A.result[0] = level_start;
        A.result[1] = tri_start;
        A.result[2] = levels;
    }
}

float host_f(int i) { float f; memcpy(&f, &i, 4); return f; }
float host_o2f(int i) { return host_f(i >= 0 ? i : i ^ 0x7fffffff); }

// The build's working arrays lie in one allocation: a cudaMalloc and a cudaFree
// of 32 MB cost 35 and 43 us each, and there were 26 (1.4 of the 11.5 ms of a
// 5.2M-triangle build, 0.45 of the 2.25 ms at 82k).  Arrays are first asked for,
// then placed.
class Arena {
  public:
    ~Arena() { dfree(base_); }
    template <class T> void want(T **p, size_t count) {
        asks_.push_back({reinterpret_cast<void **>(p), size_});
        size_ += (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
    }
    kgk_status place(const char *what) {
        KGK_TRY(dalloc(&base_, size_, what));
        for (const auto &a : asks_) *a.first = base_ + a.second;
        return KGK_OK;
    }

  private:
    std::vector<std::pair<void **, size_t>> asks_;
    unsigned char *base_ = nullptr;
    size_t size_ = 0;
};

}  // namespace

// ---------------------------------------------------------------------------
kgk_status bvh_build(DevScene &s, cudaStream_t st, BvhBuildStats *out) {
    const int n = s.n_tris;
    if (n <= 0) return fail(KGK_ERR_INVALID_ARGUMENT, "bvh_build: scene has no triangles");
    const int max_leaf = n > kLargeSceneTris ? kLeafLarge : kMaxLeaf;
    dfree(s.nodes);
    s.nodes = nullptr;
    dfree(s.tri_rec);
    s.tri_rec = nullptr;
    s.n_nodes = 0;

    cudaEvent_t e0, e1;
    KGK_CUDA(cudaEventCreate(&e0));
    KGK_CUDA(cudaEventCreate(&e1));
    KGK_CUDA(cudaEventRecord(e0, st));

    float4 *plo, *phi;
    int *ref, *ref_tmp, *gbounds, *err, *bfirst, *bcount;
    BinNode *nodes;
    unsigned *dec;
    const int cap = 2 * n + 1;
    Task *d_tasks;
    Split *d_splits;
    Chunk *d_chunks;
    int *d_gbins, *d_hist, *d_before;
    unsigned short *d_codes;
    const int max_large = n / kSmall + 2;
    const int chunk = n > kLargeChunkTris ? kChunkLarge : kChunkSmall;
    const int max_chunks = n / chunk + 2 * max_large + 2;
    CollapseArgs C{};
    C.cap = cap;
    C.list_cap = n / 2 + 2;  // a level's tasks hold two triangles or more each
    C.wide_cap = n + 1;
    C.n_tris = n;
    C.max_leaf = max_leaf;
    int dev = 0, sms = 0, resident = 0;
    KGK_CUDA(cudaGetDevice(&dev));
    KGK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    KGK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_collapse, kCollapseThreads, 0));
    if (resident < 1) return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: the collapse does not fit an SM");
    // never more blocks than fit at once, nor than have a task for every 8 lanes
    const int collapse_blocks = std::max(1, std::min(sms * resident, n / (kCollapseThreads / 8)));
    Arena arena;
    arena.want(&plo, n);
    arena.want(&phi, n);
    arena.want(&ref, n);
    arena.want(&ref_tmp, n);
    arena.want(&gbounds, 16);
    arena.want(&err, 4);
    arena.want(&nodes, cap);
    arena.want(&bfirst, cap);
    arena.want(&bcount, cap);
    arena.want(&dec, cap);
    arena.want(&d_tasks, max_large);
    arena.want(&d_splits, max_large);
    arena.want(&d_chunks, max_chunks);
    arena.want(&d_gbins, (size_t)max_large * 3 * kBins * kBinInts);
    arena.want(&d_hist, (size_t)max_chunks * kHist);
    arena.want(&d_before, max_chunks);
    arena.want(&d_codes, n);
    arena.want(&C.tasks[0], C.list_cap);
    arena.want(&C.tasks[1], C.list_cap);
    arena.want(&C.child_list, 8 * (size_t)C.list_cap);
    arena.want(&C.counts, C.list_cap);
    arena.want(&C.sums, collapse_blocks);
    arena.want(&C.result, 4);
    KGK_TRY(arena.place("bvh build"));
    // slots the small builder reserves but does not use read as leaves
    // (hi.w = -1) that no node points to
    KGK_CUDA(cudaMemsetAsync(nodes, 0xFF, (size_t)cap * sizeof(BinNode), st));
    KGK_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));

    k_init_bounds<<<1, 32, 0, st>>>(gbounds);
    k_prim_bounds<<<std::min((n + 255) / 256, 1216), 256, 0, st>>>(s.verts, n, plo, phi, ref, gbounds);
    KGK_CUDA(cudaGetLastError());
    int hb[12];
    KGK_CUDA(cudaMemcpyAsync(hb, gbounds, sizeof hb, cudaMemcpyDeviceToHost, st));
    KGK_CUDA(cudaStreamSynchronize(st));

    // root
    Task root{};
    root.node = 0;
    root.begin = 0;
    root.count = n;
    for (int a = 0; a < 3; ++a) {
        root.clo[a] = host_o2f(hb[6 + a]);
        root.chi[a] = host_o2f(hb[9 + a]);
    }
    std::vector<int> h_ids;
    std::vector<BinNode> h_vals;
    std::vector<int> h_first, h_count, h_parent;  // h_parent[q]: of nodes 1 + 2q and 2 + 2q
    auto add_node = [&](int id, const float *lo, const float *hi, int first, int count) {
        BinNode nd;
        nd.lo = make_float4(lo[0], lo[1], lo[2], 0.0f);
        nd.hi = make_float4(hi[0], hi[1], hi[2], 0.0f);
        h_ids.push_back(id);
        h_vals.push_back(nd);
        h_first.push_back(first);
        h_count.push_back(count);
        return (int)h_ids.size() - 1;
    };
    float rlo[3] = {host_o2f(hb[0]), host_o2f(hb[1]), host_o2f(hb[2])};
    float rhi[3] = {host_o2f(hb[3]), host_o2f(hb[4]), host_o2f(hb[5])};
    add_node(0, rlo, rhi, 0, n);
    int node_counter = 1;

    std::vector<Task> large, small;
    if (n > kSmall) large.push_back(root);
    else small.push_back(root);

    // the refs go back and forth between two buffers, a level each way; a task
    // that becomes small stays where its level put it
    int *const refs[2] = {ref, ref_tmp};
    int cur = 0;
    while (!large.empty()) {
        const int nL = (int)large.size();
        if (nL > max_large) return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: large-task list overflow");
        std::vector<Chunk> chunks;
        for (int t = 0; t < nL; ++t) {
            large[t].first_chunk = (int)chunks.size();
            for (int b = large[t].begin; b < large[t].begin + large[t].count; b += chunk)
                chunks.push_back({t, b, std::min(b + chunk, large[t].begin + large[t].count), 0});
        }
        const int nc = (int)chunks.size();
        if (nc > max_chunks) return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: chunk list overflow");
        KGK_CUDA(cudaMemcpyAsync(d_tasks, large.data(), sizeof(Task) * nL, cudaMemcpyHostToDevice, st));
        KGK_CUDA(cudaMemcpyAsync(d_chunks, chunks.data(), sizeof(Chunk) * nc, cudaMemcpyHostToDevice, st));
        const int nbins = nL * 3 * kBins * kBinInts;
        k_init_global_bins<<<(nbins + 255) / 256, 256, 0, st>>>(d_gbins, nL);
        k_bin_large<<<nc, kThreads, 0, st>>>(d_chunks, d_tasks, refs[cur], plo, phi, d_gbins, d_codes, d_hist);
        k_split_large<<<nL, 32, 0, st>>>(d_tasks, nL, d_gbins, d_splits, chunk, d_hist, d_before, err);
        KGK_CUDA(cudaGetLastError());
        std::vector<Split> sp(nL);
        KGK_CUDA(cudaMemcpyAsync(sp.data(), d_splits, sizeof(Split) * nL, cudaMemcpyDeviceToHost, st));
        KGK_CUDA(cudaStreamSynchronize(st));
        // runs while the next level's tasks are listed
        auto *scatter = chunk == kChunkLarge ? k_part_scatter<kChunkLarge / kThreads>
                                             : k_part_scatter<kChunkSmall / kThreads>;
        scatter<<<nc, kThreads, 0, st>>>(d_chunks, d_tasks, d_splits, d_before, refs[cur], d_codes, refs[cur ^ 1], n,
                                         err);
        KGK_CUDA(cudaGetLastError());
        for (int t = 0; t < nL; ++t)
            if (sp[t].nleft < 1 || sp[t].nleft >= large[t].count)
                return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: a split left one side empty");
        std::vector<Task> next;
        for (int t = 0; t < nL; ++t) {
            const Task &tk = large[t];
            const Split &s2 = sp[t];
            const int l = node_counter, r = node_counter + 1;
            node_counter += 2;
            // parent's child links (ids are handed out in order: an id is its place in the list)
            if (tk.node >= (int)h_ids.size() || h_ids[tk.node] != tk.node)
                return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: lost a parent node");
            h_vals[tk.node].lo.w = host_f(l);
            h_vals[tk.node].hi.w = host_f(r);
            h_parent.push_back(tk.node);
            for (int side = 0; side < 2; ++side) {
                Task c{};
                c.node = side == 0 ? l : r;
                c.buf = cur ^ 1;
                c.begin = side == 0 ? tk.begin : tk.begin + s2.nleft;
                c.count = side == 0 ? s2.nleft : tk.count - s2.nleft;
                for (int a = 0; a < 3; ++a) { c.clo[a] = s2.clo[side][a]; c.chi[a] = s2.chi[side][a]; }
                add_node(c.node, s2.lo[side], s2.hi[side], c.begin, c.count);
                if (c.count > kSmall) next.push_back(c);
                else small.push_back(c);
            }
        }
        large.swap(next);
        cur ^= 1;
    }

    // small subtrees: each task of m primitives owns 2m-2 node slots
    const int n_top = node_counter, ns = (int)small.size();
    std::vector<int> sb(ns);
    {
        long long next = node_counter;
        for (int t = 0; t < ns; ++t) {
            sb[t] = (int)next;
            next += 2LL * small[t].count - 2;
        }
        if (next > cap) return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: node budget exceeded");
        node_counter = (int)next;
    }
    Task *d_small;
    int *d_sb, *d_parent, *d_visits, *d_ids, *d_first, *d_count;
    BinNode *d_vals;
    float4 *dp_rows, *dp_roots;
    const int n_pairs = (int)h_parent.size(), m = (int)h_ids.size();
    Arena top;
    top.want(&d_small, ns);
    top.want(&d_sb, ns);
    top.want(&d_parent, n_pairs);
    top.want(&d_visits, n_pairs);
    top.want(&dp_rows, 2 * (size_t)n_top);
    top.want(&dp_roots, 2 * (size_t)ns);
    top.want(&d_ids, m);
    top.want(&d_first, m);
    top.want(&d_count, m);
    top.want(&d_vals, m);
    KGK_TRY(top.place("bvh build, top nodes"));
    // the large levels' nodes (before the small kernel links into them)
    KGK_CUDA(cudaMemcpyAsync(d_ids, h_ids.data(), sizeof(int) * m, cudaMemcpyHostToDevice, st));
    KGK_CUDA(cudaMemcpyAsync(d_first, h_first.data(), sizeof(int) * m, cudaMemcpyHostToDevice, st));
    KGK_CUDA(cudaMemcpyAsync(d_count, h_count.data(), sizeof(int) * m, cudaMemcpyHostToDevice, st));
    KGK_CUDA(cudaMemcpyAsync(d_vals, h_vals.data(), sizeof(BinNode) * m, cudaMemcpyHostToDevice, st));
    k_write_nodes<<<(m + 255) / 256, 256, 0, st>>>(d_ids, d_vals, d_first, d_count, m, nodes, bfirst, bcount, cap,
                                                   err);
    KGK_CUDA(cudaGetLastError());
    KGK_CUDA(cudaMemcpyAsync(d_small, small.data(), sizeof(Task) * ns, cudaMemcpyHostToDevice, st));
    KGK_CUDA(cudaMemcpyAsync(d_sb, sb.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
    KGK_CUDA(cudaFuncSetAttribute(k_small_build, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SbShared)));
    k_small_build<<<ns, kSbThreads, sizeof(SbShared), st>>>(d_small, d_sb, ns, plo, phi, ref, ref_tmp, nodes, bfirst,
                                                            bcount, cap, max_leaf, err);
    KGK_CUDA(cudaGetLastError());

    // the collapse's cost table, bottom up over the binary tree
    if (n_pairs > 0) {
        KGK_CUDA(cudaMemcpyAsync(d_parent, h_parent.data(), sizeof(int) * n_pairs, cudaMemcpyHostToDevice, st));
        KGK_CUDA(cudaMemsetAsync(d_visits, 0, sizeof(int) * n_pairs, st));
    }
    KGK_CUDA(cudaFuncSetAttribute(k_dp_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DpShared)));
    k_dp_small<<<ns, kDpThreads, sizeof(DpShared), st>>>(d_small, d_sb, ns, nodes, cap, dp_roots, dec, err);
    k_dp_top<<<(ns + 127) / 128, 128, 0, st>>>(d_small, ns, nodes, d_parent, n_top, dp_roots, dp_rows, dec, d_visits,
                                               err);
    KGK_CUDA(cudaGetLastError());
    int herr = 0;
    KGK_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    KGK_CUDA(cudaStreamSynchronize(st));
    if (herr != 0)
        return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: binary build check failed (code " + std::to_string(herr) + ")");

    // collapse
    KGK_TRY(dalloc(&C.wide, C.wide_cap, "wide BVH nodes"));
    s.nodes = C.wide;
    KGK_TRY(dalloc(&C.tri_rec, 3 * (size_t)n, "BVH triangle records"));
    s.tri_rec = C.tri_rec;
    C.nodes = nodes;
    C.bfirst = bfirst;
    C.bcount = bcount;
    C.ref = ref;
    C.dec = dec;
    C.verts = s.verts;
    C.attr = s.attr;
    C.mats = s.mats;
    C.n_mats = s.n_mats;
    C.err = err;
    KGK_CUDA(cudaMemsetAsync(C.result, 0, 4 * sizeof(int), st));
    void *args[] = {&C};
    KGK_CUDA(cudaLaunchCooperativeKernel((const void *)k_collapse, dim3(collapse_blocks), dim3(kCollapseThreads), args,
                                         0, st));
    int result[4];
    KGK_CUDA(cudaMemcpyAsync(result, C.result, sizeof result, cudaMemcpyDeviceToHost, st));
    KGK_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    KGK_CUDA(cudaEventRecord(e1, st));
    KGK_CUDA(cudaStreamSynchronize(st));
    if (herr != 0)
        return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: collapse check failed (code " + std::to_string(herr) + ")");
    if (result[1] != n)
        return fail(KGK_ERR_DEVICE_CHECK, "bvh_build: collapse placed " + std::to_string(result[1]) +
                                              " of " + std::to_string(n) + " triangles");
    s.n_nodes = result[0];
    s.root = 0;
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (out) {
        out->n_binary = (uint64_t)node_counter;
        out->n_wide = (uint64_t)s.n_nodes;
        out->max_depth = (uint32_t)result[2];
        out->max_leaf = max_leaf;
        out->ms = ms;
        out->sah = 0;
    }
    return KGK_OK;
}

// ---------------------------------------------------------------------------
// Host-side structural validation of the wide BVH.
// ---------------------------------------------------------------------------
kgk_status bvh_validate(const DevScene &s, cudaStream_t st) {
    if (!s.nodes || !s.tri_rec) return fail(KGK_ERR_NOT_BUILT, "bvh_validate: no BVH");
    const int n = s.n_tris;
    std::vector<WideNode> nodes(s.n_nodes);
    std::vector<float4> tri(3 * (size_t)n);
    KGK_CUDA(cudaMemcpyAsync(nodes.data(), s.nodes, sizeof(WideNode) * nodes.size(), cudaMemcpyDeviceToHost, st));
    KGK_CUDA(cudaMemcpyAsync(tri.data(), s.tri_rec, sizeof(float4) * tri.size(), cudaMemcpyDeviceToHost, st));
    KGK_CUDA(cudaStreamSynchronize(st));
    std::vector<int> seen(n, 0);
    std::vector<int> visited(nodes.size(), 0);
    struct Item { int node; float lo[3], hi[3]; };
    std::vector<Item> stack;
    Item root{0, {-INFINITY, -INFINITY, -INFINITY}, {INFINITY, INFINITY, INFINITY}};
    stack.push_back(root);
    auto u = [](float f) { unsigned x; memcpy(&x, &f, 4); return x; };
    auto byte = [](unsigned w, int k) { return (w >> (8 * k)) & 0xffu; };
    while (!stack.empty()) {
        Item it = stack.back();
        stack.pop_back();
        if (it.node < 0 || it.node >= (int)nodes.size())
            return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: child index out of range");
        if (visited[it.node]++) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: node reached twice");
        const WideNode &w = nodes[it.node];
        float p[3] = {w.n0.x, w.n0.y, w.n0.z};
        unsigned e = u(w.n0.w);
        float sc[3];
        for (int a = 0; a < 3; ++a) sc[a] = ldexpf(1.0f, (int)byte(e, a) - 127);
        const unsigned field = u(w.n1.z), imask = byte(field, 3);
        int child_base = (int)u(w.n1.x), tri_base = (int)u(w.n1.y);
        unsigned ql[3][2] = {{u(w.n2.x), u(w.n2.y)}, {u(w.n3.x), u(w.n3.y)}, {u(w.n4.x), u(w.n4.y)}};
        unsigned qh[3][2] = {{u(w.n2.z), u(w.n2.w)}, {u(w.n3.z), u(w.n3.w)}, {u(w.n4.z), u(w.n4.w)}};
        int inner_k = 0;
        for (int sl = 0; sl < 8; ++sl) {
            const bool inner = (imask >> sl) & 1u;
            const unsigned b0 = (field >> sl) & 1u, b1 = (field >> (sl + 8)) & 1u, b2 = (field >> (sl + 16)) & 1u;
            if (b1 > b0 || b2 > b1 || (inner && b0)) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: bad leaf bits");
            if (!inner && !b0) continue;
            float lo[3], hi[3];
            for (int a = 0; a < 3; ++a) {
                lo[a] = p[a] + (float)byte(ql[a][sl / 4], sl % 4) * sc[a];
                hi[a] = p[a] + (float)byte(qh[a][sl / 4], sl % 4) * sc[a];
                if (lo[a] > hi[a]) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: inverted child box");
            }
            if (inner) {
                Item c;
                c.node = child_base + inner_k++;
                for (int a = 0; a < 3; ++a) { c.lo[a] = lo[a]; c.hi[a] = hi[a]; }
                stack.push_back(c);
            } else {
                const int k = (int)(b0 + b1 + b2);
                for (int j = 0; j < k; ++j) {
                    int ti = tri_base + __builtin_popcount(field & ((1u << (sl + 8 * j)) - 1u));
                    if (ti < 0 || ti >= n) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: triangle index out of range");
                    int id;
                    memcpy(&id, &tri[3 * (size_t)ti].w, 4);
                    if (id < 0 || id >= n || seen[id]++) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: triangle referenced twice");
                    for (int v = 0; v < 3; ++v) {
                        const float4 &q = tri[3 * (size_t)ti + v];
                        float c3[3] = {q.x, q.y, q.z};
                        for (int a = 0; a < 3; ++a) {
                            float tol = 1e-6f * (fabsf(c3[a]) + 1.0f);
                            if (c3[a] < lo[a] - tol || c3[a] > hi[a] + tol)
                                return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: triangle outside its leaf box");
                        }
                    }
                }
            }
        }
        if (__builtin_popcount(imask) != inner_k) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: imask count mismatch");
    }
    for (int i = 0; i < n; ++i)
        if (seen[i] != 1) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: triangle " + std::to_string(i) + " not referenced");
    for (size_t i = 0; i < nodes.size(); ++i)
        if (!visited[i]) return fail(KGK_ERR_DEVICE_CHECK, "bvh_validate: unreachable node");
    return KGK_OK;
}

}  // namespace kgk
