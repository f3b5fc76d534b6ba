// trace.cu - batch closest-hit and occlusion queries (the parity entry
// points kgk_trace_closest / kgk_trace_any): persistent kernels, one ray per
// lane at a time, lanes refilled from a shared counter.
#include <algorithm>

#include "kgk_internal.h"
#include "traverse.cuh"

namespace kgk {
namespace {

// kgk_ray is 40 B (dir, org, double): rays are read as five float2.
__device__ __forceinline__ void load_ray(const kgk_ray *rays, int i, float3 &o, float3 &d) {
    const float2 *p = reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(rays) + 40 * (size_t)i);
    const float2 a = p[0], b = p[1], c = p[2], e = p[3];
    d = f3(a.x, a.y, b.x);
    o = f3(c.x, c.y, e.x);
}

__device__ __forceinline__ void flush_counters(TraceCounters *ctr, unsigned nodes, unsigned tris,
                                               unsigned overflow, unsigned rays) {
    unsigned long long n = nodes, t = tris, o = overflow, r = rays;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        n += __shfl_xor_sync(~0u, n, s);
        t += __shfl_xor_sync(~0u, t, s);
        o += __shfl_xor_sync(~0u, o, s);
        r += __shfl_xor_sync(~0u, r, s);
    }
    if ((threadIdx.x & 31) == 0) {
        if (r) atomicAdd(&ctr->rays, r);
        if (o) atomicAdd(&ctr->overflows, o);
        if (n) atomicAdd(&ctr->nodes, n);
        if (t) atomicAdd(&ctr->tris, t);
    }
}

// Lanes take new rays (one atomic per warp) whenever kRefill or more of them
// are idle, so a warp does not wait for its longest ray.  warp_step visits a
// ray's nodes in trace_closest's / trace_any's order and tests the triangles of a
// visit in the order of its pairs; the closest hit, ties by the smaller id, does not
// depend on that, so the answers are the same.  kOwn: each lane tests its own
// triangles (own_step).
constexpr int kRefill = 8;

template <bool kAny, bool kCount, bool kOwn>
__global__ void __launch_bounds__(128, 8) k_trace(const WideNode *__restrict__ nodes, unsigned n_nodes,
                                               const float4 *__restrict__ tri, unsigned n_tris,
                                               const kgk_ray *__restrict__ rays, const float *__restrict__ tmax,
                                               int n, int32_t *id_out, float *t_out, uint8_t *occ,
                                               TraceCounters *ctr) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt = (1u << lane) - 1u;
    bool active = false, exhausted = false;
    int i = 0;
    unsigned done = 0;
    __shared__ WarpRays s_w[kOwn ? 1 : 4];  // kOwn: not used
    WarpRays &w = s_w[kOwn ? 0 : threadIdx.x >> 5];
    Lane c;
    OwnRay own;
    TravStack stk;
    TravStats st{0, 0, 0};
    while (true) {
        const unsigned idle = __ballot_sync(~0u, !active);
        if (!exhausted && __popc(idle) >= kRefill) {
            int base = 0;
            if (lane == 0) base = (int)atomicAdd(&ctr->fetch, (unsigned long long)__popc(idle));
            base = __shfl_sync(~0u, base, 0);
            if (base + __popc(idle) >= n) exhausted = true;
            if (!active) {
                i = base + __popc(idle & lt);
                if (i < n) {
                    float3 o, d;
                    load_ray(rays, i, o, d);
                    const float limit = kAny && tmax ? tmax[i] : kBigT;
                    if (kOwn) own_init(own, o, d, limit);
                    else lane_init(w, c, o, d, limit, kAny);
                    active = true;
                }
            }
        }
        if (!__any_sync(~0u, active)) break;
        const bool ended = kOwn ? active && own_step<kAny, kCount>(nodes, n_nodes, tri, n_tris, own, stk, st)
                                : warp_step<kCount>(nodes, n_nodes, tri, n_tris, w, c, stk, active, kAny, st);
        if (ended) {
            active = false;
            ++done;
            const bool hit = kOwn ? own.best_id != kNoHit : w.slot[lane] >= 0;
            if (kAny) {
                occ[i] = hit ? 1 : 0;
            } else {
                id_out[i] = hit ? (kOwn ? own.best_id : w.id[lane]) : -1;
                t_out[i] = hit ? (kOwn ? own.best_t : c.best_t) : kBigT;
            }
        }
    }
    flush_counters(ctr, st.nodes, st.tris, st.overflow, done);
}

// Trees of a few nodes by own_step: pairs : own triangles, us.
//   any-hit, 4,096 / 2^20 / 2^22 rays: closed rooms of 12 triangles 8.8 : 8.2, 47.6 :
//   39.2, 160 : 127, of 72 10.0 : 9.8, 58.8 : 49.1, 197 : 160, of 972 18.2 : 15.7, 91.7 :
//   69.2, 311 : 229, the Cornell box 12.5 : 13.7, 65.1 : 52.6, 221 : 174; spheres over a
//   ground, 82 11.6 : 11.6, 44.7 : 43.0, 143 : 133, 642 13.6 : 14.2, 46.8 : 46.4, 140 : 137;
//   random triangles, 24 9.8 : 10.1, 49.7 : 52.0, 163 : 172, 1,000 32.6 : 40.4, 209 : 220,
//   738 : 770.  Larger rooms gain as much, larger spheres lose up to 7 % of 2^20 rays.
//   Closest hits, 4,096 / 2^18 / 2^22 rays: rooms of 12 10.0 : 8.0, 28.7 : 26.0, 170 : 135,
//   of 72 14.4 : 15.7, 35.2 : 32.9, 301 : 262, the box 16.2 : 18.8, 40.7 : 42.7, 377 : 385,
//   82 spheres' triangles 11.6 : 11.7, 29.7 : 28.4, 152 : 143; random triangles, 24 9.9 :
//   11.8 (4,096), 173 : 182 (2^22), 128 30.2 : 38.4, 663 : 745; rooms of 972 even.
// In no case measured are own triangles behind the step that tested them so before
// the pairs; the pairs were, by up to 27 %, in rooms.
constexpr int kOwnAnyTris = 1024, kOwnTris = 128;
constexpr size_t kOwnRays = 1 << 18;

int grid_for(size_t n) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
    }
    return (int)std::min<size_t>((size_t)sms * 8, (n + 127) / 128);
}

}  // namespace

kgk_status trace_closest_dev(const DevScene &s, const kgk_ray *rays, size_t n, int32_t *id, float *t,
                             bool count, TraceCounters *ctr, cudaStream_t st) {
    if (n == 0) return KGK_OK;
    if (n > 0x7fffffff) return fail(KGK_ERR_INVALID_ARGUMENT, "trace: too many rays");
    const bool own = s.n_tris <= kOwnTris && n >= kOwnRays;
    auto *k = count ? (own ? k_trace<false, true, true> : k_trace<false, true, false>)
                    : (own ? k_trace<false, false, true> : k_trace<false, false, false>);
    k<<<grid_for(n), 128, 0, st>>>(s.nodes, (unsigned)s.n_nodes, s.tri_rec, (unsigned)s.n_tris, rays, nullptr, (int)n,
                                   id, t, nullptr, ctr);
    KGK_CUDA(cudaGetLastError());
    return KGK_OK;
}

kgk_status trace_any_dev(const DevScene &s, const kgk_ray *rays, const float *tmax, size_t n, uint8_t *occ,
                         TraceCounters *ctr, cudaStream_t st) {
    if (n == 0) return KGK_OK;
    if (n > 0x7fffffff) return fail(KGK_ERR_INVALID_ARGUMENT, "trace: too many rays");
    auto *k = s.n_tris <= kOwnAnyTris ? k_trace<true, false, true> : k_trace<true, false, false>;
    k<<<grid_for(n), 128, 0, st>>>(s.nodes, (unsigned)s.n_nodes, s.tri_rec, (unsigned)s.n_tris, rays, tmax, (int)n,
                                   nullptr, nullptr, occ, ctr);
    KGK_CUDA(cudaGetLastError());
    return KGK_OK;
}

}  // namespace kgk
