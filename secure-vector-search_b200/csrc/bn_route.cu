// bn_route.cu -- IVF routing on the device: the nprobe nearest centroids of
// every query of a batch (ivf-index/src/ivf.rs:150-164 probe_route).
//
// The distance is the reference's scalar l2_f32 (ivf-index/src/distance.rs:
// 30-36): sqrt of the sum over the dimensions, in order, of (x - y)^2, every
// operation rounded on its own (no fused multiply-add), so each distance is
// bit-identical to the host form (bn_host_probe_route, compiled without
// contraction).  Centroids are ranked by (distance, index): total_cmp order
// for the non-negative distances, ties to the lower index.  The reference's
// AVX-512 build sums in 16 lanes with fused multiply-adds instead and may
// rank near-ties differently; its scalar build agrees with this one.

#include "bn_internal.cuh"

namespace bn {
namespace {

constexpr uint32_t RT_THREADS = 64;
constexpr uint32_t RT_BATCH = 32, RT_DEPTH = 6;  // centroid values per copy group, groups in flight
constexpr uint32_t RT_SORT_THREADS = 1024;

// One of a thread's own centroid values into its own column of the ring (only
// this thread reads it, so the copy groups need no barrier).
__device__ __forceinline__ void copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// dist[q][c] for centroid c = blockIdx.x * 64 + threadIdx.x and QPT queries
// from blockIdx.y * QPT on; centroids are stored dimension-major (cent_t[i][c])
// so a warp's loads are coalesced.  The sum over the dimensions is a serial
// chain by definition, so the kernel is bound by the latency of its loads: a
// thread keeps RT_DEPTH groups of RT_BATCH of them in flight through a ring of
// its own in shared memory (one load after the other: 54 us for 640 lists of 768
// dimensions), and each serves QPT queries, whose chains overlap.  Dimensions past
// d are zero on both sides and add +0 to a sum that is never -0.
template <int QPT>
__global__ void __launch_bounds__(RT_THREADS)
route_dist_kernel(const float* __restrict__ cent_t, uint32_t nlist, uint32_t d, const float* __restrict__ queries,
                  uint32_t nq, float* __restrict__ dist) {
    extern __shared__ float ring[];  // [RT_DEPTH][RT_BATCH][RT_THREADS], then qs [d rounded up to RT_BATCH][QPT]
    float* qs = ring + RT_DEPTH * RT_BATCH * RT_THREADS;
    const uint32_t q0 = blockIdx.y * QPT;
    const uint32_t groups = (d + RT_BATCH - 1) / RT_BATCH;
    const uint32_t c = blockIdx.x * RT_THREADS + threadIdx.x;
    const bool on = c < nlist;
    auto fetch = [&](uint32_t g) {
        float* dst = ring + (g % RT_DEPTH) * RT_BATCH * RT_THREADS + threadIdx.x;
#pragma unroll 8
        for (uint32_t k = 0; k < RT_BATCH; ++k) {
            const uint32_t i = g * RT_BATCH + k;
            if (on && i < d) copy4(dst + k * RT_THREADS, cent_t + (uint64_t)i * nlist + c);
            else dst[k * RT_THREADS] = 0.0f;
        }
    };
    for (uint32_t g = 0; g < RT_DEPTH - 1; ++g) {
        if (g < groups) fetch(g);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int u = 0; u < QPT; ++u)
        for (uint32_t i = threadIdx.x; i < groups * RT_BATCH; i += RT_THREADS)
            qs[i * QPT + u] = i < d && q0 + u < nq ? queries[(uint64_t)(q0 + u) * d + i] : 0.0f;
    __syncthreads();
    float s[QPT];
#pragma unroll
    for (int u = 0; u < QPT; ++u) s[u] = 0.0f;
    for (uint32_t g = 0; g < groups; ++g) {
        if (g + RT_DEPTH - 1 < groups) fetch(g + RT_DEPTH - 1);  // the slot read in the last round
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group %0;" ::"n"(RT_DEPTH - 1) : "memory");
        const float* src = ring + (g % RT_DEPTH) * RT_BATCH * RT_THREADS + threadIdx.x;
        const float* qg = qs + g * RT_BATCH * QPT;
#pragma unroll
        for (uint32_t k = 0; k < RT_BATCH; ++k) {
            const float x = src[k * RT_THREADS];
#pragma unroll
            for (int u = 0; u < QPT; ++u) {
                const float t = __fsub_rn(qg[k * QPT + u], x);
                s[u] = __fadd_rn(s[u], __fmul_rn(t, t));
            }
        }
    }
#pragma unroll
    for (int u = 0; u < QPT; ++u)
        if (on && q0 + u < nq) dist[(uint64_t)(q0 + u) * nlist + c] = __fsqrt_rn(s[u]);
}

// At most 1024 lists: one key per thread.  Exchanges over fewer than 32
// threads are shuffles; the 15 wider ones (of 55 at 1024 keys) go through
// shared memory, two buffers in turn so that each costs one barrier.
__global__ void __launch_bounds__(RT_SORT_THREADS)
route_select_small_kernel(const float* __restrict__ dist, uint32_t nlist, uint32_t np, uint32_t* __restrict__ probes) {
    __shared__ uint64_t xch[2][RT_SORT_THREADS];
    const uint32_t q = blockIdx.x, i = threadIdx.x;  // blockDim.x: a power of two, at least 32
    uint64_t key = i < nlist ? ((uint64_t)__float_as_uint(dist[(uint64_t)q * nlist + i]) << 32) | i : ~0ull;
    uint32_t buf = 0;
    for (uint32_t size = 2; size <= blockDim.x; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            uint64_t other;
            if (stride >= 32) {
                xch[buf][i] = key;
                __syncthreads();
                other = xch[buf][i ^ stride];
                buf ^= 1;
            } else {
                other = __shfl_xor_sync(0xffffffffu, key, stride);
            }
            const bool low = (i & stride) == 0, up = (i & size) == 0;
            key = (low == up) == (key < other) ? key : other;
        }
    if (i < np) probes[(uint64_t)q * np + i] = (uint32_t)key;
}

// One CTA per query: keys (distance bits << 32 | index) -- the bits of a
// non-negative float order like the float -- bitonic-sorted ascending in
// shared memory; the first np indices are the probes.
__global__ void __launch_bounds__(RT_SORT_THREADS)
route_select_kernel(const float* __restrict__ dist, uint32_t nlist, uint32_t np, uint32_t pow2,
                    uint32_t* __restrict__ probes) {
    extern __shared__ uint64_t keys[];
    const uint32_t q = blockIdx.x;
    for (uint32_t i = threadIdx.x; i < pow2; i += blockDim.x)
        keys[i] = i < nlist ? ((uint64_t)__float_as_uint(dist[(uint64_t)q * nlist + i]) << 32) | i : ~0ull;
    for (uint32_t size = 2; size <= pow2; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < pow2 / 2; i += blockDim.x) {
                const uint32_t lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const bool up = (lo & size) == 0;
                const uint64_t a = keys[lo], b = keys[hi];
                if ((a > b) == up) {
                    keys[lo] = b;
                    keys[hi] = a;
                }
            }
        }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < np; i += blockDim.x) probes[(uint64_t)q * np + i] = (uint32_t)keys[i];
}

}  // namespace
}  // namespace bn

using namespace bn;
using namespace bn::api;

namespace {
constexpr uint32_t ROUTE_MAX_NLIST = 16384;  // the sort's keys fit in 128 KB of shared memory
constexpr uint32_t ROUTE_MAX_DIM = 8192;
}  // namespace

extern "C" {

int bn_ivf_set_centroids(bn_ivf* v, const float* centroids, uint32_t d) {
    if (!v || !centroids) return fail(BN_EINVAL, "null argument");
    if (d == 0 || d > ROUTE_MAX_DIM) return fail(BN_EINVAL, "centroid dimension %u not in 1..=%u", d, ROUTE_MAX_DIM);
    if (v->nlist > ROUTE_MAX_NLIST) return fail(BN_EINVAL, "%u lists exceed the %u the router ranks", v->nlist, ROUTE_MAX_NLIST);
    std::lock_guard<std::mutex> g(v->e.mu);
    CU(cudaSetDevice(v->e.ctx->device));
    std::vector<float> t((uint64_t)d * v->nlist);
    for (uint32_t c = 0; c < v->nlist; ++c)
        for (uint32_t i = 0; i < d; ++i) t[(uint64_t)i * v->nlist + c] = centroids[(uint64_t)c * d + i];
    TRY(v->cent_t.alloc(v->e.ctx, std::max<uint64_t>(t.size(), 1) * 4));
    CU(cudaMemcpy(v->cent_t.p, t.data(), t.size() * 4, cudaMemcpyHostToDevice));
    v->cent_d = d;
    return BN_OK;
}

int bn_ivf_route(bn_ivf* v, uint32_t B, const float* queries, uint32_t nprobe, uint32_t* probes) {
    if (!v) return fail(BN_EINVAL, "null handle");
    if (B == 0) return BN_OK;
    if (!queries || !probes) return fail(BN_EINVAL, "null argument");
    if (!v->cent_d) return fail(BN_EINVAL, "no centroids: call bn_ivf_set_centroids first");
    if (nprobe == 0) return fail(BN_EINVAL, "nprobe must be positive");
    if (B > 65535) return fail(BN_EINVAL, "B = %u exceeds 65535 queries per call", B);
    const uint32_t nlist = v->nlist, d = v->cent_d, np = std::min(nprobe, nlist);
    if (nlist == 0) return BN_OK;
    std::lock_guard<std::mutex> g(v->e.mu);
    CU(cudaSetDevice(v->e.ctx->device));
    Layout L;
    const uint64_t o_q = L.take<float>((uint64_t)B * d);
    const uint64_t o_d = L.take<float>((uint64_t)B * nlist);
    const uint64_t o_p = L.take<uint32_t>((uint64_t)B * np);
    TRY(v->e.ws.reserve(v->e.ctx, L.off));
    char* dv = v->e.ws.at<char>();
    cudaStream_t s = v->e.stream;
    CU(cudaMemcpyAsync(dv + o_q, queries, (uint64_t)B * d * 4, cudaMemcpyHostToDevice, s));
    // Queries per thread: each centroid value loaded serves QPT queries, as long
    // as the grid still covers the chip (two warps per CTA) and the query rows fit
    // beside the ring.
    const float* dc = v->cent_t.at<float>();
    const float* dq = reinterpret_cast<const float*>(dv + o_q);
    float* dd = reinterpret_cast<float*>(dv + o_d);
    const uint32_t gx = (nlist + RT_THREADS - 1) / RT_THREADS;
    const uint32_t ring = RT_DEPTH * RT_BATCH * RT_THREADS * 4, qrow = (d + RT_BATCH - 1) / RT_BATCH * RT_BATCH * 4;
    const uint32_t qpt = (uint64_t)gx * ((B + 3) / 4) >= (uint32_t)v->e.ctx->num_sms && qrow <= 16 * 1024 ? 4 : 1;
    auto dist_fn = qpt == 4 ? route_dist_kernel<4> : route_dist_kernel<1>;
    const int dist_smem = (int)(ring + qpt * qrow);
    CU(cudaFuncSetAttribute(dist_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dist_smem));
    dist_fn<<<dim3(gx, (B + qpt - 1) / qpt), RT_THREADS, dist_smem, s>>>(dc, nlist, d, dq, B, dd);
    uint32_t pow2 = 32;
    while (pow2 < nlist) pow2 <<= 1;
    uint32_t* dp = reinterpret_cast<uint32_t*>(dv + o_p);
    if (pow2 <= RT_SORT_THREADS) {
        route_select_small_kernel<<<B, pow2, 0, s>>>(dd, nlist, np, dp);
    } else {
        CU(cudaFuncSetAttribute(route_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ROUTE_MAX_NLIST * 8));
        route_select_kernel<<<B, RT_SORT_THREADS, (int)(pow2 * 8), s>>>(dd, nlist, np, pow2, dp);
    }
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(probes, dv + o_p, (uint64_t)B * np * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    return BN_OK;
}

}  // extern "C"
