// bn_kernels.cu -- CUDA-core kernels of the BN path for sm_100a.
//
// scan_tma_kernel   r = M_enc . v (crypto.rs:561-626 / kernels.cu:100-178),
//                   4-row blocks streamed into shared memory by one bulk
//                   copy each; one work item = 4 rows x 1024 columns split
//                   over four warps (a quarter row each); per element 6
//                   IMAD.WIDE into three 64-bit limb accumulators, no carries,
//                   no per-product fold; a transposed warp reduction and one
//                   fold per row at the end.
// freivalds_kernel  Protocol 2 (crypto.rs:1013-1046): u drawn on device from
//                   the ChaCha20 keystream by index, z_t = u_t^T M_enc and
//                   u_t . r partials per row chunk.
// decode_topk       decode_scores (crypto.rs:901-940) + fp_to_signed + top-k
//                   (lib.rs:452-469) in one pass over the client arrays.
// gemm_abt          keygen-side F_p GEMMs (crypto.rs:419-467).
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "bn_kernels.cuh"

namespace bn {

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void named_bar(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__global__ void or_flag_kernel(uint32_t* w, uint32_t bits) { atomicOr(w, bits); }

// ------------------------------------------------------------------ limbs
__global__ void query_limbs_kernel(const uint64_t* __restrict__ v, uint64_t total, QLimb* __restrict__ out) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    uint64_t x = v[i];
    Limbs3 b = limbs(x), c = limbs_hi(x);
    out[i] = QLimb{b.b0, b.b1, b.b2, c.b0, c.b1, c.b2, 0u, 0u};
}

// ------------------------------------------------------------------ scan

__device__ __forceinline__ uint32_t find_seg(const uint64_t* __restrict__ seg_blk, uint32_t nseg, uint32_t hint,
                                             uint64_t blk) {
    if (blk >= seg_blk[hint] && blk < seg_blk[hint + 1]) return hint;
    uint32_t lo = 0, hi = nseg;  // find last s with seg_blk[s] <= blk
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (seg_blk[mid] <= blk) lo = mid; else hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------------ scan, TMA pipeline
// One producer warp streams each 4-row block (up to 32 KiB, contiguous in
// m_enc) into a ring of shared-memory stages with a single cp.async.bulk;
// three consumer groups of four warps take the stages round-robin.  A stage
// must always fall to the same group: a barrier wait names a phase by its parity,
// so a group that met a stage on every second round only would take the round
// before last for the one it waits for whenever the round between them, another
// group's, is late (copies finish out of order, most of all on cold pages), read
// the stage early and release it twice.  With four groups on six stages that
// happened: wrong r and launch failures at 50,001 rows.  Every
// mbarrier wait is bounded: on timeout the CTA records an error in *err
// and stops, so a lost completion cannot hang the GPU.
constexpr int TS_STAGES = 6;
constexpr int TS_GROUPS = 3;
static_assert(TS_STAGES % TS_GROUPS == 0, "a stage must always fall to the same group");
constexpr int TS_CONSUMERS = 32 * 4 * TS_GROUPS;   // 384
constexpr int TS_THREADS = TS_CONSUMERS + 32;      // + producer warp
constexpr uint32_t TS_STAGE_BYTES = SCAN_ROWS * N * 8;  // 32 KiB
constexpr long long WAIT_CYCLES = 2000000000ll;    // ~1 s at 1.9 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: true when the phase with `parity` completed within `limit`
// cycles (pipeline waits take the kernel's wait_limit argument; the drain of
// the CTA's own copies keeps the full limit).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit = WAIT_CYCLES) {
    const long long t0 = clock64();
    if (limit >= WAIT_CYCLES) {
        while (!mbar_try_wait(bar, parity))
            if (clock64() - t0 > limit) return false;
        return true;
    }
    // a shortened (test) limit polls with test_wait: try_wait may stay
    // suspended until the phase completes, which would outlast the limit
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > limit) return false;
    }
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

struct ScanBlock {
    uint64_t row0;  // first m_enc row
    uint64_t out0;  // first r slot
    int nrows;
    uint32_t query;
};
__device__ __forceinline__ ScanBlock scan_block(const ScanSeg* __restrict__ segs, const uint64_t* __restrict__ seg_blk,
                                                uint32_t nseg, uint32_t& hint, uint64_t blk) {
    hint = find_seg(seg_blk, nseg, hint, blk);
    const ScanSeg sg = segs[hint];
    const uint64_t local = (blk - seg_blk[hint]) * SCAN_ROWS;
    const uint64_t left = (uint64_t)sg.rows - local;
    return ScanBlock{sg.row0 + local, sg.out0 + local, left < (uint64_t)SCAN_ROWS ? (int)left : SCAN_ROWS, sg.query};
}

__global__ void __launch_bounds__(TS_THREADS, 1)
scan_tma_kernel(const uint64_t* __restrict__ m_enc, const QLimb* __restrict__ qlimbs, const ScanSeg* __restrict__ segs,
                const uint64_t* __restrict__ seg_blk, uint32_t nseg, uint64_t total_blocks, uint64_t* __restrict__ r,
                uint32_t* __restrict__ err, long long wait_limit) {
    extern __shared__ __align__(1024) unsigned char ts_smem[];
    uint4* stage_base = reinterpret_cast<uint4*>(ts_smem);
    __shared__ uint64_t full_bar[TS_STAGES], empty_bar[TS_STAGES];
    __shared__ unsigned long long red[2][TS_GROUPS][4][SCAN_ROWS][3];
    __shared__ volatile int abort_flag;
    __shared__ volatile int group_stop[2][TS_GROUPS];  // per-iteration snapshot, double-buffered

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TS_STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 4);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    const uint64_t nblk = total_blocks > blockIdx.x ? (total_blocks - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

    if (warp == TS_CONSUMERS / 32) {  // ---------------- producer warp
        if (lane == 0) {
            uint32_t hint = 0;
            uint64_t i = 0;
            for (; i < nblk; ++i) {
                const int s = (int)(i % TS_STAGES);
                if (i >= TS_STAGES && !mbar_wait(&empty_bar[s], (uint32_t)(((i / TS_STAGES) - 1) & 1), wait_limit)) {
                    abort_flag = 1;
                    atomicOr(err, 1u);
                    break;
                }
                if (abort_flag) break;
                const ScanBlock b = scan_block(segs, seg_blk, nseg, hint, blockIdx.x + i * gridDim.x);
                const uint32_t bytes = (uint32_t)b.nrows * N * 8;
                mbar_expect_tx(&full_bar[s], bytes);
                bulk_g2s(stage_base + (uint64_t)s * (TS_STAGE_BYTES / 16), m_enc + b.row0 * N, bytes, &full_bar[s]);
            }
            // drain: no bulk copy may still be writing shared memory at exit
            for (uint64_t j = (i > TS_STAGES ? i - TS_STAGES : 0); j < i; ++j)
                mbar_wait(&full_bar[j % TS_STAGES], (uint32_t)((j / TS_STAGES) & 1));
        }
        return;
    }

    // ---------------------------------------------------- consumer groups
    const int group = warp >> 2, wq = warp & 3;
    const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
    uint32_t b0[8], b1[8], b2[8], c0[8], c1[8], c2[8];
    uint32_t cur_q = 0xffffffffu, hint = 0;
    int parity = 0;
    for (uint64_t i = group; i < nblk; i += TS_GROUPS) {
        const int s = (int)(i % TS_STAGES);
        const ScanBlock b = scan_block(segs, seg_blk, nseg, hint, blockIdx.x + i * gridDim.x);
        if (b.query != cur_q) {
            cur_q = b.query;
            const QLimb* ql = qlimbs + (uint64_t)cur_q * N + wq * 256 + 2 * lane;
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const QLimb q = ql[64 * k + e];
                    b0[2 * k + e] = q.b0; b1[2 * k + e] = q.b1; b2[2 * k + e] = q.b2;
                    c0[2 * k + e] = q.c0; c1[2 * k + e] = q.c1; c2[2 * k + e] = q.c2;
                }
        }
        const bool ok = mbar_wait(&full_bar[s], (uint32_t)((i / TS_STAGES) & 1), wait_limit);
        if (!ok) { abort_flag = 1; atomicOr(err, 2u); }
        uint64_t acc[SCAN_ROWS][3];
        const uint4* base = stage_base + (uint64_t)s * (TS_STAGE_BYTES / 16) + wq * 128 + lane;
#pragma unroll
        for (int rr = 0; rr < SCAN_ROWS; ++rr) {
            uint64_t a0 = 0, a1 = 0, a2 = 0;
            if (ok && rr < b.nrows) {
                const uint4* rp = base + rr * (N / 2);
                uint4 x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) x[k] = rp[32 * k];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int e0 = 2 * k, e1 = 2 * k + 1;
                    a0 = mac(mac(a0, x[k].x, b0[e0]), x[k].y, c0[e0]);
                    a1 = mac(mac(a1, x[k].x, b1[e0]), x[k].y, c1[e0]);
                    a2 = mac(mac(a2, x[k].x, b2[e0]), x[k].y, c2[e0]);
                    a0 = mac(mac(a0, x[k].z, b0[e1]), x[k].w, c0[e1]);
                    a1 = mac(mac(a1, x[k].z, b1[e1]), x[k].w, c1[e1]);
                    a2 = mac(mac(a2, x[k].z, b2[e1]), x[k].w, c2[e1]);
                }
            }
            acc[rr][0] = a0; acc[rr][1] = a1; acc[rr][2] = a2;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);  // this warp is done with the stage
        uint64_t w[2][3];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                uint64_t send = hi16 ? acc[q][a] : acc[q + 2][a];
                uint64_t keep = hi16 ? acc[q + 2][a] : acc[q][a];
                w[q][a] = keep + __shfl_xor_sync(FULL, send, 16);
            }
        uint64_t xs[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            uint64_t send = hi8 ? w[0][a] : w[1][a];
            uint64_t keep = hi8 ? w[1][a] : w[0][a];
            xs[a] = keep + __shfl_xor_sync(FULL, send, 8);
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1)
#pragma unroll
            for (int a = 0; a < 3; ++a) xs[a] += __shfl_xor_sync(FULL, xs[a], off);
        if ((lane & 7) == 0) {
#pragma unroll
            for (int a = 0; a < 3; ++a) red[parity][group][wq][lane >> 3][a] = xs[a];
        }
        // Stop decision: one snapshot per group and iteration, written before
        // the barrier and read after it, so the four warps agree.
        if (wq == 0 && lane == 0) group_stop[parity][group] = abort_flag;
        named_bar(1 + group, 128);
        if (group_stop[parity][group]) break;
        if (wq == 0 && lane < b.nrows) {
            uint64_t t[3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
                t[a] = red[parity][group][0][lane][a] + red[parity][group][1][lane][a] +
                       red[parity][group][2][lane][a] + red[parity][group][3][lane][a];
            r[b.out0 + lane] = combine3(t[0], t[1], t[2]);
        }
        parity ^= 1;
    }
}

// ------------------------------------------------------------------ Freivalds
constexpr int FV_THREADS = 256;
constexpr int FV_TILE = 32;

template <int TMAX>
__global__ void __launch_bounds__(FV_THREADS)
freivalds_kernel(const uint64_t* __restrict__ m_enc, const uint64_t* __restrict__ r, const VerifySeg* __restrict__ vsegs,
                 const ChaChaKey* __restrict__ keys, uint32_t t_base, uint32_t t_cnt, uint32_t trials,
                 uint32_t chunks, uint32_t chunk_rows, uint64_t* __restrict__ z_part, uint64_t* __restrict__ ur_part,
                 uint32_t* __restrict__ flags, uint32_t seg_base) {
    const uint32_t seg = seg_base + blockIdx.z, chunk = blockIdx.y;
    const uint32_t j = blockIdx.x * FV_THREADS + threadIdx.x;
    const VerifySeg vs = vsegs[seg];
    const uint64_t row_begin = (uint64_t)chunk * chunk_rows;
    const uint64_t row_end = min((uint64_t)vs.rows, row_begin + chunk_rows);
    const ChaChaKey key = keys[vs.query];

    __shared__ uint32_t ul[FV_TILE][TMAX][6];
    __shared__ uint64_t uraw[TMAX][FV_TILE];

    uint64_t acc[TMAX][3];
#pragma unroll
    for (int t = 0; t < TMAX; ++t) acc[t][0] = acc[t][1] = acc[t][2] = 0;
    uint64_t urp = 0;
    uint32_t since_fold = 0;
    const uint32_t gen_t = threadIdx.x >> 3, gen_b = threadIdx.x & 7;

    for (uint64_t tile = row_begin; tile < row_end; tile += FV_TILE) {
        const uint32_t nt = (uint32_t)min((uint64_t)FV_TILE, row_end - tile);
        __syncthreads();
        if (gen_t < t_cnt) {
            const uint64_t first = draw_index(vs, t_base + gen_t, tile);  // draw index of row `tile`
            const uint64_t blk = first / 8 + gen_b;
            if (blk * 8 < first + nt) {
                uint32_t w[16];
                chacha20_block(key, blk, w);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const uint64_t idx = blk * 8 + q;
                    if (idx >= first && idx < first + nt) {
                        uint64_t x = ((uint64_t)w[2 * q] | ((uint64_t)w[2 * q + 1] << 32)) & P;
                        if (x == P) { atomicOr(flags, DRAW_HIT_P); x = 0; }
                        const uint32_t ii = (uint32_t)(idx - first);
                        Limbs3 b = limbs(x), c = limbs_hi(x);
                        ul[ii][gen_t][0] = b.b0; ul[ii][gen_t][1] = b.b1; ul[ii][gen_t][2] = b.b2;
                        ul[ii][gen_t][3] = c.b0; ul[ii][gen_t][4] = c.b1; ul[ii][gen_t][5] = c.b2;
                        uraw[gen_t][ii] = x;
                    }
                }
            }
        }
        __syncthreads();
        const uint64_t* mp = m_enc + (vs.row0 + tile) * N + j;
        for (uint32_t ii = 0; ii < nt; ++ii) {
            const uint64_t mv = __ldg(mp + (uint64_t)ii * N);
            const uint32_t mlo = (uint32_t)mv, mhi = (uint32_t)(mv >> 32);
#pragma unroll
            for (int t = 0; t < TMAX; ++t) {
                if (t < (int)t_cnt) {
                    const uint32_t* u = ul[ii][t];
                    acc[t][0] = mac(mac(acc[t][0], mlo, u[0]), mhi, u[3]);
                    acc[t][1] = mac(mac(acc[t][1], mlo, u[1]), mhi, u[4]);
                    acc[t][2] = mac(mac(acc[t][2], mlo, u[2]), mhi, u[5]);
                }
            }
        }
        if (blockIdx.x == 0 && threadIdx.x < t_cnt) {
            for (uint32_t ii = 0; ii < nt; ++ii)
                urp = add_mod(urp, mul_mod(uraw[threadIdx.x][ii], r[vs.r0 + tile + ii]));
        }
        since_fold += nt;
        if (since_fold >= 480) {  // 512 more rows would still fit below 2^63
#pragma unroll
            for (int t = 0; t < TMAX; ++t) { acc[t][0] = fold(acc[t][0]); acc[t][1] = fold(acc[t][1]); acc[t][2] = fold(acc[t][2]); }
            since_fold = 0;
        }
    }
    const uint64_t slot = (uint64_t)seg * chunks + chunk;
#pragma unroll
    for (int t = 0; t < TMAX; ++t)
        if (t < (int)t_cnt) z_part[(slot * trials + t_base + t) * N + j] = combine3(acc[t][0], acc[t][1], acc[t][2]);
    if (blockIdx.x == 0 && threadIdx.x < t_cnt) ur_part[slot * trials + t_base + threadIdx.x] = urp;
}

__device__ __forceinline__ uint64_t block_sum_mod(uint64_t v, uint64_t* sh) {
    // 256 threads
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = add_mod(v, __shfl_xor_sync(FULL, v, off));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    uint64_t t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = add_mod(t, sh[w]);
    return t;
}

__global__ void __launch_bounds__(256)
freivalds_finish_kernel(const uint64_t* __restrict__ z_part, const uint64_t* __restrict__ ur_part,
                        const uint64_t* __restrict__ v_enc, const VerifySeg* __restrict__ vsegs, uint32_t trials,
                        uint32_t chunks, uint64_t* __restrict__ ur, uint64_t* __restrict__ zv,
                        int32_t* __restrict__ failed) {
    const uint32_t seg = blockIdx.x;
    const VerifySeg vs = vsegs[seg];
    const uint64_t* v = v_enc + (uint64_t)vs.query * N;
    __shared__ uint64_t sh[32];
    int32_t fail = -1;
    for (uint32_t t = 0; t < trials; ++t) {
        uint64_t part = 0;
        for (uint32_t j = threadIdx.x; j < N; j += blockDim.x) {
            uint64_t z = 0;
            for (uint32_t c = 0; c < chunks; ++c) z = add_mod(z, z_part[(((uint64_t)seg * chunks + c) * trials + t) * N + j]);
            part = add_mod(part, mul_mod(z, v[j]));
        }
        const uint64_t zvt = block_sum_mod(part, sh);
        if (threadIdx.x == 0) {
            uint64_t urt = 0;
            for (uint32_t c = 0; c < chunks; ++c) urt = add_mod(urt, ur_part[((uint64_t)seg * chunks + c) * trials + t]);
            ur[(uint64_t)seg * trials + t] = urt;
            zv[(uint64_t)seg * trials + t] = zvt;
            if (fail < 0 && urt != zvt) fail = (int32_t)t;
        }
    }
    if (threadIdx.x == 0) failed[seg] = fail;
}

// ------------------------------------------------------------------ L^T v
// A CTA takes 8 columns of L (64 of its bytes per row, whole sectors) for a
// run of queries: thread (slice, column) holds its 32 elements of L, rows
// slice, slice + 32, ..., in registers, all loads in flight at once, and every
// query costs the limbs of its v in shared memory and six multiply-adds per
// element.  Latency bound for one query (16 CTAs at n1 = 128, one round of
// loads: 13 -> 4 us against a cluster of 8 CTAs with a distributed-shared-
// memory sum); for many, L is read once per run of queries instead of once per
// query (512 queries: 168 us before).  A thread adds 32 terms below 2^53.2, so
// the accumulators stay below 2^64.
constexpr uint32_t LT_THREADS = 256, LT_COLS = 8, LT_ROWS = N / (LT_THREADS / LT_COLS);

struct LtShared {
    uint4 lo[N];  // {b0, b1, b2, c0} of v_j
    uint2 hi[N];  // {c1, c2}
    uint64_t red[LT_THREADS / 32][LT_COLS];
};

__device__ __forceinline__ void lt_block(LtShared& sh, const uint64_t* __restrict__ L, uint32_t n1,
                                         const uint64_t* __restrict__ v, uint32_t k0, uint32_t q0, uint32_t q1,
                                         uint64_t* __restrict__ x) {
    const uint32_t kk = threadIdx.x % LT_COLS, sl = threadIdx.x / LT_COLS;
    constexpr uint32_t SLICES = LT_THREADS / LT_COLS;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t l[LT_ROWS];
#pragma unroll
    for (uint32_t i = 0; i < LT_ROWS; ++i) l[i] = __ldg(L + (uint64_t)(sl + i * SLICES) * n1 + k0 + kk);
    for (uint32_t q = q0; q < q1; ++q) {
        for (uint32_t j = threadIdx.x; j < N; j += LT_THREADS) {
            const uint64_t w = v[(uint64_t)q * N + j];
            const Limbs3 b = limbs(w), c = limbs_hi(w);
            sh.lo[j] = make_uint4(b.b0, b.b1, b.b2, c.b0);
            sh.hi[j] = make_uint2(c.b1, c.b2);
        }
        __syncthreads();
        uint64_t a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
        for (uint32_t i = 0; i < LT_ROWS; ++i) {
            const uint4 l0 = sh.lo[sl + i * SLICES];
            const uint2 l1 = sh.hi[sl + i * SLICES];
            const uint32_t xl = (uint32_t)l[i], xh = (uint32_t)(l[i] >> 32);
            a0 = mac(mac(a0, xl, l0.x), xh, l0.w);
            a1 = mac(mac(a1, xl, l0.y), xh, l1.x);
            a2 = mac(mac(a2, xl, l0.z), xh, l1.y);
        }
        uint64_t t = combine3(a0, a1, a2);
        t = add_mod(t, __shfl_xor_sync(FULL, t, 8));
        t = add_mod(t, __shfl_xor_sync(FULL, t, 16));
        if (lane < LT_COLS) sh.red[warp][lane] = t;
        __syncthreads();  // also: the limbs are no longer read
        if (threadIdx.x < LT_COLS) {
            uint64_t s = 0;
#pragma unroll
            for (uint32_t w = 0; w < LT_THREADS / 32; ++w) s = add_mod(s, sh.red[w][threadIdx.x]);
            x[(uint64_t)q * n1 + k0 + threadIdx.x] = s;
        }
    }
}

// Queries per CTA: as many as leave two CTAs per SM, at most 16.
uint32_t lt_run(uint32_t n1, uint32_t nq) {
    const uint32_t run = (uint32_t)((uint64_t)nq * (n1 / LT_COLS) / (2 * 148));
    return run < 1 ? 1 : run > 16 ? 16 : run;
}

__global__ void __launch_bounds__(LT_THREADS)
lt_times_v_kernel(const uint64_t* __restrict__ L, uint32_t n1, const uint64_t* __restrict__ v, uint32_t nq,
                  uint32_t run, uint64_t* __restrict__ x) {
    __shared__ LtShared sh;
    const uint32_t q0 = blockIdx.y * run;
    lt_block(sh, L, n1, v, blockIdx.x * LT_COLS, q0, min(nq, q0 + run), x);
}

// Everything a query pipeline needs from v before its first pass, in one
// launch: CTAs [0, lt_ctas) take L^T v (lt_cols column groups per run of
// queries), the next wimg_ctas the diagonal byte images of the fused scan,
//   w[((q * 64 + strip) * 16 + s) * 128 + 8 j + a] = byte (s - a) of
//   v[q][strip * 16 + j] when 0 <= s - a <= 7, else 0,
// and the last one clears the run's status words and tickets.
__global__ void __launch_bounds__(LT_THREADS)
query_prep_kernel(const uint64_t* __restrict__ L, uint32_t n1, const uint64_t* __restrict__ v, uint32_t nq,
                  uint32_t run, uint32_t lt_ctas, uint64_t* __restrict__ x, uint32_t wimg_ctas, uint8_t* __restrict__ w,
                  uint32_t* __restrict__ zero, uint32_t zero_words) {
    __shared__ LtShared sh;
    after_go();
    if (blockIdx.x < lt_ctas) {
        const uint32_t cols = n1 / LT_COLS, q0 = blockIdx.x / cols * run;
        lt_block(sh, L, n1, v, blockIdx.x % cols * LT_COLS, q0, min(nq, q0 + run), x);
    } else if (blockIdx.x < lt_ctas + wimg_ctas) {
        const uint64_t e = (uint64_t)(blockIdx.x - lt_ctas) * LT_THREADS + threadIdx.x;  // (query, strip, s, j)
        const uint32_t j = (uint32_t)(e & 15), s = (uint32_t)((e >> 4) & 15);
        const uint64_t qs = e >> 8;  // q * 64 + strip
        const uint64_t y = v[(qs >> 6) * N + (qs & 63) * 16 + j];
        uint64_t word = 0;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int b = (int)s - a;
            if (b >= 0 && b <= 7) word |= ((y >> (8 * b)) & 0xffull) << (8 * a);
        }
        *reinterpret_cast<uint64_t*>(w + (qs * 16 + s) * 128 + 8 * j) = word;
    } else {
        for (uint32_t i = threadIdx.x; i < zero_words; i += LT_THREADS) zero[i] = 0;
    }
}

// ------------------------------------------------------------------ decode
// AL g + H x alone, from the column-major arrays.  A CTA takes 32 rows at a time, a
// warp an eighth of the 2 n1 columns with 16 loads in flight; the warps' shares meet
// in shared memory and a warp in turn adds them up.  Bound by HBM (2 n1 x 8 bytes per
// row): a thread per row over all columns had 8 loads in flight and, with few rows,
// few CTAs (150,001 rows, n1 = 128, 307 MB: 84 us; now 61 us, 5.0 TB/s).
constexpr uint32_t DN_WARPS = 8;

__global__ void __launch_bounds__(32 * DN_WARPS, 4)
dense_terms_kernel(const uint64_t* __restrict__ al_cm, const uint64_t* __restrict__ h_cm, uint64_t rows, uint32_t n1,
                   const uint64_t* __restrict__ g, const uint64_t* __restrict__ x, uint64_t* __restrict__ out) {
    __shared__ uint4 lim[2 * 2 * 512];  // {b0,b1,b2,c0}, {c1,c2,-,-} per column of g, then of x
    __shared__ uint64_t sh[2][DN_WARPS][32];
    for (uint32_t k = threadIdx.x; k < 2 * n1; k += blockDim.x) {
        const uint64_t w = k < n1 ? g[k] : x[k - n1];
        const Limbs3 b = limbs(w), c = limbs_hi(w);
        lim[2 * k] = make_uint4(b.b0, b.b1, b.b2, c.b0);
        lim[2 * k + 1] = make_uint4(c.b1, c.b2, 0u, 0u);
    }
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cols = 2 * n1 / DN_WARPS, c0 = warp * cols;  // a multiple of 16 (n1 >= 64), all of AL or all of H
    const uint64_t* base = c0 < n1 ? al_cm + (uint64_t)c0 * rows : h_cm + (uint64_t)(c0 - n1) * rows;
    uint32_t it = 0;
    for (uint64_t i0 = (uint64_t)blockIdx.x * 32; i0 < rows; i0 += (uint64_t)gridDim.x * 32, ++it) {
        const uint64_t i = i0 + lane;
        const uint64_t* p = base + (i < rows ? i : rows - 1);
        uint64_t a0 = 0, a1 = 0, a2 = 0;  // at most 128 columns of 2^53 + 2^50 each
        for (uint32_t k0 = 0; k0 < cols; k0 += 16) {
            uint64_t xs[16];
#pragma unroll
            for (int kk = 0; kk < 16; ++kk) xs[kk] = __ldg(p + (uint64_t)(k0 + kk) * rows);
#pragma unroll
            for (int kk = 0; kk < 16; ++kk) {
                const uint32_t lo = (uint32_t)xs[kk], hi = (uint32_t)(xs[kk] >> 32);
                const uint4 l0 = lim[2 * (c0 + k0 + kk)], l1 = lim[2 * (c0 + k0 + kk) + 1];
                a0 = mac(mac(a0, lo, l0.x), hi, l0.w);
                a1 = mac(mac(a1, lo, l0.y), hi, l1.x);
                a2 = mac(mac(a2, lo, l0.z), hi, l1.y);
            }
        }
        auto& part = sh[it & 1];
        part[warp][lane] = combine3(a0, a1, a2);
        __syncthreads();  // one per block of rows: the other buffer is rewritten only after the next one
        if (it % DN_WARPS == warp && i < rows) {
            uint64_t sum = part[0][lane];
#pragma unroll
            for (uint32_t w = 1; w < DN_WARPS; ++w) sum = add_mod(sum, part[w][lane]);
            out[i] = sum;
        }
    }
}

// Decode copies of the client state in 32-row blocks (layouts in
// bn_kernels.cuh); reads and writes are both coalesced along the rows.
__global__ void decode_layout_kernel(const uint64_t* __restrict__ al_cm, const uint64_t* __restrict__ h_cm,
                                     const uint64_t* __restrict__ mp_cm, uint64_t rows, uint32_t n1,
                                     uint64_t* __restrict__ alh_b, int8_t* __restrict__ m8_cm, uint32_t* __restrict__ bad) {
    const uint64_t rows32 = (rows + 31) / 32 * 32;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n_alh = rows32 * 2 * n1;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n_alh; e += stride) {
        const uint64_t col = (e >> 5) % (2 * n1), gr = ((e >> 5) / (2 * n1)) * 32 + (e & 31);
        uint64_t x = 0;
        if (gr < rows) x = col < n1 ? al_cm[col * rows + gr] : h_cm[(col - n1) * rows + gr];
        alh_b[e] = x;
    }
    if (!m8_cm) return;
    bool out_of_range = false;
    const uint64_t n_m = rows32 * N;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n_m; e += stride) {
        const uint64_t col = e / rows32, gr = e - col * rows32;
        int64_t v = 0;
        if (gr < rows) v = to_signed(mp_cm[col * rows + gr]);
        out_of_range |= v < -128 || v > 127;
        m8_cm[e] = (int8_t)v;
    }
    if (out_of_range) atomicOr(bad, 1u);
}

constexpr int DT_THREADS = 256;
constexpr int CAND_CAP = 2048;

__device__ __forceinline__ bool better(int64_t s1, uint32_t i1, int64_t s2, uint32_t i2) {
    return s1 > s2 || (s1 == s2 && i1 < i2);
}

// In-place bitonic sort of n (power of two) entries, best first.
__device__ void bitonic_best_first(int64_t* s, uint32_t* id, int n) {
    for (int size = 2; size <= n; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < n / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const bool up = (lo & size) == 0;
                const bool sw = up ? better(s[hi], id[hi], s[lo], id[lo]) : better(s[lo], id[lo], s[hi], id[hi]);
                if (sw) {
                    int64_t ts = s[lo]; s[lo] = s[hi]; s[hi] = ts;
                    uint32_t ti = id[lo]; id[lo] = id[hi]; id[hi] = ti;
                }
            }
        }
    __syncthreads();
}

// Candidate buffer of one CTA: entries better than the current k-th best
// are appended; when the buffer nears capacity it is sorted and cut to k.
struct TopkBuf {
    int64_t s[CAND_CAP];
    uint32_t id[CAND_CAP];
    int cnt;
    int64_t thr_s;
    uint32_t thr_i;
    int have_thr;
};

// Compaction decision, uniform across the CTA: every thread reads the count
// between two barriers, so no thread can append (next iteration) before all
// have read it; then either all threads compact or none does (topk_compact
// holds __syncthreads).
__device__ __forceinline__ bool topk_full(TopkBuf& b, int limit) {
    __syncthreads();
    const bool full = b.cnt > limit;
    __syncthreads();
    return full;
}

__device__ void topk_compact(TopkBuf& b, int k) {
    __syncthreads();
    const int cnt = b.cnt;
    int n = 1;
    while (n < cnt) n <<= 1;
    for (int i = cnt + threadIdx.x; i < n; i += blockDim.x) { b.s[i] = INT64_MIN; b.id[i] = 0xffffffffu; }
    bitonic_best_first(b.s, b.id, n);
    if (threadIdx.x == 0) {
        if (cnt >= k) {
            b.cnt = k;
            b.thr_s = b.s[k - 1];
            b.thr_i = b.id[k - 1];
            b.have_thr = 1;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void topk_offer(TopkBuf& b, bool valid, int64_t s, uint32_t id, int64_t thr_s, uint32_t thr_i,
                                           int have_thr) {
    if (valid && (!have_thr || better(s, id, thr_s, thr_i))) {
        const int pos = atomicAdd(&b.cnt, 1);
        b.s[pos] = s;
        b.id[pos] = id;
    }
}

// Sum of +-x (sign in bit 31 of the entry) over a gathered column list,
// folded lazily: every term is < 2^61, three terms fit below 2^63.
__device__ __forceinline__ uint64_t signed_term(uint64_t x, bool neg) { return neg ? P - x : x; }

// AL_i . g + H_i . x for corpus row gr from the 32-row-blocked alh_b: the 2 n1 columns
// of the row's block are contiguous, so a warp's batch of 32 column loads is one 8 KB
// run.  lim[2k], lim[2k + 1] hold the limbs of g_k (k < n1) and of x_(k-n1) (k >= n1).
// Every column adds lo*b + hi*c < 2^53 + 2^50 (hi < 2^29: residues are < 2^61) to an
// accumulator, so the 2 n1 <= 1024 columns stay below 2^64 with no fold.  (In the form
// of dense_terms_block the whole-unit decode of 64 queries over 50,000 rows took 1936 us
// against 1815, one query over 100,000 rows 338 for the call against 328.)
__device__ __forceinline__ uint64_t dense_terms_row(const uint64_t* __restrict__ alh_b, uint32_t n1, uint64_t gr,
                                                    const uint4* __restrict__ lim) {
    const uint64_t* p = alh_b + (gr >> 5) * (2ull * n1) * 32 + (gr & 31);
    uint64_t a0 = 0, a1 = 0, a2 = 0;
    for (uint32_t k0 = 0; k0 < 2 * n1; k0 += 32) {  // 2 n1 is a multiple of 32 (n1 >= 64)
        uint64_t xs[32];
#pragma unroll
        for (int kk = 0; kk < 32; ++kk) xs[kk] = __ldg(p + (uint64_t)(k0 + kk) * 32);
#pragma unroll
        for (int kk = 0; kk < 32; ++kk) {
            const uint4 l0 = lim[2 * (k0 + kk)], l1 = lim[2 * (k0 + kk) + 1];  // {b0,b1,b2,c0}, {c1,c2,-,-}
            const uint32_t xl = (uint32_t)xs[kk], xh = (uint32_t)(xs[kk] >> 32);
            a0 = mac(mac(a0, xl, l0.x), xh, l0.w);
            a1 = mac(mac(a1, xl, l0.y), xh, l1.x);
            a2 = mac(mac(a2, xl, l0.z), xh, l1.y);
        }
    }
    return combine3(a0, a1, a2);
}

// The same for the columns [k_begin, k_end) (multiples of 32) of the 32 rows of block
// blk, row l's share to lane l: the split decode, where a warp has a quarter of the
// columns and no other unit's loads to hide behind.  A 16-byte load takes two rows of
// two columns per warp (lanes 0-15 rows 2l, 2l + 1 of column k, lanes 16-31 of column
// k + 1), so a column's limbs are read from shared memory half as often.
__device__ __forceinline__ uint64_t dense_terms_block(const uint64_t* __restrict__ alh_b, uint32_t n1, uint64_t blk,
                                                      const uint4* __restrict__ lim, uint32_t k_begin, uint32_t k_end,
                                                      uint32_t lane) {
    const uint32_t half = lane >> 4;
    const ulonglong2* p =
        reinterpret_cast<const ulonglong2*>(alh_b + blk * (2ull * n1) * 32 + (uint64_t)half * 32 + 2 * (lane & 15));
    uint64_t a[2][3] = {};  // rows 2 (l & 15), + 1
    for (uint32_t k0 = k_begin; k0 < k_end; k0 += 32) {
        ulonglong2 xs[16];
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) xs[kk] = __ldg(p + (uint64_t)(k0 + 2 * kk) * 16);
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const uint32_t col = k0 + 2 * kk + half;
            const uint4 l0 = lim[2 * col], l1 = lim[2 * col + 1];  // {b0,b1,b2,c0}, {c1,c2,-,-}
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint64_t x = e ? xs[kk].y : xs[kk].x;
                const uint32_t xl = (uint32_t)x, xh = (uint32_t)(x >> 32);
                a[e][0] = mac(mac(a[e][0], xl, l0.x), xh, l0.w);
                a[e][1] = mac(mac(a[e][1], xl, l0.y), xh, l1.x);
                a[e][2] = mac(mac(a[e][2], xl, l0.z), xh, l1.y);
            }
        }
    }
    // lanes l and l ^ 16 hold the even and the odd columns of the same two rows:
    // the lower one takes the first row's halves, the upper one the second's
    uint64_t t[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        t[i] = (half ? a[1][i] : a[0][i]) + __shfl_xor_sync(FULL, half ? a[0][i] : a[1][i], 16);
    return __shfl_sync(FULL, combine3(t[0], t[1], t[2]), (lane >> 1) | ((lane & 1) << 4));
}

// Two zero-extended 16-bit halves from bytes 0, 1 (sel 0x4140) or 2, 3
// (sel 0x4342) of x (selector nibble 4 picks a zero byte).
__device__ __forceinline__ uint32_t zext_pair(uint32_t x, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(x), "r"(sel));
    return d;
}

// M . T for the warp's 32-row block (lane l = row 32 blk + l): the T
// columns go 32 at a time, one per lane; a lane loads its column's 32 row
// bytes (one 32-byte run of the column-major int8 copy: the warps decoding
// neighbouring blocks at the same time read neighbouring runs of the same
// columns, so DRAM pages serve many of them).  Each byte m becomes the
// unsigned m + 128 (xor 0x80) for a +1 entry or 127 - m (xor 0x7f) for a -1
// entry, widened to 16-bit halves; a reduce-scatter over the lanes (lane bit
// 4 keeps rows 0-15 or 16-31, then bits 3..0) with plain 32-bit adds (32
// terms <= 255 stay below 2^16, so no carry crosses a half) leaves lane l
// the biased sum of row l over those 32 columns.  The bias, 128 per +1
// entry and 127 per -1 entry, is taken off at the end.  Four groups of
// loads are in flight at a time.  Returns the exact integer.
__device__ __forceinline__ int32_t m_times_t_warp(const int8_t* __restrict__ m8_cm, uint64_t rows32, uint64_t blk,
                                                  const uint32_t* __restrict__ tl, uint32_t tn, uint32_t lane) {
    const int8_t* base = m8_cm + blk * 32;  // column c's run: base + c * rows32, 32-byte aligned
    int32_t acc = 0, bias = 0;
    for (uint32_t g0 = 0; g0 < tn; g0 += 4 * 32) {
        uint4 lo[4], hi[4];
        uint32_t mask[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t c = g0 + u * 32 + lane;
            lo[u] = hi[u] = make_uint4(0u, 0u, 0u, 0u);
            mask[u] = 0;  // past tn: zero bytes, no bias
            if (c < tn) {
                const uint32_t e = tl[c];
                const uint4* run = reinterpret_cast<const uint4*>(base + (uint64_t)(e & 0x3ffu) * rows32);
                lo[u] = __ldg(run);
                hi[u] = __ldg(run + 1);
                mask[u] = (e >> 31) ? 0x7f7f7f7fu : 0x80808080u;
            }
            const uint32_t pos = __ballot_sync(FULL, mask[u] == 0x80808080u), neg = __ballot_sync(FULL, mask[u] == 0x7f7f7f7fu);
            bias += 128 * __popc(pos) + 127 * __popc(neg);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (g0 + u * 32 >= tn) break;  // warp-uniform
            const uint32_t wds[8] = {lo[u].x ^ mask[u], lo[u].y ^ mask[u], lo[u].z ^ mask[u], lo[u].w ^ mask[u],
                                     hi[u].x ^ mask[u], hi[u].y ^ mask[u], hi[u].z ^ mask[u], hi[u].w ^ mask[u]};
            uint32_t v[16];  // v[w]: rows 2w (low half), 2w + 1 (high half)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[2 * i] = zext_pair(wds[i], 0x4140u);
                v[2 * i + 1] = zext_pair(wds[i], 0x4342u);
            }
            // reduce-scatter: after the step over lane bit b the lane keeps
            // the half of its words that its bit b selects
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const bool up = lane & 16;
                const uint32_t send = up ? v[w] : v[w + 8], keep = up ? v[w + 8] : v[w];
                v[w] = keep + __shfl_xor_sync(FULL, send, 16);
            }
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const bool up = lane & 8;
                const uint32_t send = up ? v[w] : v[w + 4], keep = up ? v[w + 4] : v[w];
                v[w] = keep + __shfl_xor_sync(FULL, send, 8);
            }
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const bool up = lane & 4;
                const uint32_t send = up ? v[w] : v[w + 2], keep = up ? v[w + 2] : v[w];
                v[w] = keep + __shfl_xor_sync(FULL, send, 4);
            }
            {
                const bool up = lane & 2;
                const uint32_t send = up ? v[0] : v[1], keep = up ? v[1] : v[0];
                v[0] = keep + __shfl_xor_sync(FULL, send, 2);
            }
            const uint32_t pair = v[0] + __shfl_xor_sync(FULL, v[0], 1);
            acc += (int32_t)((lane & 1) ? (pair >> 16) : (pair & 0xffffu));
        }
    }
    return acc - bias;
}

// The T entries [c, c_end) of M_i . T from the column-major residues
// (plaintext not int8-valued): one row per lane, gathers lazily folded.
__device__ __forceinline__ uint64_t m_times_t_cm(const uint64_t* __restrict__ mp_cm, uint64_t rows, uint64_t gr,
                                                 const uint32_t* __restrict__ tl, uint32_t c, uint32_t c_end) {
    uint64_t m_t = 0;
    for (; c + 16 <= c_end; c += 16) {  // 16 gathers in flight, folded two terms at a time
        uint64_t x[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) x[q] = __ldg(mp_cm + (uint64_t)(tl[c + q] & 0x3ffu) * rows + gr);
#pragma unroll
        for (int q = 0; q < 16; q += 2)
            m_t = fold(m_t) + signed_term(x[q], tl[c + q] >> 31) + signed_term(x[q + 1], tl[c + q + 1] >> 31);
    }
    for (; c < c_end; ++c) {
        const uint32_t e = tl[c];
        m_t = fold(m_t) + signed_term(__ldg(mp_cm + (uint64_t)(e & 0x3ffu) * rows + gr), e >> 31);
    }
    return canon(m_t);
}

// S . v_enc for the warp's 32-row block, which is exactly one sliced-ELL
// slice ([width][32 rows] u16).  The slice is read as 16-byte chunks, chunk
// j = lane + 32 i holding entries of column slot j / 4 for rows 8 (j % 4) ..
// + 7, so a lane always sees the same 8 rows (8 (lane % 4) + 0..7) and
// keeps 8 partial sums; a reduce-scatter over lane bits 4, 3, 2 then leaves
// one row's sum per lane, and a shuffle hands row l to lane l.  Every entry
// is an index into vt = [v_enc, 0, p - v_enc] (ELL_NEG, ELL_PAD), so a term
// is one shared load and one add; the sums fold every 4 terms (4 terms
// below 2^61 on top of a folded value stay below 2^64).  Of PARTS warps that
// share a slice, warp `part` takes every PARTS-th run of 32 chunks.
template <uint32_t PARTS>
__device__ __forceinline__ uint64_t s_times_v_part(const DecodeCorpus& dc, uint64_t blk, const uint64_t* __restrict__ vt,
                                                   uint32_t part, uint32_t lane) {
    const uint32_t off = dc.s_off[blk], wdt = dc.s_w[blk];
    const uint4* base = reinterpret_cast<const uint4*>(dc.s_ell + off);  // slice data is 64 * wdt bytes
    const uint32_t chunks = wdt * 4;
    constexpr uint32_t PAD2 = ELL_PAD | (ELL_PAD << 16);
    uint64_t acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t j0 = 0; j0 < chunks; j0 += 8 * PARTS * 32) {
        uint4 ch[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t j = j0 + (u * PARTS + part) * 32 + lane;
            ch[u] = j < chunks ? __ldg(base + j) : make_uint4(PAD2, PAD2, PAD2, PAD2);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t w[4] = {ch[u].x, ch[u].y, ch[u].z, ch[u].w};
#pragma unroll
            for (int h = 0; h < 8; ++h)  // clamped into the table (ELL_TABLE - 1 holds 0)
                acc[h] += vt[min((h & 1) ? (w[h >> 1] >> 16) : (w[h >> 1] & 0xffffu), ELL_TABLE - 1)];
            if ((u & 3) == 3) {
#pragma unroll
                for (int h = 0; h < 8; ++h) acc[h] = fold(acc[h]);
            }
        }
    }
    // each step adds two values below 2^61 + 8 and folds the sum
#pragma unroll
    for (int h = 0; h < 4; ++h) {  // lane bit 4: keep rows h + 4 * bit
        const bool up = lane & 16;
        const uint64_t send = up ? acc[h] : acc[h + 4], keep = up ? acc[h + 4] : acc[h];
        acc[h] = fold(keep + __shfl_xor_sync(FULL, send, 16));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // lane bit 3
        const bool up = lane & 8;
        const uint64_t send = up ? acc[h] : acc[h + 2], keep = up ? acc[h + 2] : acc[h];
        acc[h] = fold(keep + __shfl_xor_sync(FULL, send, 8));
    }
    {  // lane bit 2
        const bool up = lane & 4;
        const uint64_t send = up ? acc[0] : acc[1], keep = up ? acc[1] : acc[0];
        acc[0] = fold(keep + __shfl_xor_sync(FULL, send, 4));
    }
    // lane l now holds row 8 (l & 3) + 4 b4 + 2 b3 + b2 (b = bits of l); lane
    // r fetches its row from the lane that holds it
    const uint32_t src = (lane >> 3) | ((lane & 1) << 2) | (((lane >> 1) & 1) << 3) | (((lane >> 2) & 1) << 4);
    return canon(__shfl_sync(FULL, acc[0], src));
}

// A warp's running top-k (k <= 32) as a list sorted best first across the
// lanes: lane i holds the i-th best (score, id), lanes >= k the empty entry
// (INT64_MIN never occurs as a score: fp_to_signed lies in (-p/2, p/2)).
// Every lane offers one candidate; those better than the k-th best are
// inserted one at a time, each at the rank the ballot of the list entries
// better than it gives, the entries below it moving down one lane.  No
// shared memory and no block barrier.
__device__ __forceinline__ void warp_topk_offer(int64_t& ls, uint32_t& li, int k, bool valid, int64_t s, uint32_t id,
                                                uint32_t lane) {
    const int64_t ts = __shfl_sync(FULL, ls, k - 1);
    const uint32_t ti = __shfl_sync(FULL, li, k - 1);
    uint32_t m = __ballot_sync(FULL, valid && better(s, id, ts, ti));
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const int64_t cs = __shfl_sync(FULL, s, src);
        const uint32_t ci = __shfl_sync(FULL, id, src);
        const int pos = __popc(__ballot_sync(FULL, (int)lane < k && better(ls, li, cs, ci)));
        const int64_t up_s = __shfl_up_sync(FULL, ls, 1);
        const uint32_t up_i = __shfl_up_sync(FULL, li, 1);
        if (pos < k) {  // warp-uniform
            if ((int)lane > pos) { ls = up_s; li = up_i; }
            if ((int)lane == pos) { ls = cs; li = ci; }
            if ((int)lane >= k) { ls = INT64_MIN; li = 0xffffffffu; }
        }
    }
}

// Merges another sorted list (os, oi; same form) into this one: the better of
// entry i and the other's entry 31 - i are the best 32 of both as a bitonic
// sequence, which five exchanges sort; lanes >= k are emptied again.
__device__ __forceinline__ void warp_topk_merge(int64_t& ls, uint32_t& li, int k, int64_t os, uint32_t oi, uint32_t lane) {
    const int64_t rs = __shfl_sync(FULL, os, 31 - lane);
    const uint32_t ri = __shfl_sync(FULL, oi, 31 - lane);
    if (better(rs, ri, ls, li)) { ls = rs; li = ri; }
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
        const int64_t ps = __shfl_xor_sync(FULL, ls, stride);
        const uint32_t pi = __shfl_xor_sync(FULL, li, stride);
        if (better(ps, pi, ls, li) == ((lane & stride) == 0)) { ls = ps; li = pi; }
    }
    if ((int)lane >= k) { ls = INT64_MIN; li = 0xffffffffu; }
}

// Merges the warps' lists into warp 0 by halves through `xs`, `xi` (32 *
// warps entries).  Returns in warp 0's lanes.
__device__ __forceinline__ void warp_topk_reduce(int64_t& ls, uint32_t& li, int k, int64_t* xs, uint32_t* xi,
                                                 uint32_t warp, uint32_t lane) {
    for (uint32_t half = DT_THREADS / 64; half > 0; half >>= 1) {
        if (warp >= half && warp < 2 * half) {
            xs[warp * 32 + lane] = ls;
            xi[warp * 32 + lane] = li;
        }
        __syncthreads();
        if (warp < half) {
            const uint32_t o = (warp + half) * 32 + lane;
            warp_topk_merge(ls, li, k, xs[o], xi[o], lane);
        }
    }
    __syncthreads();
}

// A warp decodes one unit: a segment's rows inside one aligned 32-row block
// of the corpus (lane l = row 32 blk + l; lanes outside the segment idle in
// the row work but join the block-wide M T and S v).  A CTA takes tiles of
// 8 units of its query in turn (the host gives each query CTAs in
// proportion to its units).  Mv = r - (AL g + H x) - M T - S v, ranked by
// fp_to_signed into the CTA's candidate buffer (WARP_LISTS: k <= 32, every
// warp's own list, merged at the end with no barrier in the loop); the CTA's
// best k go to the scratch lists, and the last CTA of the query to finish (a
// ticket taken after a device-scope fence, no waiting) merges them.
//
// SPLIT (decode_split): the CTA's eight warps share one unit at a time, four a
// quarter of the dense columns each, two S v and two M T, and one of them, the next
// for the next unit, adds the shares up and ranks them: a corpus of 5,000 rows is 157
// units, which whole-unit warps put on 20 CTAs (50 us) and this on 157 (37 us).
constexpr uint32_t DT_WARPS = DT_THREADS / 32;
constexpr uint32_t DT_DENSE = 4, DT_S = 2, DT_T = 2;  // SPLIT: warps per part (2 n1 / 4 is a multiple of 32)

template <bool WARP_LISTS, bool SPLIT>
__global__ void __launch_bounds__(DT_THREADS, DECODE_CTAS_PER_SM)
decode_topk_kernel(const uint64_t* __restrict__ r, DecodeCorpus dc, const ScanSeg* __restrict__ segs,
                   const uint64_t* __restrict__ seg_unit, const DecodeQuery* __restrict__ queries,
                   const uint64_t* __restrict__ vv, const uint64_t* __restrict__ gg, const uint64_t* __restrict__ xx,
                   const uint32_t* __restrict__ t_ent, const uint32_t* __restrict__ t_nnz, uint32_t k, TopkScratch ts,
                   uint64_t* __restrict__ mv_out, uint32_t* __restrict__ out_ids, int64_t* __restrict__ out_scores,
                   uint32_t* __restrict__ out_n, uint32_t nq) {
    uint32_t lo = 0, hi = nq;  // the query owning this CTA: last one with cta0 <= blockIdx.x
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (queries[mid].cta0 <= blockIdx.x) lo = mid; else hi = mid;
    }
    const uint32_t q = lo;
    const DecodeQuery dq = queries[q];
    const uint32_t cta = blockIdx.x - dq.cta0;
    const uint32_t n1 = dc.n1;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // 2 x uint4 per column: g's n1 columns, then x's; SPLIT: after them the warps'
    // shares of a unit's 32 rows, units in turn
    extern __shared__ uint4 dyn_limbs[];
    __shared__ uint64_t vt[ELL_TABLE];  // [v_enc, 0, p - v_enc, 0]: the S . v table
    __shared__ uint32_t tl[N];
    struct WarpXchg {  // the warps' lists on their way to warp 0
        int64_t s[DT_THREADS];
        uint32_t id[DT_THREADS];
    };
    __shared__ typename std::conditional<WARP_LISTS, WarpXchg, TopkBuf>::type buf;
    __shared__ int last_s;
    const uint32_t tn = min(t_nnz[q], (uint32_t)N);
    // the query's inputs, then x and r, which earlier kernels of this run compute
    auto put_limbs = [&](uint32_t kk, uint64_t w) {
        const Limbs3 b = limbs(w), c = limbs_hi(w);
        dyn_limbs[2 * kk] = make_uint4(b.b0, b.b1, b.b2, c.b0);
        dyn_limbs[2 * kk + 1] = make_uint4(c.b1, c.b2, 0u, 0u);
    };
    for (uint32_t kk = threadIdx.x; kk < n1; kk += blockDim.x) put_limbs(kk, gg[(uint64_t)q * n1 + kk]);
    for (uint32_t j = threadIdx.x; j < N; j += blockDim.x) {
        const uint64_t x = vv[(uint64_t)q * N + j];
        vt[j] = x;
        vt[ELL_NEG + j] = x ? P - x : 0;
    }
    if (threadIdx.x == 0) vt[ELL_PAD] = vt[ELL_TABLE - 1] = 0;
    for (uint32_t c = threadIdx.x; c < tn; c += blockDim.x) tl[c] = t_ent[(uint64_t)q * N + c];
    after_wait();
    for (uint32_t kk = threadIdx.x; kk < n1; kk += blockDim.x) put_limbs(n1 + kk, __ldcg(xx + (uint64_t)q * n1 + kk));
    if constexpr (!WARP_LISTS)
        if (threadIdx.x == 0) { buf.cnt = 0; buf.have_thr = 0; buf.thr_s = INT64_MIN; buf.thr_i = 0xffffffffu; }
    __syncthreads();
    int64_t ls = INT64_MIN;  // WARP_LISTS: this warp's list (lane i: i-th best)
    uint32_t li = 0xffffffffu;

    uint64_t u_begin = 0, u_count = 0;  // nseg == 0: every probed list of this query was empty
    if (dq.nseg) {
        u_begin = seg_unit[dq.seg0];
        u_count = seg_unit[dq.seg0 + dq.nseg] - u_begin;
    }
    if constexpr (SPLIT) {
        // The candidate buffer needs no check: it takes all rows of a query that
        // decode_split sends here with it.
        static_assert(WARP_LISTS || DECODE_SPLIT_UNITS * 32 <= CAND_CAP, "candidate buffer smaller than a query's rows");
        uint32_t it = 0;
        for (uint64_t u = cta; u < u_count; u += dq.ctas, ++it) {
            const uint64_t gu = u_begin + u;
            uint32_t sa = dq.seg0, sb = dq.seg0 + dq.nseg;  // last segment with seg_unit <= gu
            while (sb - sa > 1) {
                const uint32_t mid = (sa + sb) >> 1;
                if (seg_unit[mid] <= gu) sa = mid; else sb = mid;
            }
            const ScanSeg sg = segs[sa];
            const uint64_t blk = (sg.row0 >> 5) + (gu - seg_unit[sa]);
            const uint64_t gr = blk * 32 + lane;
            const bool valid = gr >= sg.row0 && gr < sg.row0 + sg.rows;
            const uint64_t ridx = sg.out0 + (gr - sg.row0);
            const bool mine = it % DT_WARPS == warp;  // this warp adds the unit up
            uint64_t rv = 0;
            uint32_t id = 0;
            if (mine && valid) {
                rv = __ldcg(r + ridx);
                id = dc.ids ? dc.ids[gr] : (uint32_t)gr;
            }
            uint64_t part = 0;
            if (warp < DT_DENSE) {
                const uint32_t cols = 2 * n1 / DT_DENSE;
                part = dense_terms_block(dc.alh_b, n1, blk, dyn_limbs, warp * cols, (warp + 1) * cols, lane);
            } else if (warp < DT_DENSE + DT_S) {
                part = s_times_v_part<DT_S>(dc, blk, vt, warp - DT_DENSE, lane);
            } else {  // half of the T entries each, whole groups of 32
                const uint32_t per = (tn / DT_T + 31) & ~31u, c0 = min(tn, (warp - DT_DENSE - DT_S) * per);
                const uint32_t c1 = warp == DT_WARPS - 1 ? tn : min(tn, per);
                if (dc.m8_cm) {
                    const int32_t mt = m_times_t_warp(dc.m8_cm, (dc.rows + 31) & ~31ull, blk, tl + c0, c1 - c0, lane);
                    part = mt >= 0 ? (uint64_t)mt : P - (uint64_t)(-(int64_t)mt);
                } else if (valid) {
                    part = m_times_t_cm(dc.mp_cm, dc.rows, gr, tl, c0, c1);
                }
            }
            auto sh = reinterpret_cast<uint64_t(*)[32]>(dyn_limbs + 4 * n1) + (it & 1) * DT_WARPS;
            sh[warp][lane] = part;
            __syncthreads();  // one per unit: the other buffer is rewritten only after the next one
            if (mine) {
                uint64_t sum = part;
#pragma unroll
                for (uint32_t w = 1; w < DT_WARPS; ++w) sum = add_mod(sum, sh[(warp + w) % DT_WARPS][lane]);
                const uint64_t mv = sub_mod(rv, sum);
                if (valid && mv_out) mv_out[ridx] = mv;
                const int64_t score = to_signed(mv);
                if constexpr (WARP_LISTS) warp_topk_offer(ls, li, (int)k, valid, score, id, lane);
                else topk_offer(buf, valid, score, id, buf.thr_s, buf.thr_i, buf.have_thr);
            }
        }
    } else {
        const uint64_t tiles = (u_count + DT_WARPS - 1) / DT_WARPS;
        // The buffer is checked (two CTA barriers) every DT_CHECK tiles, not
        // every tile, so the warps may drift apart within that window; between
        // checks at most DT_CHECK * 256 rows append, and a check compacts above
        // CAND_CAP - DT_CHECK * 256 = 1024 >= k entries.
        constexpr uint32_t DT_CHECK = 4;
        static_assert(CAND_CAP - DT_CHECK * DT_THREADS >= TOPK_MAX, "candidate buffer too small for the check interval");
        uint32_t it = 0;
        for (uint64_t tile = cta; tile < tiles; tile += dq.ctas, ++it) {
            const uint64_t u = tile * DT_WARPS + warp;
            bool valid = false;
            int64_t score = 0;
            uint32_t id = 0;
            if (u < u_count) {  // warp-uniform
                const uint64_t gu = u_begin + u;
                uint32_t sa = dq.seg0, sb = dq.seg0 + dq.nseg;  // last segment with seg_unit <= gu
                while (sb - sa > 1) {
                    const uint32_t mid = (sa + sb) >> 1;
                    if (seg_unit[mid] <= gu) sa = mid; else sb = mid;
                }
                const ScanSeg sg = segs[sa];
                const uint64_t blk = (sg.row0 >> 5) + (gu - seg_unit[sa]);
                const uint64_t gr = blk * 32 + lane;
                valid = gr >= sg.row0 && gr < sg.row0 + sg.rows;
                const uint64_t ridx = sg.out0 + (gr - sg.row0);
                uint64_t rv = 0;
                if (valid) {
                    rv = __ldcg(r + ridx);
                    id = dc.ids ? dc.ids[gr] : (uint32_t)gr;
                }
                uint64_t m_t = 0;
                if (dc.m8_cm) {
                    const int32_t mt = m_times_t_warp(dc.m8_cm, (dc.rows + 31) & ~31ull, blk, tl, tn, lane);
                    m_t = mt >= 0 ? (uint64_t)mt : P - (uint64_t)(-(int64_t)mt);
                }
                const uint64_t s_v = s_times_v_part<1>(dc, blk, vt, 0, lane);
                if (valid) {
                    const uint64_t dense = dense_terms_row(dc.alh_b, n1, gr, dyn_limbs);
                    if (!dc.m8_cm) m_t = m_times_t_cm(dc.mp_cm, dc.rows, gr, tl, 0, tn);
                    const uint64_t mv = sub_mod(sub_mod(rv, add_mod(dense, m_t)), s_v);
                    if (mv_out) mv_out[ridx] = mv;
                    score = to_signed(mv);
                }
            }
            if constexpr (WARP_LISTS) {
                warp_topk_offer(ls, li, (int)k, valid, score, id, lane);
            } else {
                const int64_t th_s = buf.thr_s;
                const uint32_t th_i = buf.thr_i;
                const int ht = buf.have_thr;
                topk_offer(buf, valid, score, id, th_s, th_i, ht);
                if (it % DT_CHECK == DT_CHECK - 1 && topk_full(buf, CAND_CAP - DT_CHECK * DT_THREADS))
                    topk_compact(buf, (int)k);
            }
        }
    }
    const uint32_t ctas = dq.ctas;
    const uint64_t slot = blockIdx.x;
    if constexpr (WARP_LISTS) {
        warp_topk_reduce(ls, li, (int)k, buf.s, buf.id, warp, lane);
        if (warp == 0) {
            const uint32_t keep = __popc(__ballot_sync(FULL, lane < k && ls != INT64_MIN));
            if (lane < keep) {
                ts.cand_s[slot * k + lane] = ls;
                ts.cand_i[slot * k + lane] = li;
            }
            if (lane == 0) ts.cand_n[slot] = keep;
        }
    } else {
        topk_compact(buf, (int)k);
        const int keep = min(buf.cnt, (int)k);
        for (int i = threadIdx.x; i < keep; i += blockDim.x) {
            ts.cand_s[slot * k + i] = buf.s[i];
            ts.cand_i[slot * k + i] = buf.id[i];
        }
        if (threadIdx.x == 0) ts.cand_n[slot] = (uint32_t)keep;
    }
    __threadfence();  // this CTA's lists are visible device-wide before its ticket
    __syncthreads();
    if (threadIdx.x == 0) last_s = atomicAdd(&ts.done[q], 1u) == ctas - 1;
    __syncthreads();
    if (!last_s) return;

    // ---------------------------------------------------------- merge (last CTA of the query)
    __threadfence();
    const uint64_t total = (uint64_t)ctas * k;
    if constexpr (WARP_LISTS) {
        // warp w takes entries w * 32 + lane + 256 i into its list; then warp 0 merges the lists
        ls = INT64_MIN;
        li = 0xffffffffu;
        for (uint64_t t0 = (uint64_t)warp * 32; t0 < total; t0 += DT_THREADS) {
            const uint64_t e = t0 + lane;
            bool v = false;
            int64_t sc = 0;
            uint32_t id = 0;
            if (e < total) {
                const uint64_t sl = (uint64_t)dq.cta0 + e / k;
                const uint32_t i = (uint32_t)(e % k);
                v = i < __ldcg(ts.cand_n + sl);
                if (v) {
                    sc = __ldcg(ts.cand_s + sl * k + i);
                    id = __ldcg(ts.cand_i + sl * k + i);
                }
            }
            warp_topk_offer(ls, li, (int)k, v, sc, id, lane);
        }
        warp_topk_reduce(ls, li, (int)k, buf.s, buf.id, warp, lane);
        if (warp == 0) {
            const uint32_t keep = __popc(__ballot_sync(FULL, lane < k && ls != INT64_MIN));
            if (lane < keep) {
                out_ids[(uint64_t)q * k + lane] = li;
                out_scores[(uint64_t)q * k + lane] = ls;
            }
            if (lane == 0) {
                out_n[q] = keep;
                ts.done[q] = 0;
            }
        }
        return;
    } else {
        if (threadIdx.x == 0) { buf.cnt = 0; buf.have_thr = 0; buf.thr_s = INT64_MIN; buf.thr_i = 0xffffffffu; }
        __syncthreads();
    // Four tiles of entries per round: their loads (written by other CTAs
    // during this launch, so read through L2) are all in flight before the
    // offers; entries past a list's count are loaded and ignored.
    for (uint64_t t0 = 0; t0 < total; t0 += 4 * DT_THREADS) {
        bool valid[4];
        int64_t sc[4];
        uint32_t id[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t e = t0 + u * DT_THREADS + threadIdx.x;
            valid[u] = false;
            sc[u] = 0;
            id[u] = 0;
            if (e < total) {
                const uint64_t sl = (uint64_t)dq.cta0 + e / k;
                const uint32_t i = (uint32_t)(e % k);
                const uint32_t n = __ldcg(ts.cand_n + sl);
                sc[u] = __ldcg(ts.cand_s + sl * k + i);
                id[u] = __ldcg(ts.cand_i + sl * k + i);
                valid[u] = i < n;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t th_s = buf.thr_s;
            const uint32_t th_i = buf.thr_i;
            const int ht = buf.have_thr;
            topk_offer(buf, valid[u], sc[u], id[u], th_s, th_i, ht);
            if (topk_full(buf, CAND_CAP - DT_THREADS)) topk_compact(buf, (int)k);
        }
    }
    topk_compact(buf, (int)k);
    const int out_keep = min(buf.cnt, (int)k);
    for (int i = threadIdx.x; i < out_keep; i += blockDim.x) {
        out_ids[(uint64_t)q * k + i] = buf.id[i];
        out_scores[(uint64_t)q * k + i] = buf.s[i];
    }
    if (threadIdx.x == 0) {
        out_n[q] = (uint32_t)out_keep;
        ts.done[q] = 0;
    }
    }
}

__global__ void __launch_bounds__(DT_THREADS)
topk_merge_kernel(const int64_t* __restrict__ cand_s, const uint32_t* __restrict__ cand_i,
                  const uint32_t* __restrict__ cand_n, uint32_t ctas, uint32_t k, uint32_t* __restrict__ out_ids,
                  int64_t* __restrict__ out_scores, uint32_t* __restrict__ out_n) {
    const uint32_t q = blockIdx.x;
    __shared__ TopkBuf buf;
    if (threadIdx.x == 0) { buf.cnt = 0; buf.have_thr = 0; buf.thr_s = INT64_MIN; buf.thr_i = 0xffffffffu; }
    __syncthreads();
    const uint64_t total = (uint64_t)ctas * k;
    for (uint64_t tile = 0; tile < total; tile += DT_THREADS) {
        const uint64_t e = tile + threadIdx.x;
        bool valid = false;
        int64_t s = 0;
        uint32_t id = 0;
        if (e < total) {
            const uint32_t c = (uint32_t)(e / k), i = (uint32_t)(e % k);
            const uint64_t slot = (uint64_t)q * ctas + c;
            if (i < cand_n[slot]) { valid = true; s = cand_s[slot * k + i]; id = cand_i[slot * k + i]; }
        }
        const int64_t ts = buf.thr_s;
        const uint32_t ti = buf.thr_i;
        const int ht = buf.have_thr;
        topk_offer(buf, valid, s, id, ts, ti, ht);
        if (topk_full(buf, CAND_CAP - DT_THREADS)) topk_compact(buf, (int)k);
    }
    topk_compact(buf, (int)k);
    const int keep = min(buf.cnt, (int)k);
    for (int i = threadIdx.x; i < keep; i += blockDim.x) {
        out_ids[(uint64_t)q * k + i] = buf.id[i];
        out_scores[(uint64_t)q * k + i] = buf.s[i];
    }
    if (threadIdx.x == 0) out_n[q] = (uint32_t)keep;
}

// The same for k <= 32 with the warps' own lists.
__global__ void __launch_bounds__(DT_THREADS)
topk_merge_warp_kernel(const int64_t* __restrict__ cand_s, const uint32_t* __restrict__ cand_i,
                       const uint32_t* __restrict__ cand_n, uint32_t ctas, uint32_t k, uint32_t* __restrict__ out_ids,
                       int64_t* __restrict__ out_scores, uint32_t* __restrict__ out_n) {
    const uint32_t q = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ int64_t xs[DT_THREADS];
    __shared__ uint32_t xi[DT_THREADS];
    int64_t ls = INT64_MIN;
    uint32_t li = 0xffffffffu;
    const uint32_t total = ctas * k;
    for (uint32_t t0 = warp * 32; t0 < total; t0 += DT_THREADS) {
        const uint32_t e = t0 + lane;
        bool v = false;
        int64_t sc = 0;
        uint32_t id = 0;
        if (e < total) {
            const uint64_t slot = (uint64_t)q * ctas + e / k;
            sc = cand_s[slot * k + e % k];  // entries past the list's count are loaded and ignored
            id = cand_i[slot * k + e % k];
            v = e % k < cand_n[slot];
        }
        warp_topk_offer(ls, li, (int)k, v, sc, id, lane);
    }
    warp_topk_reduce(ls, li, (int)k, xs, xi, warp, lane);
    if (warp == 0) {
        const uint32_t keep = __popc(__ballot_sync(FULL, lane < k && ls != INT64_MIN));
        if (lane < keep) {
            out_ids[(uint64_t)q * k + lane] = li;
            out_scores[(uint64_t)q * k + lane] = ls;
        }
        if (lane == 0) out_n[q] = keep;
    }
}

// Top-k of residues combined on the fly: query q's row i scores
// to_signed(a + b - c) (b, c nullable) with a = ra[q * ld + i] etc., ids[i]
// (or i); mv_out (nullable) receives the combined residues at the same
// offsets.  Same per-CTA candidate buffers as decode_topk_kernel, merged by
// topk_merge_kernel.
__global__ void __launch_bounds__(DT_THREADS)
topk_rows_kernel(const uint64_t* __restrict__ ra, const uint64_t* __restrict__ rb, const uint64_t* __restrict__ rc,
                 uint64_t ld, uint64_t rows, const uint64_t* __restrict__ qoff, const uint32_t* __restrict__ ids,
                 uint32_t k, int64_t* __restrict__ cand_s, uint32_t* __restrict__ cand_i, uint32_t* __restrict__ cand_n,
                 uint64_t* __restrict__ mv_out) {
    const uint32_t q = blockIdx.y;
    __shared__ TopkBuf buf;
    if (threadIdx.x == 0) { buf.cnt = 0; buf.have_thr = 0; buf.thr_s = INT64_MIN; buf.thr_i = 0xffffffffu; }
    __syncthreads();
    // rows of this query: [lo, hi) of row q (ld apart), or of the flat
    // segmented array [qoff[q], qoff[q+1]) (lo rounded down to even so the
    // paired loads stay 16-byte aligned; the extra entry is masked)
    const uint64_t base = qoff ? 0 : (uint64_t)q * ld;
    const uint64_t first = qoff ? qoff[q] : 0, hi = qoff ? qoff[q + 1] : rows;
    const uint64_t lo = first & ~1ull, span = hi > lo ? hi - lo : 0;
    const uint64_t per = ((span + gridDim.x - 1) / gridDim.x + 1) & ~1ull;
    const uint64_t v_begin = lo + min(span, (uint64_t)blockIdx.x * per);
    const uint64_t v_end = min(hi, v_begin + per);
    for (uint64_t tile = v_begin; tile < v_end; tile += 2 * DT_THREADS) {
        const uint64_t i0 = tile + 2 * threadIdx.x;
        const bool valid[2] = {i0 < v_end && i0 >= first, i0 + 1 < v_end};
        uint64_t mv[2] = {0, 0};
        if (i0 < v_end) {  // v_begin, per and ld are even: the pair is 16-byte aligned and inside the row of ld
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(ra + base + i0);
            mv[0] = x.x;
            mv[1] = x.y;
            if (rb) {
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(rb + base + i0);
                mv[0] = add_mod(mv[0], y.x);
                mv[1] = add_mod(mv[1], y.y);
            }
            if (rc) {
                const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(rc + base + i0);
                mv[0] = sub_mod(mv[0], z.x);
                mv[1] = sub_mod(mv[1], z.y);
            }
            if (mv_out) {
                if (valid[0]) mv_out[base + i0] = mv[0];
                if (valid[1]) mv_out[base + i0 + 1] = mv[1];
            }
        }
        int64_t sc[2];
        uint32_t id[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            sc[h] = to_signed(mv[h]);
            id[h] = valid[h] ? (ids ? ids[i0 + h] : (uint32_t)(i0 + h)) : 0;
        }
        const int64_t ts = buf.thr_s;
        const uint32_t ti = buf.thr_i;
        const int ht = buf.have_thr;
        topk_offer(buf, valid[0], sc[0], id[0], ts, ti, ht);
        topk_offer(buf, valid[1], sc[1], id[1], ts, ti, ht);
        if (topk_full(buf, CAND_CAP - 2 * DT_THREADS)) topk_compact(buf, (int)k);
    }
    topk_compact(buf, (int)k);
    const int keep = min(buf.cnt, (int)k);
    const uint64_t slot = (uint64_t)q * gridDim.x + blockIdx.x;
    for (int i = threadIdx.x; i < keep; i += blockDim.x) {
        cand_s[slot * k + i] = buf.s[i];
        cand_i[slot * k + i] = buf.id[i];
    }
    if (threadIdx.x == 0) cand_n[slot] = (uint32_t)keep;
}

// topk_rows_kernel for k <= 32: every warp keeps its own list, so the loop
// holds no block barrier, and a thread has TR_UNROLL pairs of rows of all
// three arrays in flight (the candidate buffer's two barriers per 512 rows
// held the pass at 0.4 TB/s with 8 queries).
constexpr uint32_t TR_UNROLL = 4;

__global__ void __launch_bounds__(DT_THREADS)
topk_rows_warp_kernel(const uint64_t* __restrict__ ra, const uint64_t* __restrict__ rb, const uint64_t* __restrict__ rc,
                      uint64_t ld, uint64_t rows, const uint64_t* __restrict__ qoff, const uint32_t* __restrict__ ids,
                      uint32_t k, int64_t* __restrict__ cand_s, uint32_t* __restrict__ cand_i,
                      uint32_t* __restrict__ cand_n, uint64_t* __restrict__ mv_out) {
    const uint32_t q = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ int64_t xs[DT_THREADS];
    __shared__ uint32_t xi[DT_THREADS];
    int64_t ls = INT64_MIN;
    uint32_t li = 0xffffffffu;
    const uint64_t base = qoff ? 0 : (uint64_t)q * ld;  // the same row ranges as topk_rows_kernel
    const uint64_t first = qoff ? qoff[q] : 0, hi = qoff ? qoff[q + 1] : rows;
    const uint64_t lo = first & ~1ull, span = hi > lo ? hi - lo : 0;
    const uint64_t per = ((span + gridDim.x - 1) / gridDim.x + 1) & ~1ull;
    const uint64_t v_begin = lo + min(span, (uint64_t)blockIdx.x * per);
    const uint64_t v_end = min(hi, v_begin + per);
    for (uint64_t tile = v_begin; tile < v_end; tile += 2 * DT_THREADS * TR_UNROLL) {
        ulonglong2 x[TR_UNROLL], y[TR_UNROLL], z[TR_UNROLL];
#pragma unroll
        for (uint32_t u = 0; u < TR_UNROLL; ++u) {
            const uint64_t i0 = tile + 2 * (u * DT_THREADS + threadIdx.x);
            x[u] = y[u] = z[u] = make_ulonglong2(0, 0);
            if (i0 < v_end) {  // 16-byte aligned and inside the row of ld, as in topk_rows_kernel
                x[u] = *reinterpret_cast<const ulonglong2*>(ra + base + i0);
                if (rb) y[u] = *reinterpret_cast<const ulonglong2*>(rb + base + i0);
                if (rc) z[u] = *reinterpret_cast<const ulonglong2*>(rc + base + i0);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < TR_UNROLL; ++u) {
            const uint64_t i0 = tile + 2 * (u * DT_THREADS + threadIdx.x);
            const bool valid[2] = {i0 < v_end && i0 >= first, i0 + 1 < v_end};
            const uint64_t mv[2] = {sub_mod(add_mod(x[u].x, y[u].x), z[u].x), sub_mod(add_mod(x[u].y, y[u].y), z[u].y)};
            const int64_t ts = __shfl_sync(FULL, ls, k - 1);  // scores below the k-th best need no id
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (mv_out && valid[h]) mv_out[base + i0 + h] = mv[h];
                const int64_t sc = to_signed(mv[h]);
                const bool v = valid[h] && sc >= ts;
                const uint32_t id = v ? (ids ? ids[i0 + h] : (uint32_t)(i0 + h)) : 0;
                if (__any_sync(FULL, v)) warp_topk_offer(ls, li, (int)k, v, sc, id, lane);
            }
        }
    }
    warp_topk_reduce(ls, li, (int)k, xs, xi, warp, lane);
    if (warp == 0) {
        const uint64_t slot = (uint64_t)q * gridDim.x + blockIdx.x;
        const uint32_t keep = __popc(__ballot_sync(FULL, lane < k && ls != INT64_MIN));
        if (lane < keep) {
            cand_s[slot * k + lane] = ls;
            cand_i[slot * k + lane] = li;
        }
        if (lane == 0) cand_n[slot] = keep;
    }
}

// k <= 32, what a warp's lanes hold: the warp-list kernels; larger k: the CTA
// candidate buffers.
void launch_topk(const uint64_t* d_a, const uint64_t* d_b, const uint64_t* d_c, uint64_t ld, uint64_t rows,
                 const uint64_t* d_qoff, uint32_t nq, const uint32_t* d_ids, uint32_t k, int ctas_per_query,
                 const TopkScratch& scratch, uint32_t* d_out_ids, int64_t* d_out_scores, uint32_t* d_out_n,
                 uint64_t* d_mv_out, cudaStream_t s) {
    if (!nq) return;
    const bool warp_lists = k >= 1 && k <= WARP_TOPK_MAX;
    const dim3 grid(ctas_per_query, nq);
    auto rows_fn = warp_lists ? topk_rows_warp_kernel : topk_rows_kernel;
    auto merge_fn = warp_lists ? topk_merge_warp_kernel : topk_merge_kernel;
    rows_fn<<<grid, DT_THREADS, 0, s>>>(d_a, d_b, d_c, ld, rows, d_qoff, d_ids, k, scratch.cand_s, scratch.cand_i,
                                        scratch.cand_n, d_mv_out);
    merge_fn<<<nq, DT_THREADS, 0, s>>>(scratch.cand_s, scratch.cand_i, scratch.cand_n, (uint32_t)ctas_per_query, k,
                                       d_out_ids, d_out_scores, d_out_n);
}

// ------------------------------------------------------------------ keygen GEMM
constexpr int GT = 64;   // output tile
constexpr int GK = 16;   // K chunk

__global__ void __launch_bounds__(256)
gemm_abt_kernel(const uint64_t* __restrict__ A, const uint64_t* __restrict__ B, const uint64_t* __restrict__ D,
                uint64_t rows, uint32_t cols, uint32_t K, uint64_t* __restrict__ C) {
    __shared__ uint64_t As[GT][GK + 1];
    __shared__ uint32_t Bs[GK][GT][6];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const uint64_t row0 = (uint64_t)blockIdx.x * GT;
    const uint32_t col0 = blockIdx.y * GT;
    uint64_t acc[4][4][3];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = acc[a][b][2] = 0;
    for (uint32_t kk = 0; kk < K; kk += GK) {
        for (int e = threadIdx.x; e < GT * GK; e += 256) {
            const int rr = e / GK, k = e % GK;
            const uint64_t gr = row0 + rr;
            As[rr][k] = gr < rows ? A[gr * K + kk + k] : 0;
            const uint32_t gc = col0 + rr;
            const uint64_t bv = gc < cols ? B[(uint64_t)gc * K + kk + k] : 0;
            Limbs3 lb = limbs(bv), lc = limbs_hi(bv);
            Bs[k][rr][0] = lb.b0; Bs[k][rr][1] = lb.b1; Bs[k][rr][2] = lb.b2;
            Bs[k][rr][3] = lc.b0; Bs[k][rr][4] = lc.b1; Bs[k][rr][5] = lc.b2;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < GK; ++k) {
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const uint64_t m = As[ty + 16 * a][k];
                const uint32_t lo = (uint32_t)m, hi = (uint32_t)(m >> 32);
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint32_t* l = Bs[k][tx + 16 * b];
                    acc[a][b][0] = mac(mac(acc[a][b][0], lo, l[0]), hi, l[3]);
                    acc[a][b][1] = mac(mac(acc[a][b][1], lo, l[1]), hi, l[4]);
                    acc[a][b][2] = mac(mac(acc[a][b][2], lo, l[2]), hi, l[5]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint64_t gr = row0 + ty + 16 * a;
            const uint32_t gc = col0 + tx + 16 * b;
            if (gr < rows && gc < cols) {
                uint64_t v = combine3(acc[a][b][0], acc[a][b][1], acc[a][b][2]);
                if (D) v = add_mod(v, D[gr * cols + gc]);
                C[gr * cols + gc] = v;
            }
        }
}

// A warp per row, 32 entries at a time; entries of one batch that name the same
// column (a CSR may repeat one) are applied one after the other.
__global__ void apply_sparse_kernel(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ idx,
                                    const int8_t* __restrict__ sign, uint64_t rows, uint32_t cols, uint64_t* C) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < rows; i += warps) {
        const uint64_t b = rowptr[i], e = rowptr[i + 1];
        for (uint64_t c = b; c < e; c += 32) {
            const bool on = c + lane < e;
            const uint32_t col = on ? idx[c + lane] : 0xffffffffu - lane;  // idle lanes: columns of their own
            const bool neg = on && sign[c + lane] < 0;
            const uint32_t same = __match_any_sync(FULL, col);
            const uint32_t rank = __popc(same & ((1u << lane) - 1));
            const uint32_t turns = __reduce_max_sync(FULL, rank);
            for (uint32_t t = 0; t <= turns; ++t) {
                if (on && rank == t) {
                    uint64_t* p = C + i * cols + col;
                    *p = neg ? sub_mod(*p, 1) : add_mod(*p, 1);
                }
                __syncwarp();
            }
        }
    }
}

__global__ void transpose_u64_kernel(const uint64_t* __restrict__ in, uint64_t rows, uint32_t cols,
                                     uint64_t* __restrict__ out, uint64_t out_ld) {
    __shared__ uint64_t t[32][33];
    const uint64_t r0 = (uint64_t)blockIdx.x * 32;
    const uint32_t c0 = blockIdx.y * 32;
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const uint64_t r = r0 + yy;
        const uint32_t c = c0 + threadIdx.x;
        t[yy][threadIdx.x] = (r < rows && c < cols) ? in[r * cols + c] : 0;
    }
    __syncthreads();
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const uint32_t c = c0 + yy;
        const uint64_t r = r0 + threadIdx.x;
        if (r < rows && c < cols) out[(uint64_t)c * out_ld + r] = t[threadIdx.x][yy];
    }
}

// The entries of a row may stand in any of its slots; they are dealt out so that
// the decode's table loads meet few bank conflicts.  One of those loads reads, in
// each half of a warp, 4 consecutive slots x 4 groups of 8 rows, and the 16
// 8-byte bank pairs are the table index mod 16: slot k of row group g prefers
// indices of class (k mod 4) + 4 ((g + k / 4) mod 4), which are 16 different ones
// over such a load, and every row meets every class once in 16 slots.  Entries
// whose class has no slot left (7 % at the mean of 128 per row) fill the others.
__global__ void csr_to_ell_kernel(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ idx,
                                  const int8_t* __restrict__ sign, uint64_t rows, const uint32_t* __restrict__ s_off,
                                  const uint16_t* __restrict__ s_w, uint16_t* __restrict__ ell) {
    // every row position of every slice is written: the positions past the
    // last row of the last slice hold padding
    const uint64_t rows32 = (rows + 31) & ~31ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows32; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t slice = i >> 5;
        const uint32_t sl = (uint32_t)(i & 31), w = s_w[slice], grp = sl >> 3;
        uint16_t* out = ell + s_off[slice] + sl;
        const uint64_t b = i < rows ? rowptr[i] : 0, e = i < rows ? rowptr[i + 1] : 0;
        for (uint32_t c = 0; c < w; ++c) out[c * 32] = (uint16_t)ELL_PAD;
        uint32_t fill = 0;  // second pass: slots below are taken
        for (int pass = 0; pass < 2; ++pass) {
            uint8_t period[16] = {};  // per class: entries met so far, one per 16 slots
            for (uint64_t c = b; c < e; ++c) {
                const uint32_t f = idx[c] + (sign[c] < 0 ? ELL_NEG : 0u), cls = f & 15;
                const uint32_t k = (cls & 3) + 4 * (((cls >> 2) - grp) & 3) + 16u * period[cls];
                if (period[cls] < 255) ++period[cls];
                if (pass == 0 && k < w) out[k * 32] = (uint16_t)f;
                if (pass == 1 && k >= w) {
                    while (out[fill * 32] != ELL_PAD) ++fill;  // the row has at most w entries
                    out[fill * 32] = (uint16_t)f;
                }
            }
        }
    }
}

inline unsigned grid_for(uint64_t n, unsigned threads, unsigned cap = 65535u * 16u) {
    uint64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

}  // namespace

// ------------------------------------------------------------------ launchers
void launch_query_limbs(const uint64_t* d_v, uint32_t nq, QLimb* d_limbs, cudaStream_t s) {
    const uint64_t total = (uint64_t)nq * N;
    query_limbs_kernel<<<grid_for(total, 256), 256, 0, s>>>(d_v, total, d_limbs);
}

void launch_scan(const uint64_t* d_m_enc, const QLimb* d_limbs, const ScanSeg* d_segs, const uint64_t* d_seg_blk,
                 uint32_t nseg, uint64_t total_blocks, uint64_t* d_r, int num_sms, uint32_t* d_err, cudaStream_t s,
                 long long wait_cycles) {
    if (total_blocks == 0) return;
    const int smem = TS_STAGES * TS_STAGE_BYTES;
    cudaFuncSetAttribute(scan_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);  // per device
    unsigned grid = (unsigned)(total_blocks < (uint64_t)num_sms ? total_blocks : (uint64_t)num_sms);
    scan_tma_kernel<<<grid, TS_THREADS, smem, s>>>(d_m_enc, d_limbs, d_segs, d_seg_blk, nseg, total_blocks, d_r, d_err,
                                                   wait_cycles > 0 ? wait_cycles : WAIT_CYCLES);
}

FreivaldsPlan plan_freivalds(uint64_t max_rows, uint32_t nseg, int num_sms) {
    // aim for ~2 waves of 4-column-block CTAs over all segments
    uint64_t target_ctas = (uint64_t)num_sms * 4;
    uint64_t per_seg = target_ctas / (4ull * (nseg ? nseg : 1));
    if (per_seg < 1) per_seg = 1;
    uint64_t chunk_rows = (max_rows + per_seg - 1) / per_seg;
    chunk_rows = ((chunk_rows + FV_TILE - 1) / FV_TILE) * FV_TILE;
    if (chunk_rows < FV_TILE) chunk_rows = FV_TILE;
    uint64_t chunks = (max_rows + chunk_rows - 1) / chunk_rows;
    if (chunks < 1) chunks = 1;
    return FreivaldsPlan{(uint32_t)chunks, (uint32_t)chunk_rows};
}

void launch_or_flag(uint32_t* d_word, uint32_t bits, cudaStream_t s) { or_flag_kernel<<<1, 1, 0, s>>>(d_word, bits); }

cudaError_t preload_freivalds_kernels() {
    cudaFuncAttributes a;
    const void* fns[] = {reinterpret_cast<const void*>(freivalds_kernel<24>),
                         reinterpret_cast<const void*>(freivalds_kernel<8>),
                         reinterpret_cast<const void*>(freivalds_kernel<4>),
                         reinterpret_cast<const void*>(freivalds_finish_kernel),
                         reinterpret_cast<const void*>(or_flag_kernel)};
    for (const void* f : fns) {
        const cudaError_t e = cudaFuncGetAttributes(&a, f);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void launch_freivalds(const uint64_t* d_m_enc, const uint64_t* d_r, const VerifySeg* d_vsegs, uint32_t nseg,
                      const ChaChaKey* d_keys, uint32_t trials, FreivaldsPlan plan, uint64_t* d_z_part,
                      uint64_t* d_ur_part, uint32_t* d_flags, cudaStream_t s) {
    for (uint32_t s0 = 0; s0 < nseg; s0 += 65535u) {
        const uint32_t ns = nseg - s0 < 65535u ? nseg - s0 : 65535u;
        dim3 grid(N / FV_THREADS, plan.chunks, ns);
        for (uint32_t t0 = 0; t0 < trials;) {
            const uint32_t left = trials - t0;
            if (left > 8) {
                const uint32_t c = left < 24 ? left : 24;
                freivalds_kernel<24><<<grid, FV_THREADS, 0, s>>>(d_m_enc, d_r, d_vsegs, d_keys, t0, c, trials, plan.chunks,
                                                                 plan.chunk_rows, d_z_part, d_ur_part, d_flags, s0);
                t0 += c;
            } else if (left > 4) {
                freivalds_kernel<8><<<grid, FV_THREADS, 0, s>>>(d_m_enc, d_r, d_vsegs, d_keys, t0, left, trials,
                                                                plan.chunks, plan.chunk_rows, d_z_part, d_ur_part, d_flags, s0);
                t0 += left;
            } else {
                freivalds_kernel<4><<<grid, FV_THREADS, 0, s>>>(d_m_enc, d_r, d_vsegs, d_keys, t0, left, trials,
                                                                plan.chunks, plan.chunk_rows, d_z_part, d_ur_part, d_flags, s0);
                t0 += left;
            }
        }
    }
}

void launch_freivalds_finish(const uint64_t* d_z_part, const uint64_t* d_ur_part, const uint64_t* d_v_enc,
                             const VerifySeg* d_vsegs, uint32_t nseg, uint32_t trials, FreivaldsPlan plan,
                             uint64_t* d_ur, uint64_t* d_zv, int32_t* d_failed, cudaStream_t s) {
    freivalds_finish_kernel<<<nseg, 256, 0, s>>>(d_z_part, d_ur_part, d_v_enc, d_vsegs, trials, plan.chunks, d_ur, d_zv,
                                                 d_failed);
}

void launch_lt_times_v(const uint64_t* d_L, uint32_t n1, const uint64_t* d_v, uint32_t nq, uint64_t* d_x,
                       cudaStream_t s) {
    if (!nq) return;
    const uint32_t run = lt_run(n1, nq);
    lt_times_v_kernel<<<dim3(n1 / LT_COLS, (nq + run - 1) / run), LT_THREADS, 0, s>>>(d_L, n1, d_v, nq, run, d_x);
}

void launch_query_prep(const uint64_t* d_L, uint32_t n1, const uint64_t* d_v, uint32_t nq, uint64_t* d_x, uint8_t* d_w,
                       uint32_t* d_zero, uint32_t zero_words, cudaStream_t s) {
    const uint32_t run = lt_run(n1, nq);
    const uint32_t lt_ctas = d_x ? (nq + run - 1) / run * (n1 / LT_COLS) : 0;
    const uint32_t wimg_ctas = d_w ? nq * (64 * 16 * 16 / LT_THREADS) : 0;
    query_prep_kernel<<<lt_ctas + wimg_ctas + 1, LT_THREADS, 0, s>>>(d_L, n1, d_v, nq, run, lt_ctas, d_x, wimg_ctas, d_w,
                                                                      d_zero, zero_words);
}

void launch_dense_terms(const uint64_t* d_al_cm, const uint64_t* d_h_cm, uint64_t rows, uint32_t n1,
                        const uint64_t* d_g, const uint64_t* d_x, uint64_t* d_out, cudaStream_t s) {
    dense_terms_kernel<<<grid_for(rows, 32, 148 * 4), 32 * DN_WARPS, 0, s>>>(d_al_cm, d_h_cm, rows, n1, d_g, d_x, d_out);
}

void launch_decode_layout(const uint64_t* d_al_cm, const uint64_t* d_h_cm, const uint64_t* d_mp_cm, uint64_t rows,
                          uint32_t n1, uint64_t* d_alh_b, int8_t* d_m8_cm, uint32_t* d_bad, cudaStream_t s) {
    cudaMemsetAsync(d_bad, 0, 4, s);
    if (!rows) return;
    decode_layout_kernel<<<148 * 16, 256, 0, s>>>(d_al_cm, d_h_cm, d_mp_cm, rows, n1, d_alh_b, d_m8_cm, d_bad);
}

void launch_decode_topk(const uint64_t* d_r, const DecodeCorpus& dc, const ScanSeg* d_segs, const uint64_t* d_seg_unit,
                        const DecodeQuery* d_q, uint32_t nq, const uint64_t* d_v, const uint64_t* d_g, const uint64_t* d_x, const uint32_t* d_t,
                        const uint32_t* d_t_nnz, uint32_t k, uint32_t total_ctas, bool split, TopkScratch scratch,
                        uint64_t* d_mv_out, uint32_t* d_out_ids, int64_t* d_out_scores, uint32_t* d_out_n,
                        cudaStream_t s) {
    if (!nq) return;
    const unsigned shares = split ? 2 * DT_WARPS * 32 * 8 : 0, dyn = 2 * 2 * dc.n1 * 16 + shares;
    const bool lists = k >= 1 && k <= WARP_TOPK_MAX;  // every warp keeps its own list
    auto fn = split ? (lists ? decode_topk_kernel<true, true> : decode_topk_kernel<false, true>)
                    : (lists ? decode_topk_kernel<true, false> : decode_topk_kernel<false, false>);
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * 2 * 512 * 16 + shares));
    // A split decode is short, and its set-up is worth overlapping with the kernels
    // before it (5,000 rows: 118 -> 105 us for the call with the whole chain).  A long
    // one is not: started among the CTAs of the kernels before it, it lost more than
    // the 3 us of set-up (four queries over 100,003 rows 1032 -> 1091 us).
    if (split)
        launch_after(fn, total_ctas, DT_THREADS, dyn, s, d_r, dc, d_segs, d_seg_unit, d_q, d_v, d_g, d_x, d_t, d_t_nnz, k,
                     scratch, d_mv_out, d_out_ids, d_out_scores, d_out_n, nq);
    else
        fn<<<total_ctas, DT_THREADS, dyn, s>>>(d_r, dc, d_segs, d_seg_unit, d_q, d_v, d_g, d_x, d_t, d_t_nnz, k, scratch,
                                               d_mv_out, d_out_ids, d_out_scores, d_out_n, nq);
}

void launch_topk_rows(const uint64_t* d_a, const uint64_t* d_b, const uint64_t* d_c, uint64_t ld, uint64_t rows,
                      uint32_t nq, const uint32_t* d_ids, uint32_t k, int ctas_per_query, TopkScratch scratch,
                      uint32_t* d_out_ids, int64_t* d_out_scores, uint32_t* d_out_n, uint64_t* d_mv_out,
                      cudaStream_t s) {
    launch_topk(d_a, d_b, d_c, ld, rows, nullptr, nq, d_ids, k, ctas_per_query, scratch, d_out_ids, d_out_scores, d_out_n,
                d_mv_out, s);
}

void launch_topk_segs(const uint64_t* d_a, const uint64_t* d_b, const uint64_t* d_c, const uint64_t* d_qoff,
                      uint32_t nq, const uint32_t* d_ids, uint32_t k, int ctas_per_query, TopkScratch scratch,
                      uint32_t* d_out_ids, int64_t* d_out_scores, uint32_t* d_out_n, cudaStream_t s) {
    launch_topk(d_a, d_b, d_c, 0, 0, d_qoff, nq, d_ids, k, ctas_per_query, scratch, d_out_ids, d_out_scores, d_out_n,
                nullptr, s);
}

void launch_gemm_abt(const uint64_t* d_A, const uint64_t* d_B, const uint64_t* d_D, uint64_t rows, uint32_t cols,
                     uint32_t K, uint64_t* d_C, cudaStream_t s) {
    dim3 grid((unsigned)((rows + GT - 1) / GT), (cols + GT - 1) / GT);
    gemm_abt_kernel<<<grid, 256, 0, s>>>(d_A, d_B, d_D, rows, cols, K, d_C);
}

void launch_apply_sparse(const uint64_t* d_rowptr, const uint32_t* d_idx, const int8_t* d_sign, uint64_t rows,
                         uint32_t cols, uint64_t* d_C, cudaStream_t s) {
    apply_sparse_kernel<<<grid_for(rows * 32, 256, 148 * 16), 256, 0, s>>>(d_rowptr, d_idx, d_sign, rows, cols, d_C);
}

void launch_transpose_u64(const uint64_t* d_in, uint64_t rows, uint32_t cols, uint64_t* d_out, uint64_t out_ld,
                          cudaStream_t s) {
    dim3 grid((unsigned)((rows + 31) / 32), (cols + 31) / 32);
    transpose_u64_kernel<<<grid, dim3(32, 8), 0, s>>>(d_in, rows, cols, d_out, out_ld);
}

void launch_csr_to_ell(const uint64_t* d_rowptr, const uint32_t* d_idx, const int8_t* d_sign, uint64_t rows,
                       const uint32_t* d_s_off, const uint16_t* d_s_w, uint16_t* d_s_ell, cudaStream_t s) {
    csr_to_ell_kernel<<<grid_for((rows + 31) & ~31ull, 256, 148 * 16), 256, 0, s>>>(d_rowptr, d_idx, d_sign, rows, d_s_off,
                                                                                   d_s_w, d_s_ell);
}

}  // namespace bn
