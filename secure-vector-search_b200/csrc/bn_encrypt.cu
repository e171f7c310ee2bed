// bn_encrypt.cu -- the two dense products of the encryption on the tensor
// cores: M_enc = M + H L^T (+ S) and AL = M L (crypto.rs:405-478).
//
// Both are products of u64 residues with the 1024 x n1 matrix L, so they are
// the byte-planar GEMM of block scoring (bn_batch.cuh) with L's rows or columns
// in the place of the queries: A = byte planes of a chunk of H (or M) rows, W =
// byte planes of L (or L^T).  The GEMM writes its results column by column; a
// transpose brings them to rows and adds M.  4,096 rows at n1 = 128 on the CUDA
// cores took 855 + 955 us (six multiply-adds per term, 128 CTAs for AL).
#include <cuda_runtime.h>

#include <algorithm>

#include "bn_batch.cuh"
#include "bn_internal.cuh"
#include "bn_tc.cuh"

namespace bn {
namespace api {

namespace {

// out[i * out_ld + j] = in[j * rows + i] (+ add[i * out_ld + j] mod p), i < rows, j < cols.
__global__ void transpose_add_kernel(const uint64_t* __restrict__ in, uint32_t rows, uint32_t cols,
                                     const uint64_t* __restrict__ add, uint64_t* __restrict__ out, uint64_t out_ld) {
    __shared__ uint64_t t[32][33];
    const uint32_t i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    for (uint32_t y = threadIdx.y; y < 32; y += blockDim.y) {
        const uint32_t i = i0 + threadIdx.x, j = j0 + y;
        t[y][threadIdx.x] = i < rows && j < cols ? in[(uint64_t)j * rows + i] : 0;
    }
    __syncthreads();
    for (uint32_t y = threadIdx.y; y < 32; y += blockDim.y) {
        const uint32_t i = i0 + y, j = j0 + threadIdx.x;
        if (i < rows && j < cols) {
            const uint64_t at = (uint64_t)i * out_ld + j;
            out[at] = add ? add_mod(t[threadIdx.x][y], add[at]) : t[threadIdx.x][y];
        }
    }
}

void launch_transpose_add(const uint64_t* in, uint32_t rows, uint32_t cols, const uint64_t* add, uint64_t* out,
                          uint64_t out_ld, cudaStream_t s) {
    transpose_add_kernel<<<dim3((rows + 31) / 32, (cols + 31) / 32), dim3(32, 8), 0, s>>>(in, rows, cols, add, out, out_ld);
}

// out[y * rows + x] = sum_k A[x][k] W[y][k] mod p from byte planes: A K-blocked
// (rows of 128 bytes), W row-major, k_bytes per plane row.
int planar_product(const void* a, uint64_t rows, const void* w, uint32_t cols, uint32_t k_bytes, uint64_t* out,
                   uint32_t* err, int sms, cudaStream_t s) {
    BgParams p{};
    p.mode = BG_PLANAR;
    p.a_tiles = (uint32_t)((rows * 8 + BG_AROWS - 1) / BG_AROWS);
    p.w_tile = 256;
    p.w_tiles = (8 * cols + p.w_tile - 1) / p.w_tile;
    p.k_bytes = p.k_panel = k_bytes;
    p.x_count = (uint32_t)rows;
    p.y_count = cols;
    p.out = out;
    p.out_ld = rows;
    p.a_blocked = 1;
    p.ksteps2 = k_bytes % (2 * BG_KSTEP) == 0;
    const uint64_t a_rows = (uint64_t)p.a_tiles * BG_AROWS * (k_bytes / BG_KSTEP);  // of 128 bytes
    CUtensorMap ta, tw, ta2, tw2;
    cudaError_t e = make_tmap_u8(&ta, a, BG_KSTEP, a_rows, BG_KSTEP, BG_AROWS);
    if (e == cudaSuccess) e = make_tmap_u8(&tw, w, k_bytes, 8ull * cols, BG_KSTEP, p.w_tile);
    if (e == cudaSuccess && p.ksteps2) e = make_tmap_u8(&ta2, a, BG_KSTEP, a_rows, BG_KSTEP, 2 * BG_AROWS);
    if (e == cudaSuccess && p.ksteps2) e = make_tmap_u8_ksteps2(&tw2, w, k_bytes, 8ull * cols, p.w_tile);
    if (e != cudaSuccess) return fail(BN_ECUDA, "tensor map of the encryption operands: %s", cudaGetErrorString(e));
    launch_bgemm(ta, tw, p, bgemm_max_stages(p), sms, err, s, p.ksteps2 ? &ta2 : nullptr, p.ksteps2 ? &tw2 : nullptr);
    return BN_OK;
}

}  // namespace

// Rows per pass: 8,192 (its planes and results take about 140 MB at n1 = 128).
constexpr uint64_t ENC_ROWS = 8192;

int encrypt_dense(bn_ctx* ctx, const uint64_t* d_mq, uint64_t rows, uint32_t n1, const uint64_t* d_L,
                  const uint64_t* d_H, uint64_t* d_enc, uint64_t* d_al, DevMem& ws, cudaStream_t s) {
    const uint64_t chunk = std::min<uint64_t>(ENC_ROWS, align_up(rows, 16));
    const uint32_t kh = (uint32_t)align_up(n1, BG_KSTEP);  // bytes of an H or L plane row, zero-padded
    Layout l;
    const uint64_t o_err = l.take<uint32_t>(1), o_lt = l.take<uint64_t>((uint64_t)n1 * N),
                   o_ltp = l.take<uint8_t>(8ull * n1 * N), o_lp = l.take<uint8_t>(8ull * N * kh),
                   o_hp = l.take<uint8_t>(8 * chunk * kh), o_mp = l.take<uint8_t>(8 * chunk * N),
                   o_oe = l.take<uint64_t>(chunk * N), o_oa = l.take<uint64_t>(chunk * n1);
    if (ws.alloc(ctx, l.off + 1024) != BN_OK) {  // over the budget, or the device is full: the caller has a way without
        cudaGetLastError();
        return BN_EBUDGET;
    }
    char* d = ws.at<char>();
    uint32_t* err = reinterpret_cast<uint32_t*>(d + o_err);
    uint64_t* lt = reinterpret_cast<uint64_t*>(d + o_lt);
    uint64_t* oe = reinterpret_cast<uint64_t*>(d + o_oe);
    uint64_t* oa = reinterpret_cast<uint64_t*>(d + o_oa);
    auto u8 = [&](uint64_t o) { return reinterpret_cast<uint8_t*>(d + o); };
    const int sms = ctx->num_sms;
    CU(cudaMemsetAsync(err, 0, 4, s));
    if (kh != n1) CU(cudaMemsetAsync(d + o_lp, 0, o_mp - o_lp, s));  // the pad columns of both
    launch_transpose_add(d_L, n1, N, nullptr, lt, N, s);  // L is [N][n1]: lt[k][j] = L[j][k]
    launch_planar_rows(lt, n1, N, N, u8(o_ltp), N, s);
    launch_planar_rows(d_L, N, n1, n1, u8(o_lp), kh, s);
    for (uint64_t r0 = 0; r0 < rows; r0 += chunk) {
        const uint32_t cr = (uint32_t)std::min(chunk, rows - r0);
        launch_planar_rows(d_H + r0 * n1, cr, n1, n1, u8(o_hp), 0, s, nullptr, kh / BG_KSTEP);
        TRY(planar_product(d + o_hp, cr, d + o_lp, N, kh, oe, err, sms, s));
        launch_transpose_add(oe, cr, N, d_mq + r0 * N, d_enc + r0 * N, N, s);
        launch_planar_rows(d_mq + r0 * N, cr, N, N, u8(o_mp), 0, s, nullptr, N / BG_KSTEP);
        TRY(planar_product(d + o_mp, cr, d + o_ltp, n1, N, oa, err, sms, s));
        launch_transpose_add(oa, cr, n1, nullptr, d_al + r0 * n1, n1, s);
    }
    CU(cudaGetLastError());
    uint32_t flags = 0;
    CU(cudaMemcpyAsync(&flags, err, 4, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    return device_flags_status(flags);
}

}  // namespace api
}  // namespace bn
