// bn_xfer.cu -- copies between pageable host memory and the device.
//
// A cudaMemcpy of pageable memory is copied by the driver through its own
// staging on one host thread (and takes the first-touch page faults of a fresh
// output array on it): 1.2 MB of r took about as long as the scan that computed
// it.  Here such copies go through a few pinned slots of the context, filled
// or emptied by several threads while the previous slot is on the link.
#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <cstring>

#include "bn_internal.cuh"

namespace bn {
namespace api {

namespace {

// A team of threads for the larger checks and copies: always of the same size,
// for OpenMP ends and makes threads whenever a team differs from the last one, and
// that of the library's host functions (all threads) where those are no more than
// TEAM.  With one thread per 128 KB a call's check and its copies took teams of
// different sizes: verify of 150,000 rows 512 us (378 without any), now 373; a
// quantise between such calls 196 us, now 11.  Below CHECK_FROM and COPY_FROM bytes
// one core is done before a team that has gone to sleep wakes up (50 us), and a copy
// up is left to the driver (verify of 60,000 rows, 480 KB: staged 199 us, now 196; a
// copy down gains by its slots from MIN_BYTES on: products of 40,000 rows 170 -> 113).
constexpr int TEAM = 16;
constexpr uint64_t CHECK_FROM = 1u << 20, COPY_FROM = 512u << 10;
int threads_for(uint64_t bytes, uint64_t from) { return bytes < from ? 1 : std::min(TEAM, omp_get_max_threads()); }

void parallel_memcpy(void* dst, const void* src, uint64_t bytes, int nt) {
    if (nt == 1) {
        memcpy(dst, src, bytes);
        return;
    }
    const uint64_t per = (bytes / nt + 4095) & ~4095ull;
#pragma omp parallel for num_threads(nt) schedule(static, 1)
    for (int t = 0; t < nt; ++t) {
        const uint64_t b = std::min(bytes, per * t), e = t == nt - 1 ? bytes : std::min(bytes, per * (t + 1));
        if (e > b) memcpy(static_cast<char*>(dst) + b, static_cast<const char*>(src) + b, e - b);
    }
}

bool is_pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Whether a copy of `bytes` may use the context's slots (caller holds st.mu); if not
// it goes to the driver, as it would without them.  They are made once the copies
// they could have served add up to FROM_BYTES: to pin and to release 6 MB takes 6 + 5 ms,
// about what the slots save on 64 MB of copies (a context that only drew the keys of
// 4,096 rows took 10 ms for it with slots made at once, 4.3 ms without).  Where they
// cannot be made, the next try comes after as many bytes again.
bool stage_ready(HostStage& st, uint64_t bytes) {
    if (st.p) return true;
    st.asked += bytes;
    if (st.asked < HostStage::FROM_BYTES) return false;
    st.asked = 0;
    for (cudaEvent_t& e : st.ev)
        if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            e = nullptr;
            cudaGetLastError();
            return false;
        }
    if (cudaMallocHost(&st.p, HostStage::SLOTS * HostStage::SLOT_BYTES) != cudaSuccess) {
        st.p = nullptr;
        cudaGetLastError();
        return false;
    }
    return true;
}

// Bytes per slot of one copy: quarters of it, so that a copy of a few hundred
// KB also overlaps its two halves, up to a whole slot.
uint64_t slot_bytes(uint64_t bytes) {
    return std::min<uint64_t>(HostStage::SLOT_BYTES, std::max<uint64_t>(256u << 10, align_up(bytes / 4, 4096)));
}

}  // namespace

HostStage::~HostStage() {
    for (cudaEvent_t e : ev)
        if (e) cudaEventDestroy(e);
    if (p) cudaFreeHost(p);
}

int stage_h2d(bn_ctx* ctx, void* dst, const void* src, uint64_t bytes, cudaStream_t s) {
    if (!bytes) return BN_OK;
    HostStage& st = ctx->stage;
    std::unique_lock<std::mutex> g(st.mu, std::defer_lock);
    if (bytes < COPY_FROM || !is_pageable(src) || !g.try_lock() ||  // another thread's copy is staged
        !stage_ready(st, bytes)) {
        CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
        return BN_OK;
    }
    const uint64_t step = slot_bytes(bytes);
    const int nt = threads_for(bytes, COPY_FROM);
    for (uint64_t off = 0, i = 0; off < bytes; off += step, ++i) {
        const uint64_t n = std::min(step, bytes - off);
        const int k = (int)(i % HostStage::SLOTS);
        char* slot = static_cast<char*>(st.p) + k * HostStage::SLOT_BYTES;
        CU(cudaEventSynchronize(st.ev[k]));  // the slot's last copy has left it
        parallel_memcpy(slot, static_cast<const char*>(src) + off, n, nt);
        CU(cudaMemcpyAsync(static_cast<char*>(dst) + off, slot, n, cudaMemcpyHostToDevice, s));
        CU(cudaEventRecord(st.ev[k], s));
    }
    return BN_OK;
}

int stage_d2h(bn_ctx* ctx, void* dst, const void* src, uint64_t bytes, cudaStream_t s) {
    if (!bytes) return BN_OK;
    HostStage& st = ctx->stage;
    std::unique_lock<std::mutex> g(st.mu, std::defer_lock);
    if (bytes < HostStage::MIN_BYTES || !is_pageable(dst) || !g.try_lock() || !stage_ready(st, bytes)) {
        CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
        CU(cudaStreamSynchronize(s));
        return BN_OK;
    }
    const uint64_t step = slot_bytes(bytes), total = (bytes + step - 1) / step;
    const int nt = threads_for(bytes, COPY_FROM);
    for (uint64_t i = 0; i < total + HostStage::SLOTS - 1; ++i) {
        if (i < total) {
            const int k = (int)(i % HostStage::SLOTS);
            const uint64_t off = i * step, n = std::min(step, bytes - off);
            if (i < HostStage::SLOTS) CU(cudaEventSynchronize(st.ev[k]));  // an earlier call's copy may still read it
            CU(cudaMemcpyAsync(static_cast<char*>(st.p) + k * HostStage::SLOT_BYTES, static_cast<const char*>(src) + off, n,
                               cudaMemcpyDeviceToHost, s));
            CU(cudaEventRecord(st.ev[k], s));
        }
        if (i + 1 >= HostStage::SLOTS) {
            const uint64_t j = i + 1 - HostStage::SLOTS;  // the oldest copy in flight
            const int k = (int)(j % HostStage::SLOTS);
            const uint64_t off = j * step;
            CU(cudaEventSynchronize(st.ev[k]));
            parallel_memcpy(static_cast<char*>(dst) + off, static_cast<char*>(st.p) + k * HostStage::SLOT_BYTES,
                            std::min(step, bytes - off), nt);
        }
    }
    return BN_OK;
}

// a >= p = 2^61 - 1 exactly when a or a + 1 has a bit from 61 on, so a run is
// checked with one OR per element; the first offender is named.
int validate_residues(const uint64_t* a, uint64_t count, const char* what) {
    constexpr uint64_t RUN = 1u << 15;
    const int64_t runs = (int64_t)((count + RUN - 1) / RUN);
    int64_t bad = runs;
    const int nt = threads_for(count * 8, CHECK_FROM);
#pragma omp parallel for num_threads(nt) schedule(static) reduction(min : bad) if (nt > 1)
    for (int64_t b = 0; b < runs; ++b) {
        const uint64_t i0 = b * RUN, i1 = std::min<uint64_t>(count, i0 + RUN);
        uint64_t any = 0;
        for (uint64_t i = i0; i < i1; ++i) any |= a[i] | (a[i] + 1);
        if (any >> 61) bad = std::min(bad, b);
    }
    if (bad == runs) return BN_OK;
    uint64_t i = bad * RUN;
    while (a[i] < P) ++i;
    return fail(BN_EINVAL, "%s[%llu] = %llu is not a canonical residue mod 2^61-1", what, (unsigned long long)i,
                (unsigned long long)a[i]);
}

uint64_t first_bad_entry(bn_sparse_csr S, uint64_t nnz) {
    constexpr uint64_t RUN = 1u << 15;
    for (uint64_t i0 = 0; i0 < nnz; i0 += RUN) {
        const uint64_t i1 = std::min(nnz, i0 + RUN);
        uint32_t any = 0;  // a column from n on, or a sign whose square is not 1
        for (uint64_t i = i0; i < i1; ++i) any |= S.idx[i] / N;
        for (uint64_t i = i0; i < i1; ++i) any |= (uint32_t)(S.sign[i] * S.sign[i]) ^ 1u;
        for (uint64_t i = i0; any && i < i1; ++i)
            if (S.idx[i] >= N || (S.sign[i] != 1 && S.sign[i] != -1)) return i;
    }
    return nnz;
}

}  // namespace api
}  // namespace bn
