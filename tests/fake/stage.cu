// The staged host copies (bn_xfer.cu) over a runtime of this file's own, on the
// CPU: streams are queues of copies that run only when something waits for them,
// "device" memory is host memory, and pinning can be made to fail.
//   stage copies   copies both ways from two threads through one context, sources
//                  overwritten as soon as stage_h2d returns
//   stage pinfail  prints how often 200 copies of 1 MB tried to pin the slots
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <thread>
#include <vector>

#include "bn_internal.cuh"

namespace fake {
std::mutex mu;
struct Queue {
    std::vector<std::function<void()>> ops;
    size_t done = 0;
    void run(size_t to) {
        for (; done < to; ++done) ops[done]();
    }
};
std::map<cudaStream_t, Queue> queues;
std::map<cudaEvent_t, std::pair<cudaStream_t, size_t>> marks;
std::vector<std::pair<char*, size_t>> pinned;
int pin_calls = 0;
bool pin_fails = false;

bool is_pinned(const void* p) {
    for (auto& x : pinned)
        if (p >= x.first && p < x.first + x.second) return true;
    return false;
}
cudaError_t getAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> g(mu);
    a->type = is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t eventCreate(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(malloc(1));
    return cudaSuccess;
}
cudaError_t eventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t mallocHost(void** p, size_t n) {
    std::lock_guard<std::mutex> g(mu);
    ++pin_calls;
    if (pin_fails) return cudaErrorMemoryAllocation;
    *p = malloc(n);
    pinned.emplace_back(static_cast<char*>(*p), n);
    return cudaSuccess;
}
cudaError_t freeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t memcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    std::lock_guard<std::mutex> g(mu);
    Queue& q = queues[st];
    const bool host_pinned = is_pinned(kind == cudaMemcpyHostToDevice ? s : d);
    q.ops.push_back([=] { memcpy(d, s, n); });
    if (!host_pinned) q.run(q.ops.size());  // a pageable copy has left or reached the host on return
    return cudaSuccess;
}
cudaError_t eventRecord(cudaEvent_t e, cudaStream_t st) {
    std::lock_guard<std::mutex> g(mu);
    marks[e] = {st, queues[st].ops.size()};
    return cudaSuccess;
}
cudaError_t eventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::mutex> g(mu);
    auto it = marks.find(e);
    if (it != marks.end()) queues[it->second.first].run(it->second.second);
    return cudaSuccess;
}
cudaError_t streamSynchronize(cudaStream_t st) {
    std::lock_guard<std::mutex> g(mu);
    Queue& q = queues[st];
    q.run(q.ops.size());
    return cudaSuccess;
}
cudaError_t getLastError() { return cudaSuccess; }
}  // namespace fake

namespace bn {
namespace api {
int fail(int code, const char* fmt, ...) {
    va_list a;
    va_start(a, fmt);
    vfprintf(stderr, fmt, a);
    va_end(a);
    return code;
}
}  // namespace api
}  // namespace bn

#define cudaPointerGetAttributes fake::getAttributes
#define cudaEventCreateWithFlags fake::eventCreate
#define cudaEventDestroy fake::eventDestroy
#define cudaMallocHost fake::mallocHost
#define cudaFreeHost fake::freeHost
#define cudaMemcpyAsync fake::memcpyAsync
#define cudaEventRecord fake::eventRecord
#define cudaEventSynchronize fake::eventSynchronize
#define cudaStreamSynchronize fake::streamSynchronize
#define cudaGetLastError fake::getLastError
#include "bn_xfer.cu"

using namespace bn::api;

static int copies() {
    bn_ctx ctx;
    std::vector<char> warm(8u << 20), dev(8u << 20);  // 64 MB of copies: the slots are made
    for (int i = 0; i < 9; ++i)
        if (stage_h2d(&ctx, dev.data(), warm.data(), warm.size(), nullptr) != BN_OK) return 1;
    if (!ctx.stage.p) return 2;
    int bad[2] = {0, 0};
    auto work = [&](int t) {
        const cudaStream_t s = reinterpret_cast<cudaStream_t>(uintptr_t(16 + 16 * t));
        for (int i = 0; i < 60; ++i) {
            const size_t n = 100000 + 61111u * ((i * 7 + t) % 50) + i;  // 0.1 to 3 MB, odd
            std::vector<char> src(n), d(n), back(n, 0);
            for (size_t x = 0; x < n; ++x) src[x] = (char)(x * 31 + x / 4096 + i * 5 + t);
            const std::vector<char> want = src;
            if (stage_h2d(&ctx, d.data(), src.data(), n, s) != BN_OK) bad[t] = 3;
            memset(src.data(), 0x5a, n);
            if (stage_d2h(&ctx, back.data(), d.data(), n, s) != BN_OK) bad[t] = 4;
            if (back != want) bad[t] = 5;
        }
        fake::streamSynchronize(s);
    };
    std::thread a(work, 0), b(work, 1);
    a.join();
    b.join();
    // a pinned array is not staged; its copy is in the stream's order
    char* pin = nullptr;
    fake::mallocHost(reinterpret_cast<void**>(&pin), 1u << 20);
    memset(pin, 7, 1u << 20);
    std::vector<char> d(1u << 20, 0);
    if (stage_h2d(&ctx, d.data(), pin, 1u << 20, nullptr) != BN_OK) return 6;
    fake::streamSynchronize(nullptr);
    if (d != std::vector<char>(1u << 20, 7)) return 7;
    memset(pin, 0, 1u << 20);
    if (stage_d2h(&ctx, pin, d.data(), 1u << 20, nullptr) != BN_OK || memcmp(pin, d.data(), 1u << 20)) return 8;
    return bad[0] | bad[1];
}

int main(int argc, char** argv) {
    if (argc > 1 && !strcmp(argv[1], "pinfail")) {
        fake::pin_fails = true;
        bn_ctx ctx;
        std::vector<char> src(1u << 20, 3), dev(1u << 20);
        for (int i = 0; i < 200; ++i)
            if (stage_h2d(&ctx, dev.data(), src.data(), src.size(), nullptr) != BN_OK || dev != src) return 1;
        printf("%d\n", fake::pin_calls);
        return 0;
    }
    return copies();
}
