// allow_smem with stand-ins for the two runtime calls: the limit is raised once
// on every device a kernel is launched on, again after a failure, and by each
// of several threads that come to a device first at most once too often.
#include <stdio.h>

#include <atomic>
#include <thread>
#include <vector>

#include "../../ltpmg_gb300/csrc/ltp_smem.h"

static thread_local int device = 0;
static std::atomic<int> raised[100];
static std::atomic<bool> fail{false};

extern "C" cudaError_t cudaGetDevice(int *d) {
    *d = device;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
    if (fail) return cudaErrorInvalidValue;
    if (f == nullptr || a != cudaFuncAttributeMaxDynamicSharedMemorySize || v != 65536) return cudaErrorUnknown;
    raised[device]++;
    return cudaSuccess;
}

static void kernel(int) {}

#define CHECK(x)                                \
    if (!(x)) {                                 \
        printf("line %d: %s\n", __LINE__, #x);  \
        return 1;                               \
    }

int main() {
    std::atomic<uint64_t> done{0}, other{0};
    fail = true;
    CHECK(ltp::allow_smem(kernel, 65536, done) == cudaErrorInvalidValue);
    fail = false;
    for (int round = 0; round < 3; round++)
        for (device = 0; device < 64; device++) CHECK(ltp::allow_smem(kernel, 65536, done) == cudaSuccess);
    for (int d = 0; d < 64; d++) CHECK(raised[d] == 1);
    device = 70;
    CHECK(ltp::allow_smem(kernel, 65536, done) == cudaSuccess && ltp::allow_smem(kernel, 65536, done) == cudaSuccess);
    CHECK(raised[70] == 2 && raised[6] == 1);
    std::vector<std::thread> t;
    std::atomic<int> bad{0};
    for (int k = 0; k < 8; k++)
        t.emplace_back([&]() {
            for (device = 0; device < 64; device++)
                if (ltp::allow_smem(kernel, 65536, other) != cudaSuccess) bad++;
        });
    for (auto &x : t) x.join();
    CHECK(bad == 0 && other == ~0ull);
    for (int d = 0; d < 64; d++) CHECK(raised[d] >= 2 && raised[d] <= 9);
    puts("ok");
    return 0;
}
