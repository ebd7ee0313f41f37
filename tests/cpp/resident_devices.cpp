// The per-device launch facts of vs_resident.h against a runtime of two
// devices made here: each device gets its own values and its own opt-in to
// large shared memory, whatever the order and the number of threads.
#include "vs_resident.h"

#include <cstdio>
#include <thread>
#include <vector>

namespace {
thread_local int t_dev = 0;
std::atomic<int> g_set[2];
const int kSms[2] = {148, 132}, kPerSm[2] = {5, 3};
int fail(const char *what) {
    std::printf("FAIL %s\n", what);
    return 1;
}
void kernel_a(int) {}
void kernel_b(int) {}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) {
    *d = t_dev;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int dev) {
    if (a != cudaDevAttrMultiProcessorCount || dev < 0 || dev > 1) return cudaErrorInvalidValue;
    *v = kSms[dev];
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int threads, size_t) {
    *n = kPerSm[t_dev] * 128 / threads;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int threads, size_t b, unsigned) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, threads, b);
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) {
    ++g_set[t_dev];
    return cudaSuccess;
}
}

int main() {
    std::atomic<int> bad{0};
    std::vector<std::thread> threads;
    for (int k = 0; k < 8; ++k)
        threads.emplace_back([&, k] {
            for (int i = 0; i < 2000; ++i) {
                t_dev = (k + i) & 1;
                unsigned a = 0, b = 0;
                int sms = 0;
                if (vs::device_sms(&sms) != cudaSuccess || sms != kSms[t_dev]) ++bad;
                if (vs::resident_blocks<kernel_a>(&a) != cudaSuccess || a != unsigned(kSms[t_dev] * kPerSm[t_dev])) ++bad;
                if (vs::resident_blocks<kernel_b>(&b, 64) != cudaSuccess || b != unsigned(kSms[t_dev] * kPerSm[t_dev] * 2)) ++bad;
                if (vs::allow_shared<kernel_a>(200000) != cudaSuccess || g_set[t_dev].load() == 0) ++bad;
            }
        });
    for (std::thread &t : threads) t.join();
    if (bad.load()) return fail("values of another device");
    t_dev = vs::kMaxDevices;
    unsigned g = 0;
    int sms = 0;
    if (vs::resident_blocks<kernel_a>(&g) != cudaErrorInvalidDevice || vs::device_sms(&sms) != cudaErrorInvalidDevice)
        return fail("a device outside the tables");
    std::printf("ok\n");
    return 0;
}
