// The per-thread caches of the host-buffer calls (host_cache.h) against a fake CUDA runtime of two
// devices: a buffer or plan made on one device is never handed out on the other; and when a capture
// is uploaded in parts.  Exit status 0
// when every check holds; the line of the first that fails otherwise.
#include <cstdlib>
#include <map>

#include "host_cache.h"

static int current = 0, plans_destroyed = 0;
static std::map<void *, int> owner;  // allocation -> device

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = current, cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = std::malloc(n);
    owner[*p] = current;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    owner.erase(p);
    std::free(p);
    return cudaSuccess;
}
int bpgb_plan_destroy(bpgb_plan) { return plans_destroyed++, BPGB_OK; }
}
namespace bpgb {
int cuda_error(cudaError_t, const char *) { return BPGB_ERR_CUDA; }
}  // namespace bpgb

#define CHECK(x) \
    if (!(x)) return __LINE__ % 256

int main() {
    using namespace bpgb;
    DeviceBuffer b;
    CHECK(b.reserve(64) == BPGB_OK && owner.at(b.ptr) == 0);
    void *first = b.ptr;
    CHECK(b.reserve(32) == BPGB_OK && b.ptr == first);  // grow-only
    current = 1;
    CHECK(b.reserve(32) == BPGB_OK && owner.at(b.ptr) == 1);
    CHECK(owner.size() == 1);  // the other device's memory is given back
    CHECK(b.reserve(128) == BPGB_OK && owner.at(b.ptr) == 1 && b.bytes == 128);
    current = 0;
    CHECK(b.reserve(128) == BPGB_OK && owner.at(b.ptr) == 0);

    HostPlanCache cache;
    bpgb_pair pairs[2] = {};
    const uint32_t n[3] = {4, 5, 6};
    bpgb_options o{};
    const auto plan = reinterpret_cast<bpgb_plan>(&o);
    cache.keep(plan, 0, pairs, 2, 8, n, nullptr, nullptr, 1.0f, 0.5f, o);
    CHECK(cache.find(0, pairs, 2, 8, n, nullptr, nullptr, 1.0f, 0.5f, o) == plan);
    CHECK(cache.find(1, pairs, 2, 8, n, nullptr, nullptr, 1.0f, 0.5f, o) == nullptr);
    CHECK(cache.find(0, pairs, 2, 9, n, nullptr, nullptr, 1.0f, 0.5f, o) == nullptr);
    cache.clear();
    CHECK(plans_destroyed == 1);

    // One copy where parts hide less than they cost, measured at these bytes and updates; at most
    // the parts that a plan has.
    const uint64_t mb = 1 << 20;
    CHECK(host_parts(false, 4 * mb, 1024ull * 32 * 32 * 32, 4) == 1);
    CHECK(host_parts(true, 4 * mb, 1024ull * 32 * 32 * 32, 4) == 1);
    CHECK(host_parts(false, 128 * mb, 16384ull * 8 * 8 * 8, 4) == 1);
    CHECK(host_parts(true, 128 * mb, 16384ull * 8 * 8 * 8, 4) == 1);
    CHECK(host_parts(false, 2 * mb, 576ull * 200 * 200 * 200, 4) == 1);
    CHECK(host_parts(false, 32 * mb, 4096ull * 64 * 64 * 64, 4) == 4);
    CHECK(host_parts(false, 32 * mb, 4096ull * 64 * 64 * 64, 2) == 2);
    CHECK(host_parts(false, 32 * mb, 4096ull * 64 * 64 * 64, 1) == 1);
    CHECK(host_parts(true, 32 * mb, 4096ull * 32 * 32 * 32, 4) == 4);
    CHECK(host_parts(false, 32 * mb, 4096ull * 32 * 32 * 32, 4) == 1);
    CHECK(host_parts(false, 8 * mb, 4096ull * 96 * 96 * 96, 4) == 4);
    return 0;
}
