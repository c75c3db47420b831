// What the host-buffer entry points keep between calls, per thread: device buffers and the last
// geometry's plan.  Both belong to the device they were made on.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <vector>

#include "bpgb_internal.h"

namespace bpgb {

// A grow-only buffer on the current device, reused across calls (avoids cudaMalloc per call).
struct DeviceBuffer {
    void *ptr = nullptr;
    size_t bytes = 0;
    int device = -1;

    int reserve(size_t need) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
        if (dev == device && need <= bytes) return BPGB_OK;
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
        e = cudaMalloc(&ptr, need);
        if (e != cudaSuccess) {
            ptr = nullptr;
            return cuda_error(e, "cudaMalloc");
        }
        bytes = need;
        device = dev;
        return BPGB_OK;
    }
    ~DeviceBuffer() {
        // Process teardown may run after the CUDA context is gone; freeing then is harmless.
        if (ptr) cudaFree(ptr);
    }
};

// The host drop-in call's plan of the last geometry it saw, keyed by the device and
// every input the plan depends on (the pairs compared byte for byte).
struct HostPlanCache {
    bpgb_plan plan = nullptr;
    std::vector<bpgb_pair> pairs;
    std::vector<unsigned char> key;

    static std::vector<unsigned char> make_key(int device, uint64_t num_pairs, uint32_t T,
                                               const uint32_t *n, const float *zero,
                                               const float *inc, float t0, float deltaT,
                                               const bpgb_options &o) {
        std::vector<unsigned char> k;
        auto put = [&](const void *p, size_t b) {
            const unsigned char *c = (const unsigned char *)p;
            k.insert(k.end(), c, c + b);
        };
        const float none[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        put(&device, sizeof device);
        put(&num_pairs, sizeof num_pairs);
        put(&T, sizeof T);
        put(n, 3 * sizeof(uint32_t));
        put(zero ? zero : none, 3 * sizeof(float));
        put(inc ? inc : none, 9 * sizeof(float));
        put(&t0, sizeof t0);
        put(&deltaT, sizeof deltaT);
        put(&o, sizeof o);
        return k;
    }
    bpgb_plan find(int device, const bpgb_pair *p, uint64_t np, uint32_t T, const uint32_t *n,
                   const float *zero, const float *inc, float t0, float deltaT,
                   const bpgb_options &o) const {
        if (!plan || pairs.size() != np) return nullptr;
        if (make_key(device, np, T, n, zero, inc, t0, deltaT, o) != key) return nullptr;
        if (np && std::memcmp(pairs.data(), p, np * sizeof(bpgb_pair)) != 0) return nullptr;
        return plan;
    }
    void keep(bpgb_plan pl, int device, const bpgb_pair *p, uint64_t np, uint32_t T,
              const uint32_t *n, const float *zero, const float *inc, float t0, float deltaT,
              const bpgb_options &o) {
        plan = pl;
        pairs.assign(p, p + np);
        key = make_key(device, np, T, n, zero, inc, t0, deltaT, o);
    }
    void clear() {
        if (plan) bpgb_plan_destroy(plan);
        plan = nullptr;
        pairs.clear();
        key.clear();
    }
    ~HostPlanCache() { clear(); }
};

// Parts (of at most `most`) in which a host call uploads its rows, the pair splits of each running
// while the next one is copied.  Hidden is the shorter of upload (170 GB/s) and pass (3.6 x 10^12
// updates/s), less the last part of it; each further copy and launch costs, from pageable memory about
// 45 us in all, from pinned 10.  Measured at 2 to 128 MB into 8^3 to 96^3 voxels, single copy / four
// parts in us: pageable 4 MB 32^3 105 / 144, 8 MB 64^3 421 / 420, 16 MB 32^3 211 / 224,
// 48^3 307 / 254, 32 MB 64^3 577 / 506, 64 MB 40^3 588 / 600, 48^3 624 / 571; pinned 8 MB 16^3
// 116 / 125, 48^3 244 / 241, 32 MB 32^3 275 / 263, 64^3 538 / 458.  From 2 x 10^9 updates on the cost
// is under 1%.
inline uint32_t host_parts(bool pinned, uint64_t bytes, uint64_t updates, uint32_t most) {
    const bool hides = pinned ? bytes >= 8000000 && updates >= 100000000
                              : bytes >= 11000000 && updates >= 300000000;
    return hides || (bytes >= 4000000 && updates >= 2000000000) ? most : 1;
}

}  // namespace bpgb
