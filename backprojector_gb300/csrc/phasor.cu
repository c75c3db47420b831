// Phasor-field pulse convolution (bp::phasor_pulse, backproject.hpp:430-479) on the GPU.
//
// out[r, t] = sum_{k=0}^{K-1} H[r, t + k - K/2] * (cos_k, sin_k) over read indices in
// (0, T) (index 0 is excluded, :468).  The sum runs in tap order with a separate FP32
// multiply and add per tap, as the reference's loop does, so the result matches a CPU
// evaluation of that loop bit for bit.
//
// Bound: the FP32 pipe and issue, two multiplies and two adds per output and tap (fused or
// reordered sums would change bits).  A thread owns 8 consecutive outputs, so each row value,
// loaded once into a register, serves the 8 outputs as the taps slide over it: 33 issue slots
// per tap and 8 outputs, where strided outputs, each with its own load, took 41.  Each CTA
// stages one row segment plus its halo in shared memory (zeros outside (0, T), which
// reproduces the index test), groups of 8 values 48 bytes apart so that the lanes' 16-byte
// loads hit distinct banks.  Measured on 16,384 rows of 4,096 bins and 503 taps: 4.79 ms
// with strided outputs, 3.96 with a window of registers, 3.87 with one for the last K mod 8 taps
// too (3.4 ms at 128 FP32 results per SM and clock; 71 taps 0.768 -> 0.627 ms).  Packed FP32x2 sums
// measured 4.12 ms; packed products are fused with packed sums whatever their rounding
// modifiers, which changes bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "bpgb_device.cuh"
#include "bpgb_internal.h"

namespace bpgb {
namespace {

constexpr int kPer = 8;              // consecutive outputs per thread
constexpr int kMaxThreads = 128;
constexpr int kSeg = kMaxThreads * kPer;
constexpr int kTapBlock = 512;       // taps staged at a time, a multiple of kPer
constexpr int kGroupWords = kPer + 4;  // a staged group of 8 values, padded

// Threads of a CTA (8 outputs each) and segments of a row: T split evenly over as few
// segments as kSeg allows.
struct PulseShape {
    uint32_t nseg, threads;
    uint32_t smem;
};

PulseShape pulse_shape(uint32_t T, int K) {
    PulseShape p;
    p.nseg = (T + kSeg - 1) / kSeg;
    const uint32_t per = (T + p.nseg - 1) / p.nseg;
    p.threads = ((per + kPer - 1) / kPer + 31) / 32 * 32;
    const int kt = std::min(K, kTapBlock);
    const uint32_t groups = p.threads + (kt + kPer - 1) / kPer + 2;
    p.smem = (groups * kGroupWords + 2 * (kt + 1)) * sizeof(float);
    return p;
}

// acc += x * c, products and sums rounded separately.
__device__ __forceinline__ void mul_add(float2 &acc, float x, float2 c) {
    acc.x = __fadd_rn(acc.x, __fmul_rn(x, c.x));
    acc.y = __fadd_rn(acc.y, __fmul_rn(x, c.y));
}

// REST: K is not a multiple of kPer.
template <bool REST>
__global__ void __launch_bounds__(kMaxThreads)
    phasor_pulse_kernel(const float *__restrict__ H, uint32_t T, uint32_t in_pitch,
                        const float2 *__restrict__ taps, int K, float2 *__restrict__ out,
                        uint32_t out_pitch, uint32_t nseg, int vec) {
    extern __shared__ __align__(16) float sm[];
    wait_previous();
    const int groups = blockDim.x + (min(K, kTapBlock) + kPer - 1) / kPer + 2;
    float4 *tp4 = reinterpret_cast<float4 *>(sm + (size_t)groups * kGroupWords);
    float2 *tp = reinterpret_cast<float2 *>(tp4);
    const uint64_t r = blockIdx.x / nseg;
    const uint32_t sg = blockIdx.x % nseg;
    const int64_t t_begin = (int64_t)sg * blockDim.x * kPer;
    const float *row = H + r * in_pitch;
    auto load_group = [&](int g, float (&x)[kPer]) {
        const float4 *p = reinterpret_cast<const float4 *>(sm + (size_t)g * kGroupWords);
        const float4 a = p[0], b = p[1];
        x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
        x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    };
    float2 acc[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) acc[j] = make_float2(0.0f, 0.0f);
    for (int k0 = 0; k0 < K; k0 += kTapBlock) {
        const int kt = min(K - k0, kTapBlock);
        if (k0 > 0) __syncthreads();
        for (int i = threadIdx.x; i < groups * kPer; i += blockDim.x) {
            const int64_t ri = t_begin - K / 2 + k0 + i;
            const float v = (ri > 0 && ri < (int64_t)T) ? row[ri] : 0.0f;
            sm[(i / kPer) * kGroupWords + i % kPer] = v;
        }
        for (int k = threadIdx.x; k < kt; k += blockDim.x) tp[k] = taps[k0 + k];
        __syncthreads();
        float x0[kPer], x1[kPer];
        load_group(threadIdx.x, x0);
        const int full = kt / kPer;
#pragma unroll 2
        for (int kb = 0; kb < full; kb++) {
            load_group(threadIdx.x + kb + 1, x1);
#pragma unroll
            for (int u = 0; u < kPer; u += 2) {
                const float4 c = tp4[(kb * kPer + u) / 2];
#pragma unroll
                for (int j = 0; j < kPer; j++)
                    mul_add(acc[j], u + j < kPer ? x0[u + j] : x1[u + j - kPer],
                            make_float2(c.x, c.y));
#pragma unroll
                for (int j = 0; j < kPer; j++)
                    mul_add(acc[j], u + 1 + j < kPer ? x0[u + 1 + j] : x1[u + 1 + j - kPer],
                            make_float2(c.z, c.w));
            }
#pragma unroll
            for (int j = 0; j < kPer; j++) x0[j] = x1[j];
        }
        if (!REST) continue;
        const int rest = kt - full * kPer;  // the last K mod 8 taps
        if (rest) load_group(threadIdx.x + full + 1, x1);
#pragma unroll
        for (int u = 0; u < kPer - 1; u++) {
            if (u >= rest) break;
            const float2 c = tp[full * kPer + u];
#pragma unroll
            for (int j = 0; j < kPer; j++)
                mul_add(acc[j], u + j < kPer ? x0[u + j] : x1[u + j - kPer], c);
        }
    }
    const int64_t t = t_begin + threadIdx.x * kPer;
    float2 *o = out + r * out_pitch + t;
    if (vec && t + kPer <= (int64_t)T) {
#pragma unroll
        for (int j = 0; j < kPer / 2; j++)
            reinterpret_cast<float4 *>(o)[j] =
                make_float4(acc[2 * j].x, acc[2 * j].y, acc[2 * j + 1].x, acc[2 * j + 1].y);
    } else {
#pragma unroll
        for (int j = 0; j < kPer; j++)
            if (t + j < (int64_t)T) o[j] = acc[j];
    }
}

// Few taps (K < kFewTaps): bound by the rows' and the field's bytes, so outputs strided by the
// block, whose loads and stores are contiguous across a warp and need little preparation.
// 16,384 x 4,096, this kernel against the one above: 3 taps 124 / 192 us, 15 211 / 240, 28 321 / 331, 31
// 354 / 348.  The block's size is a template argument (8 taps 155 us, 181 without).
constexpr int kFewTaps = 31;
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
    phasor_few_taps_kernel(const float *__restrict__ H, uint32_t T, uint32_t in_pitch,
                           const float2 *__restrict__ taps, int K, float2 *__restrict__ out,
                           uint32_t out_pitch, uint32_t nseg) {
    __shared__ float seg[THREADS * kPer + kFewTaps];
    __shared__ float2 tp[kFewTaps];
    wait_previous();
    const uint64_t r = blockIdx.x / nseg;
    const int64_t t_begin = (int64_t)(blockIdx.x % nseg) * THREADS * kPer;
    const float *row = H + r * in_pitch;
    for (int i = threadIdx.x; i < THREADS * kPer + K; i += THREADS) {
        const int64_t ri = t_begin - K / 2 + i;
        seg[i] = (ri > 0 && ri < (int64_t)T) ? row[ri] : 0.0f;
    }
    for (int k = threadIdx.x; k < K; k += THREADS) tp[k] = taps[k];
    __syncthreads();
    float2 acc[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) acc[j] = make_float2(0.0f, 0.0f);
    for (int k = 0; k < K; k++) {
        const float2 c = tp[k];
#pragma unroll
        for (int j = 0; j < kPer; j++) mul_add(acc[j], seg[threadIdx.x + j * THREADS + k], c);
    }
    float2 *orow = out + r * out_pitch;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        const int64_t t = t_begin + threadIdx.x + j * THREADS;
        if (t < (int64_t)T) orow[t] = acc[j];
    }
}

}  // namespace

// Device copies of pulse taps, one per (taps, device), kept for the process: the
// reconstruction path then neither allocates nor synchronises per call.
int device_taps(const float *h_taps, int K, const float2 **out) {
    static std::mutex mu;
    struct Entry {
        int dev;
        std::vector<float2> taps;
        float2 *d;
    };
    static std::vector<Entry> cache;
    int dev = 0;
    BPGB_CUDA_TRY(cudaGetDevice(&dev));
    std::vector<float2> tp(K);
    for (int k = 0; k < K; k++) tp[k] = make_float2(h_taps[k], h_taps[K + k]);
    std::lock_guard<std::mutex> lock(mu);
    for (const Entry &e : cache)
        if (e.dev == dev && e.taps.size() == tp.size() &&
            std::memcmp(e.taps.data(), tp.data(), tp.size() * sizeof(float2)) == 0) {
            *out = e.d;
            return BPGB_OK;
        }
    float2 *d = nullptr;
    BPGB_CUDA_TRY(cudaMalloc(&d, K * sizeof(float2)));
    cudaError_t e = cudaMemcpy(d, tp.data(), K * sizeof(float2), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        return cuda_error(e, "phasor taps upload");
    }
    cache.push_back({dev, std::move(tp), d});
    *out = d;
    return BPGB_OK;
}

int launch_phasor_pulse(const float *d_H, uint64_t rows, uint32_t T, uint32_t in_pitch,
                        const float *h_taps, int K, float *d_out, uint32_t out_pitch,
                        cudaStream_t stream) {
    if (rows == 0 || T == 0) return BPGB_OK;
    if (K <= 0) {
        BPGB_CUDA_TRY(cudaMemset2DAsync(d_out, (size_t)out_pitch * 8, 0, (size_t)T * 8, rows, stream));
        return BPGB_OK;
    }
    const PulseShape p = pulse_shape(T, K);
    // the limit of callers' pulses (about 16,700 taps), not of these kernels
    if ((size_t)(((kSeg + K + 1) & ~1) + 2 * K) * sizeof(float) > 200 * 1024)
        return set_error(BPGB_ERR_UNSUPPORTED, "phasor pulse too long");
    const uint64_t blocks = rows * p.nseg;
    if (blocks >= (1ull << 31)) return set_error(BPGB_ERR_UNSUPPORTED, "too many rows for one launch");
    const float2 *d_taps = nullptr;
    if (int st = device_taps(h_taps, K, &d_taps)) return st;
    if (K < kFewTaps) {
        const auto few = p.threads == 32  ? phasor_few_taps_kernel<32>
                         : p.threads == 64 ? phasor_few_taps_kernel<64>
                         : p.threads == 96 ? phasor_few_taps_kernel<96>
                                           : phasor_few_taps_kernel<128>;
        launch_after(few, (unsigned)blocks, p.threads, 0, stream, d_H, T, in_pitch,
                     d_taps, K, reinterpret_cast<float2 *>(d_out), out_pitch, p.nseg);
        count_launches(1);
        BPGB_CUDA_TRY(cudaGetLastError());
        return BPGB_OK;
    }
    const auto kernel = K % kPer ? phasor_pulse_kernel<true> : phasor_pulse_kernel<false>;
    if (int rs = reserve_dynamic_smem((const void *)kernel, p.smem)) return rs;
    // 16-byte stores where every row's outputs are 16-byte aligned
    const int vec = ((uintptr_t)d_out % 16 == 0 && out_pitch % 2 == 0) ? 1 : 0;
    launch_after(kernel, (unsigned)blocks, p.threads, p.smem, stream, d_H, T, in_pitch,
                 d_taps, K, reinterpret_cast<float2 *>(d_out), out_pitch, p.nseg, vec);
    count_launches(1);
    BPGB_CUDA_TRY(cudaGetLastError());
    return BPGB_OK;
}

}  // namespace bpgb

extern "C" {

int bpgb_phasor_taps(float wavelength, float deltaT, uint32_t times, float *taps, int cap) {
    // Reference construction (backproject.hpp:433-451): K = int(times*wl/dT),
    // C = int(wl/dT), sigma = times*wl/6; t_k = dT*(k - K/2.0) for k = 1..K; Gaussian
    // exp(-t^2 / (2 sigma^2)) in double with 2*sigma*sigma an FP32 product; phase
    // 2*pi*(k/C); cos/sin rounded to FP32, times the Gaussian in double, rounded to FP32.
    const int K = (int)((float)times * wavelength / deltaT);
    const int C = (int)(wavelength / deltaT);
    if (K <= 0 || C <= 0 || !taps || cap < K) return K;
    const float vsigma = ((float)times * wavelength) / 6.0f;
    const double denom = (double)(2.0f * vsigma * vsigma);
    for (int k = 0; k < K; k++) {
        const double kk = (double)(k + 1);
        const double t = (double)deltaT * (kk - K / 2.0);
        const double g = std::exp(-t * t / denom);
        const double prog = 2.0 * M_PI * (1.0 / C * kk);
        const float s = (float)std::sin(prog);
        const float c = (float)std::cos(prog);
        taps[k] = (float)((double)c * g);
        taps[K + k] = (float)((double)s * g);
    }
    return K;
}

int bpgb_phasor_pulse(const float *d_H, uint64_t rows, uint32_t T, uint32_t in_pitch,
                      float wavelength, float deltaT, uint32_t times, float *d_out,
                      uint32_t out_pitch, void *stream) {
    bpgb::clear_error();
    if ((rows && (!d_H || !d_out)) || in_pitch < T || out_pitch < T)
        return bpgb::set_error(BPGB_ERR_INVALID_ARGUMENT, "bad phasor pulse arguments");
    if (!(deltaT > 0.0f) || !(wavelength > 0.0f))
        return bpgb::set_error(BPGB_ERR_INVALID_ARGUMENT, "wavelength and deltaT must be > 0");
    int st = bpgb::require_device();
    if (st) return st;
    const int K = bpgb_phasor_taps(wavelength, deltaT, times, nullptr, 0);
    std::vector<float> taps(K > 0 ? 2 * (size_t)K : 1);
    if (K > 0) bpgb_phasor_taps(wavelength, deltaT, times, taps.data(), K);
    return bpgb::launch_phasor_pulse(d_H, rows, T, in_pitch, taps.data(), K, d_out, out_pitch,
                                     (cudaStream_t)stream);
}

}  // extern "C"
