// Transient-row storage conversion: FP32 rows to FP16 / BF16 with a per-capture scale
// (the FAST kernels multiply the volume back by that scale, bpgb_options.h_scale).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "bpgb_device.cuh"
#include "bpgb_internal.h"

namespace bpgb {
namespace {

// These passes move each byte once, so they are bound by HBM and need wide accesses in flight:
// rows are cut into pieces, one per CTA at a time and four or eight elements
// per thread, and rows that follow one another without padding are taken as one long row.
// 16,384 x 4,096 FP32 rows: absmax 137 -> 42 us, FP16 conversion 164 -> 54 us, scaling
// a 256^3 volume 29 -> 15 us (one element and a 64-bit division per thread before).
constexpr uint32_t kMaxPiece = 1u << 14, kMinPiece = 1u << 10;
constexpr uint32_t kSms = 152;

struct Rows {
    uint64_t rows, T;   // T elements each
    uint64_t pieces;    // of `piece` elements per row
    uint64_t pitch;     // of the input
    uint32_t piece;
};

// Few rows are cut finer, until every SM has two pieces (37 rows of 60,001 elements as FP16
// 13.5 -> 4.1 us); more pieces cost long rows more (6.2 M elements' largest: 6.3 us, 6.7 with eight).
Rows rows_of(uint64_t rows, uint64_t T, uint64_t pitch, bool flat) {
    if (flat) T *= rows, rows = 1, pitch = T;
    uint32_t piece = kMaxPiece;
    while (piece > kMinPiece && rows * ((T + piece - 1) / piece) < 2 * kSms) piece /= 2;
    return {rows, T, (T + piece - 1) / piece, pitch, piece};
}

unsigned blocks_for(const Rows &g) {
    const uint64_t n = g.rows * g.pieces;
    return (unsigned)(n < kSms * 16 ? n : kSms * 16);
}

// Padded rows too short to occupy a CTA each: a CTA takes `share` of them at a time as one run of
// share x width elements, whose row and place a multiplication with 2^32 / width gives (exact
// below 2^32 / width elements).  A CTA per row took 121 us for the largest of 200,000 rows of 8
// elements and 116 us for their conversion, against 12.3 and 8.2 us with one element and a
// 64-bit division per thread; 6.5 and 5.0 us now.
constexpr uint32_t kShortRow = 512;

struct ShortRows {
    uint64_t rows, units;
    uint32_t width, share, inverse;
};

ShortRows short_rows(uint64_t rows, uint32_t width) {
    // 4,096 elements a unit, fewer until every SM has eight units
    uint32_t elements = 4096;
    while (elements > 512 && rows * width < (uint64_t)elements * 8 * kSms) elements /= 2;
    const uint32_t share = elements > width ? elements / width : 1;
    return {rows, (rows + share - 1) / share, width, share, (uint32_t)((1ull << 32) / width + 1)};
}

unsigned blocks_for(const ShortRows &g) {
    return (unsigned)(g.units < kSms * 16 ? g.units : kSms * 16);
}

// f(row from the unit's first, place, element of the unit) for this thread's elements of unit q.
template <typename F>
__device__ __forceinline__ void short_elements(const ShortRows &g, uint64_t q, F &&f) {
    const uint32_t n = (uint32_t)min((uint64_t)g.share, g.rows - q * g.share) * g.width;
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < n; e += 256) {
        const uint32_t r = g.width == 1 ? e : __umulhi(e, g.inverse);
        f(r, e - r * g.width, e);
    }
}

// The CTA's largest |value| as float bits into out[0] (NaN counts as +inf).
__device__ __forceinline__ void block_max(unsigned int m, unsigned int *out) {
    m = __reduce_max_sync(0xffffffffu, m);
    __shared__ unsigned int warp_max[8];
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) m = max(m, warp_max[w]);
        atomicMax(out, min(m, 0x7f800000u));
    }
}

__global__ void __launch_bounds__(256)
    absmax_short_kernel(const float *__restrict__ in, const ShortRows g, uint32_t pitch,
                        unsigned int *__restrict__ out) {
    wait_previous();
    unsigned int m = 0;
    for (uint64_t q = blockIdx.x; q < g.units; q += gridDim.x) {
        const float *src = in + q * g.share * pitch;
        short_elements(g, q, [&](uint32_t r, uint32_t t, uint32_t) {
            m = max(m, __float_as_uint(__ldg(src + (uint64_t)r * pitch + t)) & 0x7fffffffu);
        });
    }
    block_max(m, out);
}

// out[0] = max |in| (float bits compare as unsigned for |x|; NaN counts as +inf).  VEC: rows
// start on 16-byte boundaries.
template <bool VEC>
__global__ void __launch_bounds__(256)
    absmax_kernel(const float *__restrict__ in, const Rows g, unsigned int *__restrict__ out) {
    wait_previous();
    unsigned int m = 0;
    auto take = [&](float v) { m = max(m, __float_as_uint(v) & 0x7fffffffu); };
    for (uint64_t q = blockIdx.x; q < g.rows * g.pieces; q += gridDim.x) {
        const uint64_t r = q / g.pieces, t0 = (q - r * g.pieces) * g.piece;
        const float *row = in + r * g.pitch + t0;
        const uint32_t T = (uint32_t)min((uint64_t)g.piece, g.T - t0);
        uint32_t t = 0;
        if (VEC) {
            const float4 *row4 = reinterpret_cast<const float4 *>(row);
#pragma unroll 4
            for (uint32_t i = threadIdx.x; i < T / 4; i += 256) {
                const float4 v = __ldg(row4 + i);
                take(v.x), take(v.y), take(v.z), take(v.w);
            }
            t = T / 4 * 4;
        }
        for (t += threadIdx.x; t < T; t += 256) take(row[t]);
    }
    block_max(m, out);
}

__device__ __forceinline__ uint32_t pack2(float a, float b, __half) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack2(float a, float b, __nv_bfloat16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ void store_h(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void store_h(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

// Output rows hold g.T elements, the first T of them from the input and zeros after.  Pieces
// are taken last first: a scan for the maximum just before leaves the last ones in L2.  VEC:
// input and output rows start on 16-byte boundaries.
template <typename HT, bool VEC>
__global__ void __launch_bounds__(256)
    to_half_kernel(const float *__restrict__ in, const Rows g, uint64_t T, float scale,
                   const float *__restrict__ d_absmax, float target, HT *__restrict__ out) {
    wait_previous();
    const float inv_scale = 1.0f / scale_of(scale, d_absmax, target);
    const uint64_t count = g.rows * g.pieces;
    for (uint64_t b = blockIdx.x; b < count; b += gridDim.x) {
        const uint64_t q = count - 1 - b, r = q / g.pieces, t0 = (q - r * g.pieces) * g.piece;
        const float *src = in + r * g.pitch + t0;
        HT *dst = out + r * g.T + t0;
        const uint32_t n = (uint32_t)min((uint64_t)g.piece, g.T - t0);
        const uint32_t m = t0 < T ? (uint32_t)min((uint64_t)n, T - t0) : 0u;  // from the input
        uint32_t t = 0;
        if (VEC) {
#pragma unroll 2
            for (uint32_t i = threadIdx.x; i < m / 8; i += 256) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(src) + 2 * i);
                const float4 b = __ldg(reinterpret_cast<const float4 *>(src) + 2 * i + 1);
                uint4 o;
                o.x = pack2(a.x * inv_scale, a.y * inv_scale, HT());
                o.y = pack2(a.z * inv_scale, a.w * inv_scale, HT());
                o.z = pack2(b.x * inv_scale, b.y * inv_scale, HT());
                o.w = pack2(b.z * inv_scale, b.w * inv_scale, HT());
                reinterpret_cast<uint4 *>(dst)[i] = o;
            }
            t = m / 8 * 8;
        }
#pragma unroll 4
        for (t += threadIdx.x; t < n; t += 256) store_h(dst + t, t < m ? __ldg(src + t) * inv_scale : 0.0f);
    }
}

// The same for short padded rows.
template <typename HT>
__global__ void __launch_bounds__(256)
    to_half_short_kernel(const float *__restrict__ in, const ShortRows g, uint32_t T, uint32_t pitch,
                         float scale, const float *__restrict__ d_absmax, float target,
                         HT *__restrict__ out) {
    wait_previous();
    const float inv_scale = 1.0f / scale_of(scale, d_absmax, target);
    for (uint64_t q = blockIdx.x; q < g.units; q += gridDim.x) {
        const float *src = in + q * g.share * pitch;
        HT *dst = out + q * g.share * g.width;
        short_elements(g, q, [&](uint32_t r, uint32_t t, uint32_t e) {
            store_h(dst + e, t < T ? __ldg(src + (uint64_t)r * pitch + t) * inv_scale : 0.0f);
        });
    }
}

// out[r][t] = in[r][from + t] for 0 <= from + t < T, else 0 (t < out_pitch).
__global__ void crop_kernel(const float *__restrict__ in, uint64_t rows, uint32_t T,
                            uint32_t in_pitch, int64_t from, uint32_t len,
                            float *__restrict__ out, uint32_t out_pitch) {
    const uint64_t n = rows * out_pitch;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = i / out_pitch, t = i - r * out_pitch;
        const int64_t src = from + (int64_t)t;
        out[i] = (t < len && src >= 0 && src < (int64_t)T) ? in[r * in_pitch + src] : 0.0f;
    }
}

template <bool VEC>
__global__ void __launch_bounds__(256)
    scale_kernel(float *__restrict__ v, uint64_t n, float scale,
                 const float *__restrict__ d_absmax, float target) {
    wait_previous();
    const float f = scale_of(scale, d_absmax, target);
    const uint64_t step = (uint64_t)gridDim.x * 256, at = blockIdx.x * 256ull + threadIdx.x;
    uint64_t i = at;
    if (VEC) {
        float4 *v4 = reinterpret_cast<float4 *>(v);
#pragma unroll 4
        for (uint64_t k = at; k < n / 4; k += step) {
            float4 x = v4[k];
            x.x *= f, x.y *= f, x.z *= f, x.w *= f;
            v4[k] = x;
        }
        i += n / 4 * 4;
    }
    for (; i < n; i += step) v[i] *= f;
}

bool aligned16(const void *p) { return (uintptr_t)p % 16 == 0; }

}  // namespace
}  // namespace bpgb

using namespace bpgb;

extern "C" {

int bpgb_rows_absmax(const float *d_H, uint64_t rows, uint32_t T, uint32_t pitch,
                     float *d_max, void *stream) {
    clear_error();
    if (!d_H || !d_max || T == 0 || pitch < T)
        return set_error(BPGB_ERR_INVALID_ARGUMENT, "bad absmax arguments");
    cudaStream_t s = (cudaStream_t)stream;
    BPGB_CUDA_TRY(cudaMemsetAsync(d_max, 0, sizeof(float), s));
    const uint64_t n = rows * T;
    if (n == 0) return BPGB_OK;
    if (rows > 1 && pitch != T && T <= kShortRow) {
        const ShortRows g = short_rows(rows, T);
        launch_after(absmax_short_kernel, blocks_for(g), 256, 0, s, d_H, g, pitch,
                     (unsigned int *)d_max);
        count_launches(1);
        BPGB_CUDA_TRY(cudaGetLastError());
        return BPGB_OK;
    }
    const Rows g = rows_of(rows, T, pitch, pitch == T);
    if (aligned16(d_H) && (g.rows == 1 || pitch % 4 == 0))
        launch_after(absmax_kernel<true>, blocks_for(g), 256, 0, s, d_H, g, (unsigned int *)d_max);
    else
        launch_after(absmax_kernel<false>, blocks_for(g), 256, 0, s, d_H, g, (unsigned int *)d_max);
    count_launches(1);
    BPGB_CUDA_TRY(cudaGetLastError());
    return BPGB_OK;
}

int bpgb_rows_to_half(const float *d_H, uint64_t rows, uint32_t T, uint32_t in_pitch, float scale,
                      const float *d_absmax, float target, int dtype, void *d_out,
                      uint32_t out_pitch, void *stream) {
    clear_error();
    if (!d_H || !d_out || T == 0 || in_pitch < T || out_pitch < T ||
        (d_absmax ? !(target > 0.0f) : !(scale > 0.0f)) ||
        (dtype != BPGB_DTYPE_F16 && dtype != BPGB_DTYPE_BF16))
        return set_error(BPGB_ERR_INVALID_ARGUMENT, "bad row conversion arguments");
    const uint64_t n = rows * out_pitch;
    if (n == 0) return BPGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const bool flat = in_pitch == T && out_pitch == T;
    if (rows > 1 && !flat && out_pitch <= kShortRow) {
        const ShortRows g = short_rows(rows, out_pitch);
        auto run = [&](auto kernel, auto *out) {
            launch_after(kernel, blocks_for(g), 256, 0, s, d_H, g, T, in_pitch, scale, d_absmax, target,
                         out);
        };
        dtype == BPGB_DTYPE_F16 ? run(to_half_short_kernel<__half>, (__half *)d_out)
                                : run(to_half_short_kernel<__nv_bfloat16>, (__nv_bfloat16 *)d_out);
        count_launches(1);
        BPGB_CUDA_TRY(cudaGetLastError());
        return BPGB_OK;
    }
    const Rows g = rows_of(rows, out_pitch, in_pitch, flat);
    const bool vec = aligned16(d_H) && aligned16(d_out) &&
                     (g.rows == 1 || (in_pitch % 4 == 0 && out_pitch % 8 == 0));
    auto run = [&](auto kernel, auto *out) {
        launch_after(kernel, blocks_for(g), 256, 0, s, d_H, g, flat ? g.T : T, scale, d_absmax, target,
                     out);
    };
    if (dtype == BPGB_DTYPE_F16)
        vec ? run(to_half_kernel<__half, true>, (__half *)d_out)
            : run(to_half_kernel<__half, false>, (__half *)d_out);
    else
        vec ? run(to_half_kernel<__nv_bfloat16, true>, (__nv_bfloat16 *)d_out)
            : run(to_half_kernel<__nv_bfloat16, false>, (__nv_bfloat16 *)d_out);
    count_launches(1);
    BPGB_CUDA_TRY(cudaGetLastError());
    return BPGB_OK;
}

int bpgb_volume_scale(float *d_volume, uint64_t n, float scale, const float *d_absmax,
                      float target, void *stream) {
    clear_error();
    if (!d_volume || (d_absmax ? !(target > 0.0f) : !(scale == scale)))
        return set_error(BPGB_ERR_INVALID_ARGUMENT, "bad volume scale arguments");
    if (n == 0) return BPGB_OK;
    const uint64_t want = (n + 1023) / 1024;
    const unsigned grid = (unsigned)(want < 152 * 16 ? want : 152 * 16);
    cudaStream_t s = (cudaStream_t)stream;
    if (aligned16(d_volume))
        launch_after(scale_kernel<true>, grid, 256, 0, s, d_volume, n, scale, d_absmax, target);
    else
        launch_after(scale_kernel<false>, grid, 256, 0, s, d_volume, n, scale, d_absmax, target);
    count_launches(1);
    BPGB_CUDA_TRY(cudaGetLastError());
    return BPGB_OK;
}

int bpgb_rows_crop(const float *d_in, uint64_t rows, uint32_t T, uint32_t in_pitch, int64_t from,
                   uint32_t len, float *d_out, uint32_t out_pitch, void *stream) {
    clear_error();
    if (!d_in || !d_out || T == 0 || in_pitch < T || len == 0 || out_pitch < len)
        return set_error(BPGB_ERR_INVALID_ARGUMENT, "bad crop arguments");
    const uint64_t n = rows * out_pitch;
    if (n == 0) return BPGB_OK;
    const unsigned grid = (unsigned)((n + 255) / 256 < 152 * 16 ? (n + 255) / 256 : 152 * 16);
    crop_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(d_in, rows, T, in_pitch, from, len, d_out,
                                                      out_pitch);
    count_launches(1);
    BPGB_CUDA_TRY(cudaGetLastError());
    return BPGB_OK;
}

}  // extern "C"
