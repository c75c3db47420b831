// Reference-exact dense backprojection (FP32 and complex64).
//
// Semantics of cuda_backprojection_impl<FT> (backproject_cuda.cu:117-175): for every
// voxel v = zero + inc[0:3]*x + inc[3:6]*y + inc[6:9]*z (:144-148) and every pair p,
//   d = laser_wall + |l_p - v| + |v - c_p| + camera_wall        (:31-46, norm3df)
//   b = (int) round((d - t0 - 0) / deltaT)                       (:155-158)
// and H[p, b] is added when 0 <= b <= T-1 (:157-159).  The arithmetic below is the same
// expression in the same order (FMA-contracted voxel position, norm3df, IEEE division,
// round-half-away), so every bin index equals the reference's; only the summation order
// differs (register sums of a group's updates in pair order, then its marked updates, then the
// pair splits, instead of strided partial sums plus a serial shared-memory reduction).  This file
// must be compiled without fast-math flags.
//
// Evaluating that expression costs about 100 instructions per update (two norm3df, an
// IEEE divide, roundf), and the reference's result is needed to the last bit only where the
// quotient lies near a half-integer.  So each update first takes a cheap quotient x (two
// approximate roots, one FMA with 1 / deltaT) whose distance from the reference's quotient
// is at most E (exact_filter bounds it over the plan's pairs and voxels from the roundings
// of both expressions).  Where x is further than E from every half-integer, round(x) is the
// reference's bin; the other updates (about 2 E of them) are marked in a bit mask per
// thread and evaluated with the reference's expression after each group of 64 pairs, one
// marked pair per lane at a time, so that a warp spends one evaluation on the marks of all
// its lanes.  Where E is no use (scales where the bound does not hold, E = 0.5, or small launches that
// would wait for their marks) a direct kernel evaluates the expression for every update.
//
// Bound: issue (24 to 28 instructions per update, the marked ones' evaluations included) and the
// latency of the L1 gathers, at 70 or 72 registers and so 13 or 14 CTAs per SM (complex rows with
// range checks spill 16 bytes).  Measured on 64 x 64 pairs that do not factor, T = 2048, 64^3
// voxels: 3.60 ms before, 0.95 ms with the filter.
//
// Layout: one CTA = 64 threads = a 4 x 4 x 16 voxel tile (z fastest, x slowest), the four
// voxels of an x line per thread as two packed FP32x2 lane pairs (4 x 8 x 8: the same time at
// 64^3, 24% more at 42 x 11 x 93).  Pair records are staged 64 at a time in shared memory,
// coordinates doubled for the packed arithmetic, and read as warp-uniform broadcasts; a
// warp's 128 voxels gather from one H row at neighbouring bins, so the global gathers
// coalesce into few sectors.  Small volumes split each tile's pairs over up to 16 CTAs, whose
// partial volumes are added in pair order.  All pairs are used (the reference skips the last
// P mod blockDim) and every voxel is visited for any N.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "bpgb_device.cuh"
#include "bpgb_internal.h"

namespace bpgb {
namespace {

constexpr int kTX = 4, kTY = 4, kTZ = 16;
constexpr int kThreads = kTY * kTZ;  // each thread owns the kTX voxels of an x line
constexpr uint32_t kMaxSplits = 16;
constexpr int kGroup = 64;           // pairs staged and marked together: two mask words

struct ExactArgs {
    uint32_t n[3];
    uint32_t tiles[3];
    float zero[3];
    float inc[9];
    float t0, dT;
    uint32_t T;
    uint64_t pitch;
    uint64_t P;
    float inv;      // 1 / dT
    float thr;      // 0.5 - E: |x - round(x)| below this decides the bin
    float half;     // (T - 1) / 2: bin b is in range when |b - half| <= half
    double invd;
    uint32_t splits;  // CTAs sharing a tile, each over a contiguous range of the pairs
    uint64_t nvox;
};

__device__ __forceinline__ void voxel_position(const ExactArgs &a, uint32_t x, uint32_t y,
                                               uint32_t z, float v[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float s = __fmaf_rn(a.inc[k], (float)x, a.zero[k]);
        s = __fmaf_rn(a.inc[3 + k], (float)y, s);
        v[k] = __fmaf_rn(a.inc[6 + k], (float)z, s);
    }
}

__device__ __forceinline__ int exact_bin(const bpgb_pair &pr, const float v[3], float t0,
                                         float dT) {
    float lpv = norm3df(pr.laser_point[0] - v[0], pr.laser_point[1] - v[1],
                        pr.laser_point[2] - v[2]);
    float vcp = norm3df(v[0] - pr.camera_point[0], v[1] - pr.camera_point[1],
                        v[2] - pr.camera_point[2]);
    float total = pr.laser_wall + lpv + vcp + pr.camera_wall;
    float r = roundf((total - t0 - 0.0f / 2) / dT);
    return (int)r;
}

__device__ __forceinline__ float load_h(const float *H, uint64_t i) { return __ldg(H + i); }
__device__ __forceinline__ float2 load_h(const float2 *H, uint64_t i) { return __ldg(H + i); }
__device__ __forceinline__ void add_to(float &a, float b) { a += b; }
__device__ __forceinline__ void add_to(float2 &a, float2 b) { a = __fadd2_rn(a, b); }
template <typename HT>
__device__ __forceinline__ HT zero_h();
template <>
__device__ __forceinline__ float zero_h<float>() { return 0.0f; }
template <>
__device__ __forceinline__ float2 zero_h<float2>() { return make_float2(0.0f, 0.0f); }

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// A staged pair: (lx, lx, ly, ly), (lz, lz, cx, cx), (cy, cy, cz, cz), (c, c, lw, cw) with
// c = (lw + cw - t0) / dT rounded once from FP64.
struct Staged {
    float4 r[4];
};

__device__ __forceinline__ void stage_pair(Staged &s, const bpgb_pair &p, const ExactArgs &a) {
    const float c = (float)(((double)p.laser_wall + (double)p.camera_wall - (double)a.t0) * a.invd);
    s.r[0] = make_float4(p.laser_point[0], p.laser_point[0], p.laser_point[1], p.laser_point[1]);
    s.r[1] = make_float4(p.laser_point[2], p.laser_point[2], p.camera_point[0], p.camera_point[0]);
    s.r[2] = make_float4(p.camera_point[1], p.camera_point[1], p.camera_point[2], p.camera_point[2]);
    s.r[3] = make_float4(c, c, p.laser_wall, p.camera_wall);
}

__device__ __forceinline__ bpgb_pair staged_pair(const Staged &s) {
    bpgb_pair p;
    p.laser_point[0] = s.r[0].x, p.laser_point[1] = s.r[0].z, p.laser_point[2] = s.r[1].x;
    p.camera_point[0] = s.r[1].z, p.camera_point[1] = s.r[2].x, p.camera_point[2] = s.r[2].z;
    p.laser_wall = s.r[3].z, p.camera_wall = s.r[3].w;
    return p;
}

// |p - v| of both voxels, nv = -v.
__device__ __forceinline__ float2 legs2(float2 px, float2 py, float2 pz, const float2 nv[3]) {
    const float2 dx = __fadd2_rn(px, nv[0]), dy = __fadd2_rn(py, nv[1]), dz = __fadd2_rn(pz, nv[2]);
    const float2 s = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    return make_float2(sqrt_approx(s.x), sqrt_approx(s.y));
}

// H at the row address biased by kMagicBits and a bin as bits(bin + kMagic).
template <typename HT>
__device__ __forceinline__ HT load_at(uint64_t row, float m) {
    return __ldg(reinterpret_cast<const HT *>(row + (uint64_t)__float_as_uint(m) * sizeof(HT)));
}

// INSIDE: every bin of the plan lies in [0, T).
template <typename HT, bool INSIDE>
__global__ void __launch_bounds__(kThreads)
    bp_exact_kernel(const HT *__restrict__ H, const bpgb_pair *__restrict__ pairs,
                    HT *__restrict__ out, const ExactArgs a) {
    constexpr int NP = kTX / 2;
    wait_previous();
    allow_next();
    __shared__ Staged sp[2][kGroup];
    uint32_t t = blockIdx.x / a.splits;
    const uint32_t z = t % a.tiles[2] * kTZ + threadIdx.x % kTZ;
    t /= a.tiles[2];
    const uint32_t x = t % a.tiles[0] * kTX;
    const uint32_t y = t / a.tiles[0] * kTY + threadIdx.x / kTZ;
    // voxels past the volume's edge repeat the last one (their gathers coincide) unstored
    auto position = [&](int w, float v[3]) {
        voxel_position(a, min(x + w, a.n[0] - 1), min(y, a.n[1] - 1), min(z, a.n[2] - 1), v);
    };
    float2 nv[NP][3];
#pragma unroll
    for (int i = 0; i < NP; i++) {
        float v0[3], v1[3];
        position(2 * i, v0);
        position(2 * i + 1, v1);
#pragma unroll
        for (int k = 0; k < 3; k++) nv[i][k] = make_float2(-v0[k], -v1[k]);
    }
    HT acc[kTX];
#pragma unroll
    for (int w = 0; w < kTX; w++) acc[w] = zero_h<HT>();
    const int last = (int)a.T - 1;
    const float2 inv2 = make_float2(a.inv, a.inv), magic2 = make_float2(kMagic, kMagic);
    const float2 neg2 = make_float2(-1.0f, -1.0f);
    const float2 nmagic2 = make_float2(-kMagic, -kMagic), nhalf2 = make_float2(-a.half, -a.half);
    const uint32_t split = blockIdx.x % a.splits;
    const uint64_t p0 = a.P * split / a.splits, p1 = a.P * (split + 1) / a.splits;
    int buf = 0;
    for (uint64_t base = p0; base < p1; base += kGroup, buf ^= 1) {
        // two buffers: a warp refills one while the other warp still reads its last group
        const uint32_t n = (uint32_t)(p1 - base < (uint64_t)kGroup ? p1 - base : (uint64_t)kGroup);
        if (threadIdx.x < n) stage_pair(sp[buf][threadIdx.x], pairs[base + threadIdx.x], a);
        __syncthreads();
        const Staged *st = sp[buf];
        // Every update of pairs [j0, j1); the ones left to the reference's expression are
        // marked (bit j - j0 of the voxel's word).
        auto sweep = [&](uint32_t j0, uint32_t j1, uint32_t (&mark)[kTX]) {
            // the row's address less that of the magic number's bits: bits(m) indexes it
            uint64_t row = (uint64_t)(H + (base + j0) * a.pitch) - (uint64_t)kMagicBits * sizeof(HT);
            uint32_t bit = 1;
#pragma unroll 4
            for (uint32_t j = j0; j < j1; j++, row += a.pitch * sizeof(HT), bit <<= 1) {
                const float4 r0 = st[j].r[0], r1 = st[j].r[1], r2 = st[j].r[2];
                const float2 c2 = *reinterpret_cast<const float2 *>(&st[j].r[3]);
#pragma unroll
                for (int i = 0; i < NP; i++) {
                    const float2 l = legs2(make_float2(r0.x, r0.y), make_float2(r0.z, r0.w),
                                           make_float2(r1.x, r1.y), nv[i]);
                    const float2 s = legs2(make_float2(r1.z, r1.w), make_float2(r2.x, r2.y),
                                           make_float2(r2.z, r2.w), nv[i]);
                    const float2 q = __ffma2_rn(__fadd2_rn(l, s), inv2, c2);
                    const float2 m = __fadd2_rn(q, magic2);
                    const float2 f = __fadd2_rn(m, nmagic2);
                    const float2 d = __ffma2_rn(f, neg2, q);
                    // the reference's bin is certain (that of a NaN is not)
                    const bool ok0 = fabsf(d.x) < a.thr, ok1 = fabsf(d.y) < a.thr;
                    bool in0 = ok0, in1 = ok1;
                    if (!INSIDE) {
                        const float2 g = __fadd2_rn(f, nhalf2);
                        in0 = in0 && fabsf(g.x) <= a.half;
                        in1 = in1 && fabsf(g.y) <= a.half;
                    }
                    if (in0) add_to(acc[2 * i], load_at<HT>(row, m.x));
                    if (in1) add_to(acc[2 * i + 1], load_at<HT>(row, m.y));
                    if (!ok0) mark[2 * i] |= bit;
                    if (!ok1) mark[2 * i + 1] |= bit;
                }
            }
        };
        uint32_t mark0[kTX] = {}, mark1[kTX] = {};
        sweep(0, min(n, 32u), mark0);
        if (n > 32) sweep(32, n, mark1);
        for (;;) {  // one marked update per lane and iteration
            uint32_t m = 0, k = 0;
#pragma unroll
            for (uint32_t w = 0; w < kTX; w++) {
                if (mark0[w]) m = mark0[w], k = w;
                if (mark1[w]) m = mark1[w], k = kTX + w;
            }
            if (!m) break;
            const uint32_t w = k % kTX, j = k / kTX * 32 + __ffs((int)m) - 1;
            m &= m - 1;
            float v[3];
            position((int)w, v);
            const int b = exact_bin(staged_pair(st[j]), v, a.t0, a.dT);
            HT hv = zero_h<HT>();
            if (b >= 0 && b <= last) hv = load_h(H, (base + j) * a.pitch + (uint64_t)b);
#pragma unroll
            for (uint32_t i = 0; i < kTX; i++) {
                if (i == k) mark0[i] = m;
                if (i + kTX == k) mark1[i] = m;
                if (i == w) add_to(acc[i], hv);
            }
        }
    }
    out += split * a.nvox;  // split's partial volume (added by exact_reduce_kernel)
#pragma unroll
    for (int w = 0; w < kTX; w++)
        if (x + w < a.n[0] && y < a.n[1] && z < a.n[2])
            out[((uint64_t)(x + w) * a.n[1] + y) * a.n[2] + z] = acc[w];
}

// Plans whose cheap quotient is not trusted: the reference's expression for every update, one
// voxel of a 4 x 8 x 8 tile per thread, pairs staged 256 at a time.  Bound by issue (about 100
// instructions per update).  It doesn't call allow_next: 6.7 CTAs per SM of 64^3 voxels are
// placed unevenly around a pass's own (80 pairs, a pass among others: 77.6 us with early starts,
// 68.8 without; 63.7 with the split's first pair and row added to the pointers once).
constexpr int kDirectX = 4, kDirectY = 8, kDirectZ = 8;
constexpr int kDirectThreads = kDirectX * kDirectY * kDirectZ;
template <typename HT>
__global__ void __launch_bounds__(kDirectThreads)
    bp_exact_direct_kernel(const HT *__restrict__ H, const bpgb_pair *__restrict__ pairs,
                           HT *__restrict__ out, const ExactArgs a) {
    wait_previous();
    __shared__ bpgb_pair sp[kDirectThreads];
    uint32_t t = blockIdx.x / a.splits;
    const uint32_t z = t % a.tiles[2] * kDirectZ + threadIdx.x % kDirectZ;
    t /= a.tiles[2];
    const uint32_t x = t % a.tiles[0] * kDirectX + threadIdx.x / (kDirectZ * kDirectY);
    const uint32_t y = t / a.tiles[0] * kDirectY + threadIdx.x / kDirectZ % kDirectY;
    float v[3];
    voxel_position(a, x, y, z, v);
    HT acc = zero_h<HT>();
    const int last = (int)a.T - 1;
    const uint32_t split = blockIdx.x % a.splits;
    const uint64_t p0 = a.P * split / a.splits, P = a.P * (split + 1) / a.splits - p0;
    H += p0 * a.pitch;
    pairs += p0;
    for (uint64_t base = 0; base < P; base += kDirectThreads) {
        __syncthreads();
        if (base + threadIdx.x < P) sp[threadIdx.x] = pairs[base + threadIdx.x];
        __syncthreads();
        const uint32_t n = (uint32_t)min((uint64_t)kDirectThreads, P - base);
        for (uint32_t j = 0; j < n; j++) {
            const int b = exact_bin(sp[j], v, a.t0, a.dT);
            if (b >= 0 && b <= last) add_to(acc, load_h(H, (base + j) * a.pitch + (uint64_t)b));
        }
    }
    if (x < a.n[0] && y < a.n[1] && z < a.n[2])
        out[split * a.nvox + ((uint64_t)x * a.n[1] + y) * a.n[2] + z] = acc;
}

// out = the splits' partial sums, added in pair order.
template <typename HT>
__global__ void exact_reduce_kernel(const HT *__restrict__ partial, HT *__restrict__ out,
                                    uint64_t nvox, uint32_t splits) {
    wait_previous();
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= nvox) return;
    HT v[kMaxSplits];
#pragma unroll
    for (uint32_t k = 0; k < kMaxSplits; k++)
        v[k] = k < splits ? partial[k * nvox + i] : zero_h<HT>();
    HT s = v[0];
#pragma unroll
    for (uint32_t k = 1; k < kMaxSplits; k++)
        if (k < splits) add_to(s, v[k]);
    out[i] = s;
}

// bins[i * P + p] for voxel ids[i]; same expression as bp_exact_kernel.
__global__ void bp_exact_bins_kernel(const bpgb_pair *__restrict__ pairs,
                                     const int64_t *__restrict__ ids, int64_t n,
                                     int32_t *__restrict__ bins, const ExactArgs a) {
    const uint64_t total = (uint64_t)n * a.P;
    for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < total;
         w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = w / a.P, p = w % a.P;
        const int64_t id = ids[i];
        const uint32_t z = (uint32_t)(id % a.n[2]);
        const uint32_t y = (uint32_t)((id / a.n[2]) % a.n[1]);
        const uint32_t x = (uint32_t)(id / ((int64_t)a.n[1] * a.n[2]));
        float v[3];
        voxel_position(a, x, y, z, v);
        const bpgb_pair pr = pairs[p];
        const int b = exact_bin(pr, v, a.t0, a.dT);
        bins[w] = (b >= 0 && b <= (int)a.T - 1) ? b : -1;
    }
}

ExactArgs make_args(uint64_t pitch, uint64_t P, const Volume &vol, const BinParams &bp) {
    ExactArgs a{};
    for (int k = 0; k < 3; k++) {
        a.n[k] = vol.n[k];
        a.zero[k] = vol.zero[k];
    }
    for (int k = 0; k < 9; k++) a.inc[k] = vol.inc[k];
    a.t0 = bp.t0;
    a.dT = bp.dT;
    a.T = bp.T;
    a.pitch = pitch;
    a.P = P;
    a.splits = 1;
    a.nvox = vol.count();
    return a;
}

}  // namespace

ExactFilter exact_filter(const bpgb_pair *pairs, uint64_t P, const Volume &vol,
                         const BinParams &bp) {
    // The largest legs, path and coordinate over the plan's pairs and voxels, in FP64.  The box
    // holds the positions as the kernels round them: far from the origin they leave the box of
    // the exact corners by up to 4 u (three FMAs and the index's conversion) of the largest sum
    // on the way, which the relative error of the legs below does not cover.
    double lo[3], hi[3], size = 0.0, legs = 0.0, reach = 0.0, wall = 0.0, least = INFINITY;
    double near = INFINITY, far = -INFINITY;
    for (int k = 0; k < 3; k++) {
        lo[k] = hi[k] = vol.zero[k];
        double sum = std::fabs((double)vol.zero[k]);
        for (int a = 0; a < 3; a++) {
            const double e = (double)vol.inc[3 * a + k] * (vol.n[a] ? vol.n[a] - 1 : 0);
            (e < 0.0 ? lo[k] : hi[k]) += e;
            sum += std::fabs(e);
        }
        const double rounding = 1.01 * std::ldexp(4.0, -24) * sum;
        lo[k] -= rounding;
        hi[k] += rounding;
        size = std::max({size, std::fabs(lo[k]), std::fabs(hi[k])});
    }
    auto nearest = [&](const float *p) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) {
            const double d = p[k] - std::min(std::max((double)p[k], lo[k]), hi[k]);
            s += d * d;
        }
        return std::sqrt(s);
    };
    auto farthest = [&](const float *p) {  // distance to the box's farthest corner
        double s = 0.0;
        for (int k = 0; k < 3; k++) {
            const double d = std::max(std::fabs(p[k] - lo[k]), std::fabs(p[k] - hi[k]));
            s += d * d;
            size = std::max(size, (double)std::fabs(p[k]));
        }
        return std::sqrt(s);
    };
    for (uint64_t p = 0; p < P; p++) {
        const double w = (double)pairs[p].laser_wall + pairs[p].camera_wall;
        const double wa = std::fabs((double)pairs[p].laser_wall) + std::fabs((double)pairs[p].camera_wall);
        const double g = farthest(pairs[p].laser_point) + farthest(pairs[p].camera_point);
        legs = std::max(legs, g);
        reach = std::max(reach, g + wa);
        wall = std::max(wall, std::fabs(w - bp.t0));
        least = std::min(least, w);  // legs are not negative
        near = std::min(near, w + nearest(pairs[p].laser_point) + nearest(pairs[p].camera_point));
        far = std::max(far, w + g);
    }
    ExactFilter f;
    // Errors in units u = 2^-24.  The reference: 6 u of each leg (norm3df, 3 ulp), u of the
    // path for each of three sums, u each of path - t0 for the shift and the quotient.  The
    // filter, on the same rounded differences: 3.5 u of each leg (3 u on the square, halved,
    // and 2 u of sqrt.approx), u of the legs each for their sum and 1 / dT, u of the
    // constant, u of the quotient for the FMA.  1% covers the second-order terms.
    const double shift = std::max(std::fabs(reach - bp.t0), std::fabs(least - bp.t0));
    const double e = 1.01 * std::ldexp(1.0, -24) * (11.5 * legs + 3.0 * reach + 3.0 * shift + wall) /
                     bp.dT;
    if (P && bp.dT > 1e-9f && size < 1e9 && bp.T <= (1u << 21) && e <= 0.05) f.error = (float)e;
    // every quotient, the filter's and the reference's, rounds into [0, T)
    f.inside = f.error < 0.5f && (near - bp.t0) / bp.dT > -0.49 + 2.0 * e &&
               (far - bp.t0) / bp.dT < (double)bp.T - 0.51 - 2.0 * e;
    return f;
}

ExactShape exact_shape(const Volume &vol, uint64_t P, const ExactFilter &filter, int sm_count) {
    auto shape = [&](bool direct, uint32_t tx, uint32_t ty, uint32_t tz, uint32_t threads,
                     uint64_t ctas, uint64_t pairs) {
        ExactShape e;
        const uint32_t t[3] = {tx, ty, tz};
        e.direct = direct;
        e.threads = threads;
        e.ctas = 1;
        for (int k = 0; k < 3; k++) {
            e.tile[k] = t[k];
            e.tiles[k] = (vol.n[k] + t[k] - 1) / t[k];
            e.ctas *= e.tiles[k];
        }
        // up to `ctas` per SM, as long as a split keeps `pairs` of them
        const uint64_t tiles = e.ctas;
        while (tiles && e.splits < kMaxSplits && e.splits * tiles < ctas * sm_count &&
               P >= pairs * (e.splits + 1))
            e.splits++;
        e.ctas = tiles * e.splits;
        return e;
    };
    // The gathers' latency wants every SM's slots (13 or 14 CTAs of 64 threads) full and an even
    // last round, and a split two groups of pairs.  1,024 tiles x 4,096 pairs: 1 split 1.24 ms,
    // 3 1.08, 5 0.970, 10 0.946; 42 x 11 x 93 voxels x 8,836 pairs: 8 splits 0.571 ms, 16 0.538.
    const ExactShape filtered = shape(false, kTX, kTY, kTZ, kThreads, 64, 2 * kGroup);
    // Direct: an even last round of 8 CTAs per SM (64^3 voxels x 1,024 pairs: 1 split 782 us, 2 766,
    // 4 710).
    const ExactShape direct = shape(true, kDirectX, kDirectY, kDirectZ, kDirectThreads, 24, 64);
    // Quotients that are not trusted would all be computed and then marked (64^3 voxels x 1,024
    // pairs: 1,680 us against 710; 2 x 16 x 3 voxels x 170 pairs: 211 us against 23).  Above a mark
    // per 50 updates a launch of few CTAs waits for the marks, too (69 x 7 x 11 voxels x 80 pairs in
    // bins of 0.3 mm: 24.9 us against 20.0), where one that fills the GPU does not (64^3 voxels x
    // 80 pairs: 39.7 us against 63.7).
    if (!(filter.error < 0.5f) || filtered.ctas > 0x7fffffffull ||
        (filter.error > 0.01f && filtered.ctas < 2ull * sm_count))
        return direct;
    return filtered;
}

int launch_exact(const void *d_H, bool is_complex, uint64_t pitch, const bpgb_pair *d_pairs,
                 uint64_t P, const Volume &vol, const BinParams &bp, const ExactFilter &filter,
                 const ExactShape &shape, void *d_partial, void *d_out, cudaStream_t stream) {
    ExactArgs a = make_args(pitch, P, vol, bp);
    const uint32_t splits = shape.splits;
    for (int k = 0; k < 3; k++) a.tiles[k] = shape.tiles[k];
    a.inv = 1.0f / bp.dT;
    a.invd = 1.0 / (double)bp.dT;
    a.thr = 0.5f - filter.error;
    a.half = 0.5f * (float)(bp.T - 1);
    a.splits = splits;
    if (shape.ctas == 0) return BPGB_OK;
    if (shape.ctas > 0x7fffffffull)
        return set_error(BPGB_ERR_UNSUPPORTED, "volume too large for the exact kernel grid");
    void *target = splits > 1 ? d_partial : d_out;
    void *args[] = {(void *)&d_H, (void *)&d_pairs, (void *)&target, (void *)&a};
    void *kern = shape.direct ? (is_complex ? (void *)bp_exact_direct_kernel<float2>
                                            : (void *)bp_exact_direct_kernel<float>)
                 : is_complex ? (filter.inside ? (void *)bp_exact_kernel<float2, true>
                                               : (void *)bp_exact_kernel<float2, false>)
                              : (filter.inside ? (void *)bp_exact_kernel<float, true>
                                               : (void *)bp_exact_kernel<float, false>);
    BPGB_CUDA_TRY(launch_after(kern, (unsigned)shape.ctas, shape.threads, args, 0, stream));
    count_launches(1);
    if (splits > 1) {
        const unsigned blocks = (unsigned)((a.nvox + 255) / 256);
        if (is_complex)
            launch_after(exact_reduce_kernel<float2>, blocks, 256, 0, stream,
                         (const float2 *)d_partial, (float2 *)d_out, a.nvox, splits);
        else
            launch_after(exact_reduce_kernel<float>, blocks, 256, 0, stream, (const float *)d_partial,
                         (float *)d_out, a.nvox, splits);
        count_launches(1);
        BPGB_CUDA_TRY(cudaGetLastError());
    }
    return BPGB_OK;
}

int launch_exact_bins(const bpgb_pair *d_pairs, uint64_t P, const Volume &vol,
                      const BinParams &bp, const int64_t *d_ids, int64_t n, int32_t *d_bins,
                      cudaStream_t stream) {
    if (n <= 0 || P == 0) return BPGB_OK;
    const ExactArgs a = make_args(0, P, vol, bp);
    const uint64_t total = (uint64_t)n * P;
    const unsigned blocks = (unsigned)std::min<uint64_t>((total + 255) / 256, 152ull * 16);
    bp_exact_bins_kernel<<<blocks, 256, 0, stream>>>(d_pairs, d_ids, n, d_bins, a);
    count_launches(1);
    BPGB_CUDA_TRY(cudaGetLastError());
    return BPGB_OK;
}

}  // namespace bpgb
