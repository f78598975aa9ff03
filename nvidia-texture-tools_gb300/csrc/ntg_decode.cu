// Block decode and error sums on the GPU: Surface::setImage2D with the D3D10 decoder
// (src/nvtt/Surface.cpp:908-1116, src/nvimage/BlockDXT.cpp) and nv::rmsColorError /
// rmsAlphaError (src/nvimage/ErrorMetric.cpp:13-71), so quality checks run at GPU speed.
#include "ntg_device.cuh"
#include "ntg_internal.h"

namespace ntg {

// The 16 values of an interpolated-alpha block (AlphaBlockDXT5::evaluatePalette, D3D10), through the table of v / 255:
// palette entry k is ((7 - j) a0 + j a1) / 7 with j = 0, 7, 1, 2, ... 6 for k = 0, 1, 2, ... 7, or over 5 with 0 and 255 last.
__device__ __forceinline__ void decode_alpha8(uint2 b, const float *unit8, float out[16]) {
    const uint64_t u = (uint64_t)b.x | ((uint64_t)b.y << 32);
    const int a0 = (int)(u & 255), a1 = (int)((u >> 8) & 255), parts = a0 > a1 ? 7 : 5;
    const unsigned magic = a0 > a1 ? 9363u : 13108u;  // x / 7 and x / 5 for x below 2^11
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const int k = (int)(u >> (16 + 3 * i)) & 7, j = k == 0 ? 0 : (k == 1 ? parts : k - 1);
        unsigned v = ((unsigned)((parts - j) * a0 + j * a1) * magic) >> 16;
        if (a0 <= a1 && k >= 6) v = k == 6 ? 0 : 255;
        out[i] = unit8[v];
    }
}

// One thread per block; writes the texels inside the image (1/255 scale, as setImage2D does). VEC: the image's width is a
// multiple of four and its planes start on 16-byte boundaries: each row of a block is one 16-byte store per
// plane. The quotients v / 255 come from a table that each CTA computes. Bound by the stores: 2048x2048 BC3 took
// 41 us with a division and a 4-byte store per texel and channel and takes 15 with 16-byte stores and the table (floor: 71 MB, 11 us).
template <bool VEC>
__global__ void __launch_bounds__(128) k_decode(int format, const uint8_t *__restrict__ blocks, int w, int h, float *__restrict__ rgba) {
    __shared__ float unit8[256];
    unit8[threadIdx.x] = (float)threadIdx.x / 255.0f;
    unit8[threadIdx.x + 128] = (float)(threadIdx.x + 128) / 255.0f;
    __syncthreads();
    const int bw = (w + 3) / 4, bh = (h + 3) / 4;
    const long long nb = (long long)bw * bh;
    const long long blk = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (blk >= nb) return;
    const int bx = (int)(blk % bw), by = (int)(blk / bw);
    const size_t n = (size_t)w * h;
    float r[16], g[16], b[16], a[16];
    const bool bc1 = format == 1 || format == 2;  // BC1a has BC1's block layout
    if (format == 6) {  // BlockATI1::decodeBlock (src/nvimage/BlockDXT.cpp:513-526)
        decode_alpha8(*reinterpret_cast<const uint2 *>(blocks + 8 * (size_t)blk), unit8, r);
#pragma unroll
        for (int i = 0; i < 16; i++) { g[i] = r[i]; b[i] = r[i]; a[i] = 1.0f; }
    } else if (bc1 || format == 4) {
        const uint2 c = *reinterpret_cast<const uint2 *>(blocks + (bc1 ? 8 : 16) * (size_t)blk + (bc1 ? 0 : 8));
        const unsigned c0 = c.x & 0xFFFF, c1 = c.x >> 16;
        Pal8 p;
        palette_d3d10(c0, c1, p);
        float pr[4], pg[4], pb[4];
#pragma unroll
        for (int k = 0; k < 4; k++) { pr[k] = unit8[p.r[k]]; pg[k] = unit8[p.g[k]]; pb[k] = unit8[p.b[k]]; }
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int k = (c.y >> (2 * i)) & 3;
            r[i] = k & 2 ? (k & 1 ? pr[3] : pr[2]) : (k & 1 ? pr[1] : pr[0]);
            g[i] = k & 2 ? (k & 1 ? pg[3] : pg[2]) : (k & 1 ? pg[1] : pg[0]);
            b[i] = k & 2 ? (k & 1 ? pb[3] : pb[2]) : (k & 1 ? pb[1] : pb[0]);
            a[i] = (c0 <= c1 && k == 3) ? 0.0f : 1.0f;
        }
        if (format == 4) decode_alpha8(*reinterpret_cast<const uint2 *>(blocks + 16 * (size_t)blk), unit8, a);
    } else {
        decode_alpha8(*reinterpret_cast<const uint2 *>(blocks + 16 * (size_t)blk), unit8, r);
        decode_alpha8(*reinterpret_cast<const uint2 *>(blocks + 16 * (size_t)blk + 8), unit8, g);
#pragma unroll
        for (int i = 0; i < 16; i++) { b[i] = 0.0f; a[i] = 1.0f; }
    }
    float *const plane[4] = {rgba, rgba + n, rgba + 2 * n, rgba + 3 * n};
    const float *const texel[4] = {r, g, b, a};
#pragma unroll
    for (int c = 0; c < 4; c++) {
        if constexpr (VEC) {
#pragma unroll
            for (int y = 0; y < 4; y++)
                if (by * 4 + y < h)
                    __stcs(reinterpret_cast<float4 *>(plane[c] + (size_t)(by * 4 + y) * w + bx * 4),
                           make_float4(texel[c][4 * y], texel[c][4 * y + 1], texel[c][4 * y + 2], texel[c][4 * y + 3]));
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int x = bx * 4 + (i & 3), y = by * 4 + (i >> 2);
                if (x < w && y < h) plane[c][(size_t)y * w + x] = texel[c][i];
            }
        }
    }
}

// A sum of non-negative floats kept as an unevaluated triple, each part the rounding error of the one before it (Knuth's
// TwoSum): exact but for the roundings of `lo`, 2^-61 of the sum for a step's twelve terms and less for a partial sum that
// joins another, where each addition in double rounds 2^-53. (A pair lost up to 2^-45 of twelve squares of unlike size.)
struct TripleSum {
    float hi = 0.0f, mid = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float x) {
        float s = hi + x, t = s - hi;
        const float e = (hi - (s - t)) + (x - t);
        hi = s;
        s = mid + e;
        t = s - mid;
        lo += (mid - (s - t)) + (e - t);
        mid = s;
    }
    __device__ __forceinline__ void add(const TripleSum &o) {
        add(o.hi); add(o.mid); add(o.lo);
        float s = hi + mid;  // the parts apart again, so that `lo` stays below 2^-47 of the sum
        mid -= s - hi; hi = s;
        s = mid + lo;
        lo -= s - mid; mid = s;
    }
    __device__ __forceinline__ double value() const { return (double)hi + ((double)mid + (double)lo); }
};

// Squared-error sums, reduced per CTA in double and accumulated atomically; four texels a step. A thread's terms are
// summed as triples of floats: the double unit takes two additions a clock and SM, and one addition per term (with
// its conversion) held the kernel to 74 us for 2048x2048 where reading the images takes 20. 29 us with the launch and the
// zeroing before it, 36 with a conversion of every step's triple. VEC: planes on 16-byte boundaries.
template <bool VEC>
__global__ void k_error_sums(const float *__restrict__ ref, const float *__restrict__ img, size_t n, int alpha_mode,
                             double *__restrict__ sums) {
    constexpr float kFar = 1e37f;
    double c = 0, al = 0;
    TripleSum rc, ra;
    const size_t steps = (n + 3) / 4;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < steps; q += (size_t)gridDim.x * blockDim.x) {
        float p[4][4], t[4][4];  // [plane][texel] of ref and img
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (VEC) {
                const float4 u = __ldg(reinterpret_cast<const float4 *>(ref + k * n) + q), v = __ldg(reinterpret_cast<const float4 *>(img + k * n) + q);
                p[k][0] = u.x; p[k][1] = u.y; p[k][2] = u.z; p[k][3] = u.w;
                t[k][0] = v.x; t[k][1] = v.y; t[k][2] = v.z; t[k][3] = v.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) {  // texels past the end: no error, with any weight
                    const size_t i = 4 * q + j;
                    p[k][j] = i < n ? ref[k * n + i] : 0.0f;
                    t[k][j] = i < n ? img[k * n + i] : 0.0f;
                }
            }
        }
        float e[4][4];
        TripleSum cs, as;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float wgt = 1;
            if (alpha_mode == 1) wgt = p[3][j] * p[3][j];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float d = p[k][j] - t[k][j];
                e[k][j] = (d * d) * wgt;
                cs.add(e[k][j]);
            }
            const float da = t[3][j] - p[3][j];
            e[3][j] = da * da;
            as.add(e[3][j]);
        }
        if (cs.hi <= kFar && as.hi <= kFar) {
            rc.add(cs);
            ra.add(as);
            if (rc.hi > kFar || ra.hi > kFar) {
                c += rc.value();
                al += ra.value();
                rc = ra = TripleSum();
            }
        } else {  // infinities, NaN, or sums towards the end of float's range
#pragma unroll
            for (int j = 0; j < 4; j++) {
                c += (double)e[0][j]; c += (double)e[1][j]; c += (double)e[2][j];
                al += (double)e[3][j];
            }
        }
    }
    c += rc.value();
    al += ra.value();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_down_sync(0xffffffffu, c, o);
        al += __shfl_down_sync(0xffffffffu, al, o);
    }
    __shared__ double s_c[32], s_a[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_c[warp] = c; s_a[warp] = al; }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        c = lane < nw ? s_c[lane] : 0.0;
        al = lane < nw ? s_a[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            c += __shfl_down_sync(0xffffffffu, c, o);
            al += __shfl_down_sync(0xffffffffu, al, o);
        }
        if (lane == 0) { atomicAdd(&sums[0], c); atomicAdd(&sums[1], al); }
    }
}

int launch_decode(int format, const uint8_t *blocks, int w, int h, float *rgba, cudaStream_t s) {
    const long long nb = (long long)((w + 3) / 4) * ((h + 3) / 4);
    if (nb == 0) return 0;
    const unsigned grid = (unsigned)((nb + 127) / 128);
    if (w % 4 == 0 && reinterpret_cast<uintptr_t>(rgba) % 16 == 0) k_decode<true><<<grid, 128, 0, s>>>(format, blocks, w, h, rgba);
    else k_decode<false><<<grid, 128, 0, s>>>(format, blocks, w, h, rgba);
    return launch_status();
}

int launch_rms(const float *ref, const float *img, int w, int h, int alpha_mode, double *sums, cudaStream_t s) {
    const size_t n = (size_t)w * h;
    if (cudaMemsetAsync(sums, 0, 2 * sizeof(double), s) != cudaSuccess) return launch_status();
    if (n == 0) return 0;
    size_t g = ((n + 3) / 4 + 255) / 256;
    if (g > 152 * 4) g = 152 * 4;
    const bool vec = n % 4 == 0 && reinterpret_cast<uintptr_t>(ref) % 16 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0;
    if (vec) k_error_sums<true><<<(unsigned)g, 256, 0, s>>>(ref, img, n, alpha_mode, sums);
    else k_error_sums<false><<<(unsigned)g, 256, 0, s>>>(ref, img, n, alpha_mode, sums);
    return launch_status();
}

NTG_DEFINE_TABLE_UPLOAD(upload_tables_decode)

}  // namespace ntg
