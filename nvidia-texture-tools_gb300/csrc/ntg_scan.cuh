// The cluster fits' scan: a cheap, provably safe filter in front of the exact evaluation of the cluster
// orderings (icbc's cluster_fit_four / cluster_fit_three for BC1, squish's Compress4 / Compress3 for BC3 and BC1a).
//
// The fits try every split of a block's sorted colours into consecutive clusters and keep the first one
// whose error, in the reference's float arithmetic, is strictly lowest. That arithmetic has to be
// reproduced for the winner only. The scan evaluates every ordering's error in centred coordinates with
// fused multiply-adds, and the orderings that could be the winner - those below the lowest scanned error plus
// twice the error bound of the two arithmetics, a few of 968 - are then evaluated exactly.
//
// Notation, for weights w_i with sum W, and cluster coefficients alpha = j / k (k = 3: four clusters,
// k = 2: three):
//   A = k sum w alpha, D = k^2 (W sum w alpha^2 - (sum w alpha)^2), v = k sum w alpha (x - mu)
//   least squares:  a = mu + (k W - A) v / D, b = mu - A v / D
//   any end points: error (k W / 2) |m|^2 + (D / (2 k W)) |d|^2 - v d, d = a - b, m = b - mu + (A / (k W)) d
// (errors times k / 2, without the ordering-independent sum w (x - mu)^2).
//
// The error bound. u = 2^-24, M the largest |component|, T = sum w |x - mu|^2 (metric included). For an
// ordering with a scanned error below 0, |fit|^2 <= 4 T, which bounds |d| and |m| by multiples of sqrt(T).
//   - The reference's own roundings: sums of W-weighted terms of size at most 1 (end points are in [0, 1])
//     and M: u W (13 + 46 M) per unit of metric weight with icbc's prefix sums; squish adds a cluster's points one by
//     one: u W (13 + 101 M) when the weights are whole (partial sums grow evenly), u W (13 + 156 M) when not.
//   - The scan's: relative to T, 2,500 u T. With whole weights D is exact; with fractional ones it loses up to
//     60 u W^2 to cancellation (8 u W^2 with weights that are multiples of 1 / 256, whose sums are exact): the end
//     points' bound grows by three times that over D, and the error by as much over W (|d| is at most 1 per channel).
//   - Snapping: both arithmetics reach the least-squares end points within eta = c u W^2 / D + 24 u. Where an end
//     point lies closer than that to the middle between two grid points they may snap apart: such an
//     ordering (about one of 120) always counts among the possible winners, and never as the lowest scanned one.
//     So does an ordering with all colours in one cluster, whose D is 0.
// Errors, bound and scanned errors all scale with the metric, so its size is free as long as none of them overflows.
// Blocks outside the bound's assumptions (NaN, infinities, |x| > 2, metric weights out of [0, 2^40]) have every
// ordering evaluated exactly. (With weights above 4 left out too, colour weights of 3 took a 2048x2048 BC1 level
// 3,475 us; 1,172 now, 1,385 with every ordering evaluated exactly by one thread per block. 1024x1024 BC3: 800, 344, 395.)
#pragma once

#include "ntg_device.cuh"

namespace ntg {

__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float max3_abs(float a, float b, float c) { return fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c)); }
__device__ __forceinline__ f32x2 f2_dup(float x) { return f2_pack(x, x); }

// Shared memory by its 32-bit address: functions that are not inlined get generic pointers.
__device__ __forceinline__ uint32_t shared_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float4 load_shared(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void store_shared(uint32_t a, float x, float y) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}

// One block's scan constants, written by the lane that owns the block and read by the whole warp.
struct ScanBlock {
    float mu[3], W;
    float eta;    // the snapping bound's numerator, in steps of the finest grid
    float slack;  // twice the error bound, for errors of scale 1
    int n;        // colours
    int flat;     // 16 colours of weight 1
    float metric[3];
};

// `ref_m`: the reference's rounding bound per unit of M (46 icbc, 101 or 156 squish); `eta_m`: the same for the end
// points (47 icbc, 90 or 153 squish); `err_d`: the bound of D's rounding in u W^2; `whole`: the weights are whole
// numbers.
__device__ __forceinline__ void scan_begin(ScanBlock &s, int n, f3 sum, float wsum, float maxabs, float scatter, bool whole,
                                           f3 metric, float ref_m, float eta_m, float err_d) {
    const float u = 5.9604645e-8f;
    s.mu[0] = sum.x / wsum; s.mu[1] = sum.y / wsum; s.mu[2] = sum.z / wsum;
    s.W = wsum;
    const float mx = fmaxf(fmaxf(metric.x, metric.y), metric.z), mn = fminf(fminf(metric.x, metric.y), metric.z);
    const bool fits = maxabs <= 2.0f && mn >= 0.0f && mx <= 1.0995116e12f && scatter <= 256.0f && wsum > 0.0f && wsum <= 16.5f;
    const float per = wsum * (13.0f + ref_m * maxabs + err_d);
    s.slack = 2.0f * u * (per * (metric.x + metric.y + metric.z) + 2500.0f * scatter * mx);
    // an infinite bound makes every ordering a possible winner
    s.eta = fits ? 63.0f * u * (eta_m * maxabs + 20.0f + 24.0f * sqrtf(scatter / wsum) + 3.0f * err_d) * wsum * wsum
                 : __int_as_float(0x7f800000);
    s.n = n;
    s.flat = n == 16 && whole && wsum == 16.0f;
    s.metric[0] = metric.x; s.metric[1] = metric.y; s.metric[2] = metric.z;
}

// The orderings as the scan's lanes read them, two at a time (32 apart): ordering i is half (i / 32) & 1 of pair
// 32 (i / 64) + i % 32. `ends`: byte offsets of the cumulative ends in a table of float4, 10 bits each (first, second,
// last; for k = 2 the second is the table's zero entry 17). For 16 colours of weight 1: -1 / D, -A and D / (2 k W).
// Two arrays of 16 bytes a pair, so that a warp's loads are whole lines.
template <int PAIRS>
struct ScanOrders {
    struct __align__(16) Ends { uint32_t ends[2]; float rn[2]; } e[PAIRS];
    struct __align__(16) Sums { float nA[2], cD[2]; } s[PAIRS];
};

// Fills the pairs from an icbc table (bytes: cumulative ends), repeating the first ordering at the end; EMPTY puts the
// ordering with every end 0, which squish tries and icbc leaves out, first. Host.
template <int K, int PAIRS, bool EMPTY = false>
inline void scan_orders(const uint32_t *table, int total, ScanOrders<PAIRS> &out) {
    for (int i = 0; i < 2 * PAIRS; i++) {
        const int at = EMPTY ? i - 1 : i;
        const uint32_t o = at < 0 ? 0 : table[at < total ? at : 0];
        const int c0 = o & 255, c1 = K == 3 ? (o >> 8) & 255 : 0, c2 = (o >> (K == 3 ? 16 : 8)) & 255;
        const int A = c0 + c1 + c2, U = K == 3 ? 5 * c0 + 3 * c1 + c2 : 3 * c0 + c2, D = 16 * U - A * A;
        const int p = 32 * (i / 64) + i % 32, h = (i / 32) & 1;
        out.e[p].ends[h] = (uint32_t)(16 * c0) | (uint32_t)(K == 3 ? 16 * c1 : 16 * 17) << 10 | (uint32_t)(16 * c2) << 20;
        out.e[p].rn[h] = -1.0f / (float)D;  // -infinity where all colours share a cluster
        out.s[p].nA[h] = (float)-A;
        out.s[p].cD[h] = (float)D / (float)(2 * K * 16);
    }
}
template <int PAIRS>
__device__ __forceinline__ uint32_t scan_ends(const ScanOrders<PAIRS> &orders, int i) {
    return orders.e[32 * (i >> 6) + (i & 31)].ends[(i >> 5) & 1];
}

// Floats as unsigned integers in the same order; the two zeros are equal.
__device__ __forceinline__ uint32_t float_order(float e) {
    const uint32_t b = __float_as_uint(e + 0.0f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float order_float(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// A warp's scratch for the block that it is at.
struct ScanScratch {
    float4 centred[18];    // a summed-area table in centred coordinates (17 entries), and a zero
    float2 e[19 * 32];     // the scanned errors (infinite where hard): 16 rows of pairs for k = 3, 3 for k = 2; then the
                           // possible winners' list
};

// A block's table for scan_rows, centred here unless it is already.
__device__ __forceinline__ void scan_centre(ScanScratch &w, const ScanBlock &blk, const float4 *table, bool centred = false) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (lane < 18) {
        float4 p = table[lane];
        if (!centred) p = make_float4(__fmaf_rn(-p.w, blk.mu[0], p.x), __fmaf_rn(-p.w, blk.mu[1], p.y), __fmaf_rn(-p.w, blk.mu[2], p.z), p.w);
        w.centred[lane] = lane == 17 ? make_float4(0, 0, 0, 0) : p;
    }
    __syncwarp();
}

// The scan of a block's orderings by all lanes of the warp: writes the scanned errors, returns this lane's lowest and
// in `hard` its hard orderings (bit r: ordering 32 r + lane), those with an end point too near a snapping tie.
// E = (k W / 2) |m|^2 - d (v - D / (2 k W) d), with nd = -d; two orderings at a time, one in each half of the packed
// registers. UNIT: unit metric; FLAT: 16 colours of weight 1. Not inlined, and k at run time, so that the loop
// stays in the instruction cache (inlined for each k it lost a quarter of its speed to instruction fetches).
template <bool UNIT, bool FLAT>
__device__ __noinline__ float scan_rows(ScanScratch *w, const ScanBlock *blk, const uint4 *__restrict__ op, int sums, int rows,
                                        int first, float k, uint32_t *hard_rows) {
    const int lane = threadIdx.x & 31;
    const float mu[3] = {blk->mu[0], blk->mu[1], blk->mu[2]}, metric[3] = {blk->metric[0], blk->metric[1], blk->metric[2]};
    const float W = blk->W, kW = k * W, cm = 0.5f * kW, ca = rcp_approx(kW), cd = 0.5f * ca, eta = blk->eta;
    const float u0 = 2.0f * k - 1.0f;  // U = u0 w0 + 3 w1 + w2
    const uint32_t base = shared_address(w->centred);
    const float inf = __int_as_float(0x7f800000);
    const float magic = 12582912.0f;  // 1.5 2^23: adding it rounds to the nearest whole number
    const f32x2 magic2 = f2_dup(magic), g31 = f2_dup(31.0f), g63 = f2_dup(63.0f);
    float best = inf;
    uint32_t bits = 0, bit = 1;
    op += lane;  // the pairs' ends; their sums lie `sums` entries on
    uint32_t ep = shared_address(w->e + 32 * first + lane);
#pragma unroll 1
    for (int j = 0; j < rows; j++, op += 32, ep += 256, bit <<= 2) {
        const uint4 r0 = __ldg(op);
        const uint32_t ends[2] = {r0.x, r0.y};
        float x[2], y[2], z[2], a[2], q[2], rn[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t o = ends[h];
            const float4 p0 = load_shared(base + (o & 1023)), p1 = load_shared(base + ((o >> 10) & 1023)), p2 = load_shared(base + (o >> 20));
            x[h] = (p0.x + p2.x) + p1.x; y[h] = (p0.y + p2.y) + p1.y; z[h] = (p0.z + p2.z) + p1.z;
            if (!FLAT) {
                a[h] = -p1.w - (p0.w + p2.w);
                q[h] = __fmaf_rn(3.0f, p1.w, __fmaf_rn(u0, p0.w, p2.w));
            }
        }
        const f32x2 v[3] = {f2_pack(x[0], x[1]), f2_pack(y[0], y[1]), f2_pack(z[0], z[1])};
        f32x2 nA, cD;
        if (FLAT) {
            const float4 r1 = __ldg(reinterpret_cast<const float4 *>(op + sums));
            rn[0] = __uint_as_float(r0.z); rn[1] = __uint_as_float(r0.w);
            nA = f2_pack(r1.x, r1.y);
            cD = f2_pack(r1.z, r1.w);
        } else {
            nA = f2_pack(a[0], a[1]);
            const f32x2 nD = f2_fma(nA, nA, f2_mul(f2_pack(q[0], q[1]), f2_dup(-W)));
            float d0, d1;
            f2_unpack(nD, d0, d1);
            rn[0] = rcp_approx(d0);
            rn[1] = rcp_approx(d1);
            cD = f2_mul(nD, f2_dup(-cd));
        }
        const f32x2 rn2 = f2_pack(rn[0], rn[1]);
        float nA0, nA1, nB0, nB1;
        f2_unpack(nA, nA0, nA1);
        f2_unpack(f2_sub(f2_dup(-kW), nA), nB0, nB1);
        const f32x2 nal = f2_mul(nA, f2_dup(ca));
        float far0 = 0.0f, far1 = 0.0f;
        f32x2 mm, gd;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const f32x2 grid = c == 1 ? g63 : g31;
            const float st = c == 1 ? 1.0f / 63.0f : 1.0f / 31.0f;
            float w0, w1;
            f2_unpack(f2_mul(v[c], rn2), w0, w1);  // -v / D
            const f32x2 ea = f2_pack(fma_sat(nB0, w0, mu[c]), fma_sat(nB1, w1, mu[c]));
            const f32x2 eb = f2_pack(fma_sat(-nA0, w0, mu[c]), fma_sat(-nA1, w1, mu[c]));
            // minus the snapped grid coordinates, and the distances to them
            const f32x2 na = f2_sub(magic2, f2_fma(ea, grid, magic2)), nb = f2_sub(magic2, f2_fma(eb, grid, magic2));
            float fa0, fa1, fb0, fb1;
            f2_unpack(f2_fma(ea, grid, na), fa0, fa1);
            f2_unpack(f2_fma(eb, grid, nb), fb0, fb1);
            far0 = max3_abs(far0, fa0, fb0);
            far1 = max3_abs(far1, fa1, fb1);
            const f32x2 nd = f2_mul(f2_sub(na, nb), f2_dup(st));
            const f32x2 mc = f2_fma(nal, nd, f2_fma(nb, f2_dup(-st), f2_dup(-mu[c]))), gc = f2_fma(cD, nd, v[c]);
            const f32x2 mw = UNIT ? mc : f2_mul(mc, f2_dup(metric[c])), gw = UNIT ? gc : f2_mul(gc, f2_dup(metric[c]));
            mm = c == 0 ? f2_mul(mw, mc) : f2_fma(mw, mc, mm);
            gd = c == 0 ? f2_mul(gw, nd) : f2_fma(gw, nd, gd);
        }
        float e0, e1;
        f2_unpack(f2_fma(f2_dup(cm), mm, gd), e0, e1);
        if (!(far0 <= __fmaf_rn(-eta, fabsf(rn[0]), 0.4999f))) { e0 = inf; bits |= bit; }
        if (!(far1 <= __fmaf_rn(-eta, fabsf(rn[1]), 0.4999f))) { e1 = inf; bits |= 2 * bit; }
        store_shared(ep, e0, e1);
        best = fminf(best, fminf(e0, e1));
    }
    *hard_rows = bits;
    return best;
}

// The scan of one fit: `rows` rows of pairs into the errors from row `first` on; returns in `bits` the lane's possible
// winners (bit r: ordering 32 r + lane), within `slack` of the warp's lowest scanned error.
template <int PAIRS>
__device__ __forceinline__ uint32_t scan_bits(ScanScratch &w, const ScanBlock &blk, const ScanOrders<PAIRS> &orders, int rows,
                                              int first, float k, bool unit) {
    const int lane = threadIdx.x & 31;
    const uint4 *const op = reinterpret_cast<const uint4 *>(&orders);
    uint32_t bits;
    const float best = !unit      ? scan_rows<false, false>(&w, &blk, op, PAIRS, rows, first, k, &bits)
                       : blk.flat ? scan_rows<true, true>(&w, &blk, op, PAIRS, rows, first, k, &bits)
                                  : scan_rows<true, false>(&w, &blk, op, PAIRS, rows, first, k, &bits);
    const float limit = order_float(__reduce_min_sync(0xffffffffu, float_order(best))) + (0.5f * k) * blk.slack;
    uint32_t bit = 1;
#pragma unroll 2
    for (int j = 0; j < rows; j++, bit <<= 2) {  // a lane reads back only its own errors
        const float2 e = w.e[32 * (first + j) + lane];
        if (e.x <= limit) bits |= bit;
        if (e.y <= limit) bits |= 2 * bit;
    }
    return bits;
}

// Appends the orderings of `bits` to the list, marked with `mark`.
__device__ __forceinline__ void scan_list(uint16_t *list, int &count, uint32_t bits, int mark) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    for (unsigned m; (m = __ballot_sync(0xffffffffu, bits != 0)) != 0; count += __popc(m)) {
        if (bits) list[count + __popc(m & below)] = (uint16_t)(mark | (32 * (__ffs(bits) - 1) + lane));
        bits &= bits - 1;
    }
}

// A lane's best exact result so far: the first ordering of the lowest error below FLT_MAX, and its end points.
struct FitBest {
    uint32_t key = 0xffffffffu;
    int order = 0x7fffffff;
    f3 a, b;
    __device__ __forceinline__ void take(float e, int o, f3 ea, f3 eb) {
        const uint32_t k = float_order(e);
        if (e < FLT_MAX && (k < key || (k == key && o < order))) { key = k; order = o; a = ea; b = eb; }
    }
    // The warp's best writes its end points to out[0..5]; zeros when there is none. Returns its ordering, -1 for none.
    __device__ __forceinline__ int finish(float *out) const {
        const uint32_t least = __reduce_min_sync(0xffffffffu, key);
        const int first = __reduce_min_sync(0xffffffffu, key == least ? order : 0x7fffffff);
        if (least == 0xffffffffu) {
            if ((threadIdx.x & 31) < 6) out[threadIdx.x & 31] = 0.0f;
        } else if (key == least && order == first) {
            out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = b.x; out[4] = b.y; out[5] = b.z;
        }
        return least == 0xffffffffu ? -1 : first;
    }
};

// ---- two blocks per warp: lanes 0-15 one block's texels, lanes 16-31 the next one's ----

constexpr unsigned kAll = 0xffffffffu;
constexpr int kFitWarps = 4;  // warps per CTA, each on its own

// Blocks per warp of a launch: one where the GPU holds a warp for each (152 SMs x 5 CTAs x 4 warps), because what such a
// launch takes is one warp's time through its blocks. One float level, two blocks per warp against one: BC1 32x32 28 and
// 21 us, 128x128 27 and 23, 192x192 (2,304 blocks) 29 and 25, 256x256 (4,096) 35 and 39; BC3 64x64 38 and 29, 192x192 39
// and 31, 256x256 41 and 44.
constexpr int fit_blocks_per_warp(long long nblocks) { return nblocks <= 152 * 5 * kFitWarps ? 1 : 2; }

// One half's scratch in shared memory.
struct HalfScratch {
    float stage[16 * 8];  // terms per texel or colour
    float pad[8];         // the two halves' stages lie on different banks
    float4 table[2][18];  // the ZERO summed-area tables (17 entries) of the two fits; squish: the one table, the points
    float4 sum;           // squish: the sum of the points
    ScanBlock block[2];   // and their scans' constants
    float ends[12];       // the fits' end points
    int order[2];         // the fits' winners (-1: none) and
    uint32_t error[2];    // their errors (float_order), where the caller wants them
};
struct WarpScratch {
    ScanScratch scan;
    HalfScratch half[2];
};

struct Half {
    int hl;         // lane in the half: texel or colour index
    int shift;      // first lane of the half
    HalfScratch *s;
    __device__ __forceinline__ float get(float v, int src) const { return __shfl_sync(kAll, v, src, 16); }
    __device__ __forceinline__ unsigned ballot(bool p) const { return (__ballot_sync(kAll, p) >> shift) & 0xffffu; }
    // Sum over i < n, in order, of the terms stage[8 i + c]; lane c of the half returns it.
    __device__ __forceinline__ float ordered(int n) const {
        float acc = 0.0f;
        const float *p = s->stage + (hl & 7);
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (i < n) acc += p[8 * i];
        return acc;
    }
    // The same over the set bits i of `mask`.
    __device__ __forceinline__ float ordered_of(unsigned mask) const {
        float acc = 0.0f;
        const float *p = s->stage + (hl & 7);
#pragma unroll
        for (int i = 0; i < 16; i++)
            if ((mask >> i) & 1) acc += p[8 * i];
        return acc;
    }
};

// A lane's position among its half's first n keys in a stable insertion sort's order: its rank, unless a key is NaN (which
// the sort leaves where it meets it).
__device__ __forceinline__ int half_rank(const Half &H, float d, int n) {
    float *const st = H.s->stage;
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const float e = H.get(d, j);
        rank += j < n && (e < d || (e == d && j < H.hl));
    }
    const bool odd = H.ballot(H.hl < n && d != d) != 0;
    __syncwarp();
    if (__any_sync(kAll, odd)) {
        float *const key = st;
        int *const ord = reinterpret_cast<int *>(st + 16), *const pos = reinterpret_cast<int *>(st + 32);
        key[H.hl] = d;
        __syncwarp();
        if (H.hl == 0) {
            for (int i = 0; i < n; i++) ord[i] = i;
            for (int i = 1; i < n; i++)
                for (int j = i; j > 0 && key[j] < key[j - 1]; j--) {
                    const float t = key[j]; key[j] = key[j - 1]; key[j - 1] = t;
                    const int o = ord[j]; ord[j] = ord[j - 1]; ord[j - 1] = o;
                }
            for (int i = 0; i < n; i++) pos[ord[i]] = i;
        }
        __syncwarp();
        if (odd && H.hl < n) rank = pos[H.hl];
        __syncwarp();
    }
    return rank;
}

// Bit i of m to bit 2 i.
__device__ __forceinline__ uint32_t spread_bits(uint32_t m) {
    m = (m | (m << 8)) & 0x00ff00ffu;
    m = (m | (m << 4)) & 0x0f0f0f0fu;
    m = (m | (m << 2)) & 0x33333333u;
    return (m | (m << 1)) & 0x55555555u;
}

// ---- one block per thread ----

// The pairs of orderings in the order in which lane_scan walks them - last end from 16 down to 0, second end, first end in
// steps of two: last << 10 | second << 5 | first of the pair's first ordering; the other has the next first end. The walk
// for n colours begins at start[n].
constexpr int kLaneWords = 33;  // of 16 pairs
struct LanePairs {
    uint16_t four[16 * kLaneWords], three[96];
    uint16_t start4[17], start3[17];
};
inline void lane_pairs(LanePairs &out) {
    int n4 = 0, n3 = 0;
    for (int c2 = 16; c2 >= 0; c2--) {
        out.start4[c2] = (uint16_t)n4;
        out.start3[c2] = (uint16_t)n3;
        for (int c1 = 0; c1 <= c2; c1++)
            for (int c0 = 0; c0 <= c1; c0 += 2) out.four[n4++] = (uint16_t)(c2 << 10 | c1 << 5 | c0);
        for (int c0 = 0; c0 <= c2; c0 += 2) out.three[n3++] = (uint16_t)(c2 << 10 | c2 << 5 | c0);
    }
}

// A thread's words of a [k][thread] array in shared memory.
__device__ __forceinline__ uint32_t load_word(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void store_word(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

// The scan of a block's orderings by one thread, scan_rows' arithmetic on pairs that differ in the first end only, so that
// two of the three table entries stay in registers. `table`: the thread's summed-area table (17 entries, 16 T bytes apart);
// `words`: its flags (4 T bytes apart): bit 2 i + h for ordering h of a word's pair i, set where the ordering's scanned error
// is within `slack` of the lowest so far or it is hard. `start`: the walk's first pair. Returns the number of words, from
// start / 16 on.
template <bool UNIT, int T>
__device__ __noinline__ int lane_scan(uint32_t table, uint32_t words, float mux, float muy, float muz, float W, float eta,
                                        float slack, int n, int start, float k, float3 metric) {
    const uint32_t stride = 16 * T;
    const float kW = k * W, cm = 0.5f * kW, ca = rcp_approx(kW), cd = 0.5f * ca;
    const float u0 = 2.0f * k - 1.0f;
    const float inf = __int_as_float(0x7f800000);
    const float magic = 12582912.0f;
    const f32x2 magic2 = f2_dup(magic), g31 = f2_dup(31.0f), g63 = f2_dup(63.0f);
    const float mu[3] = {mux, muy, muz}, mt[3] = {metric.x, metric.y, metric.z};
    float best = inf;
    uint32_t bits = 0;
    int pos = 2 * (start & 15), done = start >> 4;
    words += 4 * T * (uint32_t)done;
    const bool three = k == 2.0f;
#pragma unroll 1
    for (int c2 = n; c2 >= 1; c2--) {  // the last end is never 0
        const float4 p2 = load_shared(table + c2 * stride);
#pragma unroll 1
        for (int c1 = three ? c2 : 0; c1 <= c2; c1++) {
            const float4 p1 = three ? make_float4(0, 0, 0, 0) : load_shared(table + c1 * stride);
            const float bx = p1.x + p2.x, by = p1.y + p2.y, bz = p1.z + p2.z, bw = -p1.w - p2.w;
            const float qb = __fmaf_rn(3.0f, p1.w, p2.w);
            uint32_t at = table;
#pragma unroll 1
            for (int c0 = 0; c0 <= c1; c0 += 2, at += 2 * stride) {
                // the pair's second entry may lie one past the row's last (or on the flags): read, not used
                const float4 r0 = load_shared(at), r1 = load_shared(at + stride);
                const f32x2 nA = f2_pack(bw - r0.w, bw - r1.w), q = f2_pack(__fmaf_rn(u0, r0.w, qb), __fmaf_rn(u0, r1.w, qb));
                const f32x2 v[3] = {f2_fma(nA, f2_dup(mux), f2_pack(r0.x + bx, r1.x + bx)), f2_fma(nA, f2_dup(muy), f2_pack(r0.y + by, r1.y + by)),
                                    f2_fma(nA, f2_dup(muz), f2_pack(r0.z + bz, r1.z + bz))};
                const f32x2 nD = f2_fma(nA, nA, f2_mul(q, f2_dup(-W)));
                float d0, d1;
                f2_unpack(nD, d0, d1);
                const float rn0 = rcp_approx(d0), rn1 = rcp_approx(d1);
                const f32x2 cD = f2_mul(nD, f2_dup(-cd)), rn2 = f2_pack(rn0, rn1);
                float nA0, nA1, nB0, nB1;
                f2_unpack(nA, nA0, nA1);
                f2_unpack(f2_sub(f2_dup(-kW), nA), nB0, nB1);
                const f32x2 nal = f2_mul(nA, f2_dup(ca));
                float far0 = 0.0f, far1 = 0.0f;
                f32x2 mm, gd;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const f32x2 grid = c == 1 ? g63 : g31;
                    const float st = c == 1 ? 1.0f / 63.0f : 1.0f / 31.0f;
                    float w0, w1;
                    f2_unpack(f2_mul(v[c], rn2), w0, w1);
                    const f32x2 ea = f2_pack(fma_sat(nB0, w0, mu[c]), fma_sat(nB1, w1, mu[c]));
                    const f32x2 eb = f2_pack(fma_sat(-nA0, w0, mu[c]), fma_sat(-nA1, w1, mu[c]));
                    const f32x2 na = f2_sub(magic2, f2_fma(ea, grid, magic2)), nb = f2_sub(magic2, f2_fma(eb, grid, magic2));
                    float fa0, fa1, fb0, fb1;
                    f2_unpack(f2_fma(ea, grid, na), fa0, fa1);
                    f2_unpack(f2_fma(eb, grid, nb), fb0, fb1);
                    far0 = max3_abs(far0, fa0, fb0);
                    far1 = max3_abs(far1, fa1, fb1);
                    const f32x2 nd = f2_mul(f2_sub(na, nb), f2_dup(st));
                    const f32x2 mc = f2_fma(nal, nd, f2_fma(nb, f2_dup(-st), f2_dup(-mu[c]))), gc = f2_fma(cD, nd, v[c]);
                    const f32x2 mw = UNIT ? mc : f2_mul(mc, f2_dup(mt[c])), gw = UNIT ? gc : f2_mul(gc, f2_dup(mt[c]));
                    mm = c == 0 ? f2_mul(mw, mc) : f2_fma(mw, mc, mm);
                    gd = c == 0 ? f2_mul(gw, nd) : f2_fma(gw, nd, gd);
                }
                float e0, e1;
                f2_unpack(f2_fma(f2_dup(cm), mm, gd), e0, e1);
                const bool h0 = !(far0 <= __fmaf_rn(-eta, fabsf(rn0), 0.4999f));
                const bool h1 = !(far1 <= __fmaf_rn(-eta, fabsf(rn1), 0.4999f)), second = c0 < c1;
                best = fminf(best, fminf(h0 ? inf : e0, h1 || !second ? inf : e1));
                const float limit = best + slack;
                if (h0 || e0 <= limit) bits |= 1u << pos;
                if (second && (h1 || e1 <= limit)) bits |= 2u << pos;
                pos += 2;
                if (pos == 32) {
                    store_word(words, bits);
                    words += 4 * T;
                    done++;
                    bits = 0; pos = 0;
                }
            }
        }
    }
    if (pos) {
        store_word(words, bits);
        done++;
    }
    return done;
}

}  // namespace ntg
