// The shadow sweep: building and vegetation shadows along one sun ray.
//
// For every pixel p and ray step k the reference (src/umep_solweig.py:2201-2406)
// shifts the DSM / canopy / trunk rasters by the step offset, subtracts the
// step height dz_k (all float64) and accumulates:
//   f      = max(dsm_p, max_k(dsm[p+off_k] - dz_k))          building top seen
//   topmax = max(vegdem_p, max_k(vegdem[p+off_k] - dz_k))    canopy top seen
//   shadowed_k = f > dsm_p
//   veg    |= 1 <= #{top-dz_k, bot-dz_k, top-dz_{k-1}, bot-dz_{k-1} > dsm_p} <= 3,
//             cleared whenever shadowed_k
//   ever   |= veg
// Samples outside the raster read as exactly 0 (no dz subtracted).
//
// The per-pixel loop below evaluates these recurrences in the same float64
// operations, so every mask is bit-identical to the reference, and stops early
// when the remaining steps provably change nothing:
//   * hmax - dz_{k-1} < dsm_p (exactly) -> no later sample can rise above the
//     pixel (and, for wall pixels, hmax - dz_k <= topmax so the canopy top is
//     final); only taken when dsm_p >= 0 (and topmax >= 0), so the zero-valued
//     samples beyond the raster edge could not change anything either;
//   * a sample without canopy (top, trunk <= 0) skips the canopy compares
//     (with dsm_p >= 0 and topmax >= 0 they cannot change anything);
//   * shadowed and not a wall pixel -> every output is final;
//   * shadowed wall pixel with f - dsm_p >= wall -> wallsun is already 0;
//   * with a ray-ceiling plane (ceiling.cuh), every 4th step from step 4 on:
//     ceiling(q_k) - dz_{k-1} (rounded up) < dsm_p bounds every later
//     sample's h - dz_{j-1} below the pixel (dsm_p >= 0; for wall pixels
//     also <= topmax >= 0), so nothing further can change.
// Once a sample leaves the raster it never re-enters (the offsets grow
// monotonically), so the first outside step is applied and the loop ends.
#pragma once
#include "common.cuh"

namespace solweig {

struct ShadowResult {
    double f, topmax;
    bool shadowed, veg, ever;
};

// Height samples of the sweep: the three float64 rasters ...
struct GeoF64 {
    const double* __restrict__ dsm;
    const double* __restrict__ top;
    const double* __restrict__ bot;
    __device__ __forceinline__ void load(long long q, bool vegetation, double& a, double& t, double& b) const {
        a = __ldg(&dsm[q]);
        if (vegetation) {
            t = __ldg(&top[q]);
            b = __ldg(&bot[q]);
        }
    }
};

// ... or, when every value of all three is exactly representable in float32,
// one interleaved (dsm, canopy, trunk, 0) float4 per pixel: a single 16-byte
// load per step, widened to float64 exactly, so every compare is unchanged.
struct GeoF32x4 {
    const float4* __restrict__ geo;
    __device__ __forceinline__ void load(long long q, bool, double& a, double& t, double& b) const {
        const float4 v = __ldg(&geo[q]);
        a = v.x;
        t = v.y;
        b = v.z;
    }
};

// Walk the ray for pixel (r, c).  `is_wall` enables the wall-specific
// continuation rules; `hmax` = max over the raster of dsm, vegdem and vegdem2.
template <typename Geo>
__device__ __forceinline__ ShadowResult shadow_walk_geo(
    const Geo& geo, int rows, int cols, int r, int c, double a, double top_p, bool bush, double wall,
    const int2* __restrict__ ray, const double* __restrict__ dz, int steps, double hmax,
    bool vegetation, const float2* __restrict__ ceiling = nullptr) {
    ShadowResult s;
    s.f = a;
    s.topmax = top_p;
    s.shadowed = false;
    s.veg = bush;
    s.ever = false;
    const bool is_wall = wall > 0.0;
    // dz_prev >= clear  =>  hmax - dz_prev < a in exact arithmetic (the
    // threshold is one ulp above the rounded difference), so no later sample
    // of any of the three rasters can rise above the pixel.
    const double clear = a >= 0.0 ? nextafter(hmax - a, __longlong_as_double(0x7ff0000000000000ll))
                                  : __longlong_as_double(0x7ff0000000000000ll);
    double dz_prev = 0.0;
    int k = 0;
    for (; k < steps; ++k) {
        const int2 o = __ldg(&ray[k]);
        const double dzk = __ldg(&dz[k]);
        const int rr = r + o.x, cc = c + o.y;
        if (!in_raster(rr, cc, rows, cols)) break;
        const long long q = (long long)rr * cols + cc;
        // Early exits that cannot change any output.
        if (dz_prev >= clear && (!is_wall || (s.topmax >= 0.0 && hmax - dzk <= s.topmax))) {
            k = steps;  // nothing further can change; no outside fix-up needed
            break;
        }
        if (ceiling != nullptr && k >= 4 && (k & 3) == 0) {
            const double e = __dsub_ru((double)__ldg(&ceiling[q]).x, dz_prev);
            if (a >= 0.0 && e < a && (!is_wall || (s.topmax >= 0.0 && e <= s.topmax))) {
                k = steps;
                break;
            }
        }
        double hq, tq = 0.0, bq = 0.0;
        geo.load(q, vegetation, hq, tq, bq);
        const double aq = hq - dzk;
        s.f = fmax(s.f, aq);
        s.shadowed = s.f > a;
        if (vegetation) {
            if (tq <= 0.0 && bq <= 0.0 && a >= 0.0 && s.topmax >= 0.0) {
                // No canopy at this sample: its shifted tops are <= 0 <= a and
                // cannot raise topmax, so only the carried flags move.
                if (s.shadowed) s.veg = false;
                else s.ever = s.ever || s.veg;
            } else {
                s.topmax = fmax(s.topmax, tq - dzk);
                if (s.shadowed) {
                    s.veg = false;
                } else {
                    const int n = (int)(tq - dzk > a) + (int)(bq - dzk > a) + (int)(tq - dz_prev > a) +
                                  (int)(bq - dz_prev > a);
                    s.veg = s.veg || (n > 0 && n < 4);
                    s.ever = s.ever || s.veg;
                }
            }
        }
        if (s.shadowed && (!is_wall || s.f - a >= wall)) {
            k = steps;
            break;
        }
        dz_prev = dzk;
    }
    if (k < steps) {
        // First step whose sample is outside the raster: all shifted values are 0.
        s.f = fmax(s.f, 0.0);
        s.shadowed = s.f > a;
        if (vegetation) {
            s.topmax = fmax(s.topmax, 0.0);
            if (s.shadowed) s.veg = false;
            s.ever = s.ever || s.veg;
        }
    }
    return s;
}

// The same walk over the packed float4 geometry, for a ray known to stay in
// the raster for `kend` steps (the first step outside, or `steps`).
//
// Most samples of a walk matter to nothing: with H = max(dsm, canopy, trunk) of
// the sample, H - dz_{k-1} below `thr` (the pixel's height, or for a wall pixel
// already in shadow the building top seen) means that no compare of the step
// is above the pixel and f cannot grow.  A canopy top below the pixel enters no
// output.  So a step is one 4-byte load of the plane of H and one float32
// compare, with `lo` = dz_{k-1} rounded down (H - lo is rounded up, so a step is
// never missed), four steps at a time from the hour's records {offset, lo};
// only the steps that pass load the float4 sample and compare in
// float64, exactly as shadow_walk_geo.  The same holds for the ray ceiling
// (nothing ahead reaches thr: the walk ends) and the window maximum (skip
// kCeilSkip steps), consulted at steps 4, 8, ....
//
// Step 0 is the pixel itself (dz_0 = 0).  Once the canopy flag is set at an
// unshadowed step it is `ever`, and it only clears in shadow, so one flag is
// carried.  What bounds it: instruction issue (76 % of the cycles) and the
// latency of the loads, at 32 registers (8 blocks of 256 threads per SM; 40 and
// 48 registers were slower).  Against float64 compares and a 16-byte sample per
// step, at 71 instructions a step: sweep stage 5.37 -> 3.35 ms per 2000^2 day,
// scene set-up 38.0 -> 27.7 ms at 2000^2 (visibility of the lowest 32 patches at
// 1000^2 2.74 -> 1.68 ms), masks identical.
template <typename T>
__device__ __forceinline__ T load_at(const T* __restrict__ base, uint32_t byte) {
    return __ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + byte));
}

// Addresses are 32-bit byte offsets from the planes (the callers keep rasters
// above kPackedMaxPixels on the other walks).
constexpr long long kPackedMaxPixels = 1ll << 28;

__device__ __forceinline__ ShadowResult shadow_walk_packed(
    const float4* __restrict__ geo, const float* __restrict__ height, const float2* __restrict__ ceiling, uint32_t p,
    bool bush, double wall, const int2* __restrict__ rec, const double* __restrict__ dz, int steps, int kend,
    float hmax) {
    const uint32_t pb = 4u * p;  // byte of the pixel in the plane of H; x 2, x 4 in the others
    const float4 own = load_at(geo, 4u * pb);
    const double a = own.x;
    const bool nonneg = own.x >= 0.f;  // samples outside the raster read 0: they matter to lower pixels
    const bool is_wall = wall > 0.0;
    ShadowResult s;
    s.f = a;
    s.topmax = own.y;
    s.shadowed = false;
    s.ever = steps > 0 && (bush || (own.y > own.x) != (own.z > own.x));
    float thr = own.x;
    bool final = false;
    int k = 1;
    while (k < kend) {
        const int g = k & ~3, e = min(g + 4, kend);
        const int4 ra = __ldg(reinterpret_cast<const int4*>(rec + g));
        if (k == g && nonneg) {
            const float lo = __int_as_float(ra.y);
            if (ceiling != nullptr) {
                const float2 cm = load_at(ceiling, 2u * (pb + (uint32_t)ra.x));
                if (__fsub_ru(cm.x, lo) < thr) {
                    final = true;
                    break;
                }
                if (__fsub_ru(cm.y, lo) <= thr && k + kCeilSkip <= kend) {
                    k += kCeilSkip;
                    continue;
                }
            } else if (__fsub_ru(hmax, lo) < thr) {
                final = true;
                break;
            }
        }
        uint32_t reach = 0u;
        if (e - k == 4) {
            const int4 rb = __ldg(reinterpret_cast<const int4*>(rec + g + 2));
            const float h0 = __fsub_ru(load_at(height, pb + (uint32_t)ra.x), __int_as_float(ra.y));
            const float h1 = __fsub_ru(load_at(height, pb + (uint32_t)ra.z), __int_as_float(ra.w));
            const float h2 = __fsub_ru(load_at(height, pb + (uint32_t)rb.x), __int_as_float(rb.y));
            const float h3 = __fsub_ru(load_at(height, pb + (uint32_t)rb.z), __int_as_float(rb.w));
            if (fmaxf(fmaxf(h0, h1), fmaxf(h2, h3)) < thr) {
                k = e;
                continue;
            }
            reach = (h0 < thr ? 0u : 1u) | (h1 < thr ? 0u : 2u) | (h2 < thr ? 0u : 4u) | (h3 < thr ? 0u : 8u);
        } else {
#pragma unroll 1
            for (int i = k; i < e; ++i) {
                const int2 r = __ldg(rec + i);
                if (!(__fsub_ru(load_at(height, pb + (uint32_t)r.x), __int_as_float(r.y)) < thr)) reach |= 1u << (i - g);
            }
        }
        while (reach) {
            const int i = g + __ffs((int)reach) - 1;
            reach &= reach - 1u;
            const int2 r = __ldg(rec + i);
            const float lo = __int_as_float(r.y);
            const float4 v = load_at(geo, 4u * (pb + (uint32_t)r.x));
            if (!(__fsub_ru(v.x, lo) < thr)) {  // the building may reach the pixel
                const double top = v.x - __ldg(&dz[i]);
                if (top > s.f) {
                    s.f = top;
                    s.shadowed = true;
                    if (!is_wall || top - a >= wall) {
                        final = true;
                        break;
                    }
                    thr = __double2float_rd(top);
                }
            }
            // canopy above the pixel, while it is lit and the flag or a wall needs it
            if (!s.shadowed && (is_wall || !s.ever) && !(__fsub_ru(fmaxf(v.y, v.z), lo) < own.x)) {
                const double z = __ldg(&dz[i]), zp = __ldg(&dz[i - 1]), t = v.y, b = v.z;
                s.topmax = fmax(s.topmax, t - z);
                const int n = (int)(t - z > a) + (int)(b - z > a) + (int)(t - zp > a) + (int)(b - zp > a);
                s.ever = s.ever || (n > 0 && n < 4);
            }
        }
        if (final) break;
        k = e;
    }
    if (!final && kend < steps) {
        // First step whose sample is outside the raster: all shifted values are 0.
        s.f = fmax(s.f, 0.0);
        s.shadowed = s.f > a;
        s.topmax = fmax(s.topmax, 0.0);
    }
    s.veg = steps > 0 ? s.ever && !s.shadowed : bush;
    return s;
}

// Entries of a ray's record row: kmax steps padded to groups of four.
__host__ __device__ __forceinline__ int record_pitch(int kmax) { return (kmax + 3) & ~3; }

// Step records of one ray for shadow_walk_packed: rec[k] = {byte offset of the
// sample in a float plane, dz_{k-1} rounded down} for k < K, by one block.
__device__ __forceinline__ void ray_records_block(const int2* __restrict__ ray, const double* __restrict__ dz,
                                                  int K, int cols, int2* __restrict__ rec) {
    for (int k = threadIdx.x; k < record_pitch(K); k += blockDim.x) {
        int2 v = make_int2(0, __float_as_int(0.f));
        if (k < K) {
            const int2 o = __ldg(&ray[k]);
            v = make_int2(4 * (o.x * cols + o.y), __float_as_int(k > 0 ? __double2float_rd(__ldg(&dz[k - 1])) : 0.f));
        }
        rec[k] = v;
    }
}

// Per hour, the first step at which the ray from row r (column c) leaves the
// raster: exits[r] for the rows, exits[rows + c] for the columns (`steps`
// when it never does).  The offsets of a sun ray are monotone along both
// axes, so the steps inside form a prefix found by bisection; a table whose
// offsets are not monotone is scanned linearly.
__device__ __forceinline__ int first_outside(const int2* __restrict__ ray, int steps, bool row_axis, int pos,
                                             int extent, bool monotone) {
    auto inside = [&](int k) {
        const int2 o = __ldg(&ray[k]);
        const int v = pos + (row_axis ? o.x : o.y);
        return v >= 0 && v < extent;
    };
    if (!monotone) {
        for (int k = 0; k < steps; ++k)
            if (!inside(k)) return k;
        return steps;
    }
    int lo = 0, hi = steps;  // inside on [0, lo), answer in [lo, hi]
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (inside(mid)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// first_outside of every row (exits[r]) and column (exits[rows + c]) of a
// rows x cols raster for one ray table, by one block: the offsets are checked
// for monotony along each axis first (bisection needs it).
__device__ __forceinline__ void ray_exits_block(const int2* __restrict__ ray, int K, int rows, int cols,
                                                int* __restrict__ exits) {
    int xi = 1, xd = 1, yi = 1, yd = 1;
    for (int k = 1 + threadIdx.x; k < K; k += blockDim.x) {
        const int2 o = __ldg(&ray[k]), q = __ldg(&ray[k - 1]);
        xi &= o.x >= q.x;
        xd &= o.x <= q.x;
        yi &= o.y >= q.y;
        yd &= o.y <= q.y;
    }
    const int axi = __syncthreads_and(xi), axd = __syncthreads_and(xd);
    const int ayi = __syncthreads_and(yi), ayd = __syncthreads_and(yd);
    const bool mx = axi || axd, my = ayi || ayd;
    for (int i = threadIdx.x; i < rows + cols; i += blockDim.x)
        exits[i] = i < rows ? first_outside(ray, K, true, i, rows, mx)
                            : first_outside(ray, K, false, i - rows, cols, my);
}

__device__ __forceinline__ ShadowResult shadow_walk(
    const double* __restrict__ dsm, const double* __restrict__ top, const double* __restrict__ bot,
    int rows, int cols, int r, int c, double a, double top_p, bool bush, double wall,
    const int2* __restrict__ ray, const double* __restrict__ dz, int steps, double hmax,
    bool vegetation) {
    return shadow_walk_geo(GeoF64{dsm, top, bot}, rows, cols, r, c, a, top_p, bush, wall, ray, dz, steps, hmax,
                           vegetation);
}

// Self-shadowed wall faces (facesh) for the sun window (low, high, middle).
__device__ __forceinline__ double self_shadow_face(double aspect, double wallbol, double low,
                                                   double high, int middle) {
    return middle ? (double)(aspect < low || aspect >= high) - wallbol + 1.0
                  : 1.0 - (double)(aspect > low || aspect <= high);
}

}  // namespace solweig
