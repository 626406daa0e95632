// Kernels and launch helpers of the batched day, shared by the batched
// entry points (day.cu) and the day gradient (adjoint.cu).  Everything lives
// in an anonymous namespace: each translation unit instantiates its own copy.
#pragma once
#include <cuda_bf16.h>

#include <algorithm>

#include "ceiling.cuh"
#include "gvf_walk.cuh"
#include "hour.cuh"
#include "radiation.cuh"
#include "sweep_tma.cuh"
#include "tcgen05.cuh"

namespace solweig {

namespace {

constexpr int kDayBX = 32, kDayBY = 8;
constexpr int kK = SOLWEIG_MAX_PATCHES;   // contraction depth (patches, padded)
constexpr int kSBO = (kK / 8) * 128;      // bytes between 8-row groups of an operand
constexpr int kARows = 128;               // pixels per contraction tile (MMA M)
constexpr int kABytes = kARows * kK * 2;  // one A operand in shared memory
constexpr int kMaxDayHours = 64;
constexpr uint32_t kWaitPolls = 1u << 24;

// Element offset of (row n, patch k) in the canonical K-major layout.
__host__ __device__ __forceinline__ int canon_off(int n, int k) {
    return (n >> 3) * (kSBO / 2) + (k >> 3) * 64 + (n & 7) * 8 + (k & 7);
}

// What the radiation loop reads of one hour, rounded once from the float64 plan.
struct alignas(16) HourLoop {
    float band_down[SOLWEIG_MAX_BANDS], band_side[SOLWEIG_MAX_BANDS];
    float lw_shade, lw_sun, sw_shade, sw_sun;
    float rad_d, rad_g, rad_i_sin, rad_i_cos;
    float rad_ratio, wave_w, tan_zen, night_lup;
    float night_lup_water, ta;
    uint32_t flags;     // kHour* bits
    uint32_t pad;
    double utci[8];     // 7 coefficients, air temperature
    uint32_t test[8];   // longwave sun test of the hour
};
constexpr uint32_t kHourDay = 1u, kHourFirst = 2u, kHourUpdate = 4u, kHourUtci = 8u;

// Sunlit / shaded tables of one hour.
struct alignas(16) DayTable {
    HourLoop loop;
    double tsun[kK];        // sorted: patch sunlit  <=> tan(asvf) <  T_k
    double vshade[kK];      // sorted: patch shaded  <=> tan(asvf) >= V_k
    uint32_t suf[kK + 1][SOLWEIG_MASK_WORDS];  // patches at sorted sunlit positions >= i
    uint32_t pre[kK + 1][SOLWEIG_MASK_WORDS];  // patches at sorted shaded positions <  j
    // first sorted position whose sunlit threshold is >= bucket boundary i (see
    // tan_bucket): the count of thresholds <= t starts there for t in bucket i
    uint8_t sun_start[256];
};

// 256 buckets of tan(asvf): boundary i = tan(i * pi / 512) for i >= 1,
// -inf for i = 0 (the same float64 expression wherever it is evaluated).
__device__ __forceinline__ double tan_bucket_bound(int i) {
    return i == 0 ? __longlong_as_double(0xfff0000000000000ll) : tan((double)i * (kPi / 512.0));
}

// Largest i with tan_bucket_bound(i) <= t.
__device__ __forceinline__ int tan_bucket(double t) {
    int i = (int)(atan(t) * (512.0 / kPi));
    i = i < 0 ? 0 : (i > 255 ? 255 : i);
    while (i < 255 && tan_bucket_bound(i + 1) <= t) ++i;
    while (i > 0 && tan_bucket_bound(i) > t) --i;
    return i;
}

// Number of entries of the ascending a[0..n) that are <= t, starting from
// `from` = the number of entries below the bucket boundary of t.
__device__ __forceinline__ int count_le_from(const double* a, int n, int from, double t) {
    int i = from;
    while (i < n && a[i] <= t) ++i;
    return i;
}
static_assert(sizeof(DayTable) % 16 == 0, "DayTable must be a multiple of 16 bytes");

// Band boundaries (patch index) of the sky layouts the batched form supports.
template <int OPT>
struct Bands;
template <>
struct Bands<2> {  // 153 patches: 31, 30, 28, 24, 19, 13, 7, 1
    __host__ __device__ static constexpr int off(int b) {
        return b <= 0 ? 0 : b == 1 ? 31 : b == 2 ? 61 : b == 3 ? 89 : b == 4 ? 113 : b == 5 ? 132
               : b == 6 ? 145 : b == 7 ? 152 : 153;
    }
};
template <>
struct Bands<1> {  // 145 patches: 30, 30, 24, 24, 18, 12, 6, 1
    __host__ __device__ static constexpr int off(int b) {
        return b <= 0 ? 0 : b == 1 ? 30 : b == 2 ? 60 : b == 3 ? 84 : b == 4 ? 108 : b == 5 ? 126
               : b == 6 ? 138 : b == 7 ? 144 : 145;
    }
};

// Sums of wcos over the patches of m, and of wcos and wsin over those of mt.
template <int OPT>
__device__ __forceinline__ void band_sums(const uint32_t (&m)[SOLWEIG_MASK_WORDS], const uint32_t (&mt)[SOLWEIG_MASK_WORDS],
                                          const float* wcos, const float* wsin, float& mc, float& tc, float& ts) {
    mc = tc = ts = 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const int lo = Bands<OPT>::off(b), hi = Bands<OPT>::off(b + 1);
        int n = 0, nt = 0;
#pragma unroll
        for (int wd = 0; wd < SOLWEIG_MASK_WORDS; ++wd) {
            const int a = lo > wd * 32 ? lo : wd * 32;
            const int e = hi < wd * 32 + 32 ? hi : wd * 32 + 32;
            if (a < e) {
                const uint32_t mask = (e - a == 32) ? 0xffffffffu : (((1u << (e - a)) - 1u) << (a - wd * 32));
                n += __popc(m[wd] & mask);
                nt += __popc(mt[wd] & mask);
            }
        }
        const float c = wcos[b];
        mc = fmaf((float)n, c, mc);
        tc = fmaf((float)nt, c, tc);
        ts = fmaf((float)nt, wsin[b], ts);
    }
}

// Monotone integer keys of the doubles (NaN excluded).
__device__ __forceinline__ unsigned long long dkey(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double dval(unsigned long long k) {
    const unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)u);
}

// Smallest double t in [-inf, +inf] with pred(t) true, for pred monotone
// (false, then true); +inf when pred is false for every finite t.
template <typename Pred>
__device__ double first_true(Pred pred) {
    const double ninf = __longlong_as_double(0xfff0000000000000ll);
    const double pinf = __longlong_as_double(0x7ff0000000000000ll);
    if (pred(ninf)) return ninf;
    if (!pred(pinf)) return pinf;
    unsigned long long lo = dkey(ninf), hi = dkey(pinf);  // pred(lo) false, pred(hi) true
    while (hi - lo > 1) {
        const unsigned long long mid = lo + (hi - lo) / 2;
        if (pred(dval(mid))) hi = mid;
        else lo = mid;
    }
    return dval(hi);
}

// ---------------------------------------------------------------- kernels 1, 2

// Pixel of this thread in a block tile of bx x by pixels.  When the tile
// holds whole 8 x 4 (columns x rows) pieces, each warp takes one such piece
// instead of 32 pixels of one row: walk lengths of nearby pixels are alike in
// both directions, so the warp's longest walk is closer to its mean (30%
// fewer warp steps on the synthetic city); a warp's loads still cover 4 rows
// of 32-128 contiguous bytes, as many sectors as one row of 32 pixels.
__device__ __forceinline__ void warp_tile_pixel(int bx, int by, int& r, int& c) {
    if (bx % 8 == 0 && by % 4 == 0) {
        const int t = threadIdx.y * bx + threadIdx.x, w = t >> 5, l = t & 31;
        const int wx = w % (bx / 8), wy = w / (bx / 8);
        c = blockIdx.x * bx + wx * 8 + (l & 7);
        r = blockIdx.y * by + wy * 4 + (l >> 3);
    } else {
        c = blockIdx.x * bx + threadIdx.x;
        r = blockIdx.y * by + threadIdx.y;
    }
}

// TABLES: the packed geometry with the hours' tables (exits, step records of
// kpitch entries per hour, plane of H), else the rasters step by step.  Eight
// blocks per SM for both: the step-by-step walk is bound by the latency of its
// loads, and its few spills at 32 registers cost less than the occupancy of 40
// (2000 x 2000 px with relief, heights not exact in float32: 7.21 against 7.89 ms
// a day, 1000 x 1000 px 1.83 against 1.96).
template <bool TABLES>
__global__ void __launch_bounds__(256, 8) day_shadow_kernel(SolweigScene S, const SolweigHour* __restrict__ hours,
                                                            float4* __restrict__ quads,
                                                            float* __restrict__ lup_first,
                                                            const float2* __restrict__ ceiling,
                                                            const int* __restrict__ exits,
                                                            const int2* __restrict__ rec, int kpitch,
                                                            const float* __restrict__ height) {
    const int z = blockIdx.z;
    const SolweigHour& h = hours[z];
    if (!h.daytime) return;
    int r, c;
    warp_tile_pixel(blockDim.x, blockDim.y, r, c);
    const bool in = r < S.rows && c < S.cols;
    const long long n = (long long)S.rows * S.cols;
    if (!in) return;
    const float2* ceil_z = ceiling ? ceiling + z * n : nullptr;
    float* first_z = lup_first ? lup_first + z * n : nullptr;
    if constexpr (TABLES) {
        const SweepTables t{exits + (long long)z * (S.rows + S.cols), rec + (long long)z * kpitch, height, ceil_z};
        shadow_quad_pixel(S, h, r, c, quads + z * n, first_z, nullptr, &t);
    } else {
        shadow_quad_pixel(S, h, r, c, quads + z * n, first_z, ceil_z, nullptr);
    }
}

// Per daytime hour, the first-outside step of every row and column of the
// raster (first_outside), for the bounds-check-free sweep, and the hour's step
// records for the steps [0, min(steps, kmax)).  A monotone ray leaves the
// raster within max(rows, cols) steps, so kmax = max(rows, cols) + 2 covers
// every walk; a ray table that stays inside longer has its exits cut to kmax
// and sets the error flag to 3 (that hour's results invalid).
__global__ void __launch_bounds__(1024) day_ray_exits_kernel(SolweigScene S, const SolweigHour* __restrict__ hours,
                                                             int* __restrict__ exits, int2* __restrict__ rec,
                                                             int kmax, int* __restrict__ error) {
    const SolweigHour& h = hours[blockIdx.x];
    if (!h.daytime) return;
    int* ex = exits + (long long)blockIdx.x * (S.rows + S.cols);
    ray_exits_block(reinterpret_cast<const int2*>(h.ray_dxdy), h.steps, S.rows, S.cols, ex);
    ray_records_block(reinterpret_cast<const int2*>(h.ray_dxdy), h.ray_dz, min(h.steps, kmax), S.cols,
                      rec + (long long)blockIdx.x * record_pitch(kmax));
    if (h.steps <= kmax) return;
    __syncthreads();  // ex[] written by the whole block
    int cut = 0;
    for (int i = threadIdx.x; i < S.rows + S.cols; i += blockDim.x) {
        if (ex[i] > kmax) {
            ex[i] = kmax;
            cut = 1;
        }
    }
    if (cut) raise_day_flag(error, 3);
}

struct DayGvfArgs {
    int first, second, halo;
};

// gvf[z][0] = Lup GVF (ambient added), gvf[z][1] = albedo GVF, gvf[z][2] = shadow.
// nosh = albedo-without-shadow GVF: the same for every hour (walk geometry and
// albedo only), so every daytime launch writes the same values.
template <int TY, int FIRST, int SECOND, int TABLE, bool WATER>
__global__ void __launch_bounds__(32 * TY) day_gvf_kernel(SolweigScene S, const SolweigHour* __restrict__ hours,
                                                         DayGvfArgs ga, GvfTable<TABLE> tab,
                                                         const float4* __restrict__ quads,
                                                         const float* __restrict__ lup_first_all,
                                                         float* __restrict__ gvf, float* __restrict__ nosh) {
    const int z = blockIdx.z;
    const SolweigHour& h = hours[z];
    if (!h.daytime) return;
    const int bx = blockIdx.x, by = blockIdx.y;
    const long long n = (long long)S.rows * S.cols;
    const float4* quad = quads + z * n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int H = ga.halo, second = ga.second, first = ga.first;
    const int pitch = 32 + 2 * H;
    float4* tile = reinterpret_cast<float4*>(smem_raw);
    const int row0 = by * TY - H, col0 = bx * 32 - H;
    load_quad_tile(tile, pitch, TY + 2 * H, quad, S.rows, S.cols, row0, col0);
    __syncthreads();
    const int c = bx * 32 + threadIdx.x;
    const int r = by * TY + threadIdx.y;
    if (r >= S.rows || c >= S.cols) return;
    const long long p = (long long)r * S.cols + c;
    const float4* own_cell = tile + (threadIdx.y + H) * pitch + threadIdx.x + H;
    const float4 own = *own_cell;
    const double ta = h.ta;
    const float lwall = (float)(kSBC * 0.9 * pow4(h.tgwall + ta + 273.15) - kSBC * 0.9 * pow4(ta + 273.15));
    const float albedo_b = 0.2f;
    const uint32_t face = S.gvf_face[p];
    const bool own_ground = (__float_as_int(own.w) & kQuadGround) != 0;
    float lup, alb, nsh;
    if (WATER) {
        const float* lfp = lup_first_all + z * n;
        GvfScalars gs{lwall, albedo_b, first, second};
        auto sample = [&](int rr, int cc) -> float4 { return tile[(rr - row0) * pitch + (cc - col0)]; };
        auto lfirst = [&](int rr, int cc) -> float { return __ldg(&lfp[(long long)rr * S.cols + cc]); };
        const GvfSums g = gvf_walk(sample, lfirst, true, r, c, S.rows, S.cols, tab.offs, face, own, gs);
        lup = g.lup[0];
        alb = g.alb[0];
        nsh = g.nosh[0];
    } else {
        lup = alb = nsh = 0.f;
        const bool interior = row0 >= 0 && col0 >= 0 && row0 + TY + 2 * H <= S.rows && col0 + pitch <= S.cols;
        const float inv_first = 1.f / first, inv_first1 = 1.f / (first + 1);
        const float inv_second = 1.f / second, inv_second1 = 1.f / (second + 1);
#pragma unroll 1
        for (int j = 0; j < SOLWEIG_GVF_DIRECTIONS; ++j) {
            const bool fj = (face >> j) & 1u;
            const int base = j * (SECOND > 0 ? SECOND : second);
            GvfDir d;
            if (SECOND > 0) {
                d = interior ? gvf_direction_fixed<true, FIRST, SECOND>(own_cell, tab.delta + base, tab.offs + base, r,
                                                                        c, S.rows, S.cols, own_ground, lwall,
                                                                        albedo_b, fj)
                             : gvf_direction_fixed<false, FIRST, SECOND>(own_cell, tab.delta + base, tab.offs + base,
                                                                         r, c, S.rows, S.cols, own_ground, lwall,
                                                                         albedo_b, fj);
            } else {
                d = interior ? gvf_direction<true>(own_cell, tab.delta + base, tab.offs + base, r, c, S.rows, S.cols,
                                                   own_ground, first, second, inv_first, inv_first1, inv_second,
                                                   inv_second1, lwall, albedo_b, fj)
                             : gvf_direction<false>(own_cell, tab.delta + base, tab.offs + base, r, c, S.rows, S.cols,
                                                    own_ground, first, second, inv_first, inv_first1, inv_second,
                                                    inv_second1, lwall, albedo_b, fj);
            }
            lup += d.lup;
            alb += d.alb;
            nsh += d.nosh;
        }
        const float ob = own_ground ? 1.f : 0.f;
        nsh *= ob;
        lup += 18.f * (own.y * (1.f - ob));
        alb += 18.f * (own.z * (1.f - ob) * own.x);
        nsh += 18.f * (own.z * (1.f - ob));
    }
    const double ambient = kSBC * (double)S.emis[p] * pow4(ta + 273.15);
    gvf[(3 * z) * n + p] = (float)((double)(lup / 18.f) + ambient);
    gvf[(3 * z + 1) * n + p] = alb / 18.f;
    gvf[(3 * z + 2) * n + p] = own.x;
    nosh[p] = nsh / 18.f;
}

// ------------------------------------------------------------- kernels 3, 4, 5

// w[2h][k] = luminance, w[2h+1][k] = luminance * cos(alt) * omega (0 at night).
__global__ void day_weights_kernel(const SolweigSkyLayout* __restrict__ L, const SolweigHour* __restrict__ hours,
                                   int nhours, float* __restrict__ w) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 2 * nhours * kK) return;
    const int row = idx / kK, k = idx - row * kK;
    const SolweigHour& h = hours[row >> 1];
    float v = 0.f;
    if (h.daytime && k < L->patches) v = (row & 1) ? h.lum[k] * L->cos_alt[k] * L->omega[k] : h.lum[k];
    w[idx] = v;
}

// BF16 hi/lo split of scale * w [ncols][kK] into the canonical operand layout
// b[0][nb rows] (hi) and b[1][nb rows] (lo); rows >= ncols are zero.
__global__ void split_bf16_kernel(const float* __restrict__ w, int ncols, int nb, int patches,
                                  __nv_bfloat16* __restrict__ b, float scale = 1.f) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nb * kK) return;
    const int n = idx / kK, k = idx - n * kK;
    const float v = (n < ncols && k < patches) ? scale * w[n * kK + k] : 0.f;
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
    const int o = canon_off(n, k);
    b[o] = hi;
    b[nb * kK + o] = lo;
}

// One block per hour, kK threads.
__global__ void __launch_bounds__(kK) day_tables_kernel(const SolweigSkyLayout* __restrict__ L,
                                                        const SolweigHour* __restrict__ hours,
                                                        DayTable* __restrict__ tables) {
    __shared__ double ts[kK], vs[kK];
    __shared__ double sorted[kK];
    __shared__ int rank_t[kK], rank_v[kK];
    const SolweigHour& h = hours[blockIdx.x];
    DayTable& T = tables[blockIdx.x];
    const int P = L->patches;
    const int k = threadIdx.x;
    double tk = 0.0, vk = 0.0;
    if (k < P) {
        const double yi = h.yi[k], lo = L->sunlit_below[k], hi = L->shaded_above[k];
        tk = first_true([&](double t) { return !((t + yi) < lo); });
        vk = first_true([&](double t) { return (t + yi) > hi; });
        ts[k] = tk;
        vs[k] = vk;
    }
    __syncthreads();
    if (k < P) {
        int rt = 0, rv = 0;
        for (int j = 0; j < P; ++j) {
            rt += (ts[j] < tk || (ts[j] == tk && j < k)) ? 1 : 0;
            rv += (vs[j] < vk || (vs[j] == vk && j < k)) ? 1 : 0;
        }
        T.tsun[rt] = sorted[rt] = tk;
        T.vshade[rv] = vk;
        rank_t[k] = rt;
        rank_v[k] = rv;
    }
    __syncthreads();
    // position i's masks from the patches' ranks: no patch is looked up by rank,
    // so every thread reads the same ranks at once
    for (int i = k; i <= P; i += blockDim.x) {
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            uint32_t suf = 0u, pre = 0u;
            for (int b = 0; b < 32 && 32 * w + b < P; ++b) {
                suf |= (rank_t[32 * w + b] >= i ? 1u : 0u) << b;
                pre |= (rank_v[32 * w + b] < i ? 1u : 0u) << b;
            }
            T.suf[i][w] = suf;
            T.pre[i][w] = pre;
        }
    }
    if (k < 8) {
        uint32_t t = 0;
        for (int b = 0; b < 32 && k < SOLWEIG_MASK_WORDS; ++b) {
            const int kk = k * 32 + b;
            if (kk < P && h.daytime && h.lw_sun_test[kk]) t |= 1u << b;
        }
        T.loop.test[k] = t;
    }
    for (int i = k; i < 256; i += blockDim.x) {
        const double bound = tan_bucket_bound(i);
        int lo = 0, len = P;  // entries below the bound
        while (len > 0) {
            const int half = len >> 1;
            if (sorted[lo + half] < bound) {
                lo += half + 1;
                len -= half + 1;
            } else {
                len = half;
            }
        }
        T.sun_start[i] = (uint8_t)lo;
    }
    if (k < SOLWEIG_MAX_BANDS) {
        const bool ok = k < L->nbands;
        T.loop.band_down[k] = ok ? h.band_lsky[k] * L->band_omega[k] * L->band_sin[k] : 0.f;
        T.loop.band_side[k] = ok ? h.band_lsky[k] * L->band_omega[k] * L->band_cos[k] : 0.f;
    }
    if (k == 32) {
        const double tk = h.ta + 273.15;
        HourLoop& q = T.loop;
        q.lw_shade = (float)((0.9 * kSBC * pow4(tk)) / kPi);
        q.lw_sun = h.daytime ? (float)((0.9 * kSBC * pow4(h.ta + h.tgwall + 273.15)) / kPi) : 0.f;
        q.sw_shade = (float)((0.2 * h.rad_d * 0.5) / kPi);
        q.sw_sun = (float)((0.2 * (h.rad_i * h.cos_alt) + h.rad_d * 0.5) / kPi);
        q.rad_d = (float)h.rad_d;
        q.rad_g = (float)h.rad_g;
        q.rad_i_sin = (float)(h.rad_i * h.sin_alt);
        q.rad_i_cos = (float)(h.rad_i * h.cos_alt);
        q.rad_ratio = (float)(h.rad_d / h.rad_tot);
        q.wave_w = (float)h.wave_weight;
        q.tan_zen = (float)h.tan_zen;
        q.night_lup = (float)(kSBC * pow4(tk));
        q.night_lup_water = (float)(kSBC * 0.98 * pow4(h.twater + 273.15));
        q.ta = (float)h.ta;
        q.flags = (h.daytime ? kHourDay : 0u) | (h.firstdaytime ? kHourFirst : 0u) |
                  (h.wave_update ? kHourUpdate : 0u) | (h.utci_valid ? kHourUtci : 0u);
        q.pad = 0u;
        for (int i = 0; i < 7; ++i) q.utci[i] = h.utci[i];
        q.utci[7] = h.ta;
    }
}

// ------------------------------------------------------------------ kernel 6

struct GemmArgs {
    const uint32_t* masks;  // S/V bit planes [10][px]
    long long px;
    int patches;
    const __nv_bfloat16* b;  // [2][nb * kK] canonical hi, lo (combined: [4][nb * kK], then c * w hi, lo)
    int ncols, nb;
    float* out;  // [2 * ncols][px]: sky columns, then vegetation columns (combined: [ncols][px])
    int* error;
    // 1: one set of columns, sky sums plus the vegetation sums of weights
    // prescaled by c (the diffuse transmissivity of vegetation): both MMA
    // pairs accumulate into the same tensor-memory columns
    int combined;
};

size_t gemm_smem_bytes(int nb, bool combined) {
    return (size_t)2 * kABytes + (size_t)(combined ? 4 : 2) * nb * kK * 2 + 16;
}

// Expand 8 mask bits to 8 BF16 values (1.0 or 0.0) packed in a uint4.
// t = byte + (byte << 15) holds bit 2i at position 2i and bit 2i + 1 at
// position 16 + 2i, so (t >> 2i) & 0x10001 has the pair's two bits at 0 and
// 16, and times 0x3F80 (BF16 1.0) gives the two packed values.
__device__ __forceinline__ uint4 expand8(uint32_t byte) {
    const uint32_t t = byte * 0x8001u;
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = ((t >> (2 * i)) & 0x10001u) * 0x3F80u;
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// Persistent: one 128-pixel tile per iteration.  All 128 threads expand the
// tile's masks into the two A operands; thread 0 issues the MMAs (sky and
// vegetation, BF16 hi and lo weights accumulating into the same FP32
// columns) and commits them to an mbarrier; each warp then reads its 32 rows
// (pixels) of the accumulators from tensor memory and stores them.
__global__ void __launch_bounds__(kARows, 1) patch_gemm_kernel(GemmArgs g) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* a_sky = smem;
    unsigned char* a_veg = smem + kABytes;
    unsigned char* b_ops = smem + 2 * kABytes;  // hi then lo (combined: then c * w hi, lo)
    const int bbytes = g.nb * kK * 2;
    const int nbops = g.combined ? 4 : 2;
    uint64_t* bar = reinterpret_cast<uint64_t*>(b_ops + nbops * bbytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5;
    uint32_t ncols_tmem = 32;
    while (ncols_tmem < (uint32_t)((g.combined ? 1 : 2) * g.nb)) ncols_tmem <<= 1;

    {  // weights: global -> shared, 16 bytes per copy
        const uint4* src = reinterpret_cast<const uint4*>(g.b);
        uint4* dst = reinterpret_cast<uint4*>(b_ops);
        for (int i = tid; i < nbops * bbytes / 16; i += blockDim.x) dst[i] = src[i];
    }
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        tc::fence_mbar_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, ncols_tmem);
        tc::tmem_relinquish();
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const uint32_t idesc = tc::idesc_bf16_f32(kARows, g.nb);
    const uint32_t a_sky_addr = tc::smem_addr(a_sky), a_veg_addr = tc::smem_addr(a_veg);
    const uint32_t b_hi_addr = tc::smem_addr(b_ops), b_lo_addr = b_hi_addr + bbytes;
    uint32_t valid[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const int nbits = g.patches - 32 * w;
        valid[w] = nbits >= 32 ? 0xffffffffu : (nbits <= 0 ? 0u : ((1u << nbits) - 1u));
    }
    const long long ntiles = (g.px + kARows - 1) / kARows;
    uint32_t phase = 0;
    bool failed = false;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long p = t * kARows + tid;
        const bool in = p < g.px;
        // Expand this pixel's row of both A operands.
        unsigned char* row_sky = a_sky + (tid >> 3) * kSBO + (tid & 7) * 16;
        unsigned char* row_veg = a_veg + (tid >> 3) * kSBO + (tid & 7) * 16;
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            const uint32_t s = in ? g.masks[(long long)w * g.px + p] : 0u;
            const uint32_t v = in ? g.masks[(long long)(SOLWEIG_MASK_WORDS + w) * g.px + p] : 0u;
            const uint32_t sky = s & ~v & valid[w], veg = s & v & valid[w];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int chunk = w * 4 + j;
                *reinterpret_cast<uint4*>(row_sky + chunk * 128) = expand8((sky >> (8 * j)) & 0xFFu);
                *reinterpret_cast<uint4*>(row_veg + chunk * 128) = expand8((veg >> (8 * j)) & 0xFFu);
            }
        }
        tc::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
#pragma unroll 1
            for (int s = 0; s < kK / 16; ++s) {
                const uint64_t bh = tc::smem_desc(b_hi_addr + s * 256, 128, kSBO);
                const uint64_t bl = tc::smem_desc(b_lo_addr + s * 256, 128, kSBO);
                const uint64_t as = tc::smem_desc(a_sky_addr + s * 256, 128, kSBO);
                const uint64_t av = tc::smem_desc(a_veg_addr + s * 256, 128, kSBO);
                tc::mma_bf16(tmem, as, bh, idesc, s > 0);
                tc::mma_bf16(tmem, as, bl, idesc, true);
                if (g.combined) {
                    const uint64_t ch = tc::smem_desc(b_hi_addr + 2 * bbytes + s * 256, 128, kSBO);
                    const uint64_t cl = tc::smem_desc(b_hi_addr + 3 * bbytes + s * 256, 128, kSBO);
                    tc::mma_bf16(tmem, av, ch, idesc, true);
                    tc::mma_bf16(tmem, av, cl, idesc, true);
                } else {
                    tc::mma_bf16(tmem + g.nb, av, bh, idesc, s > 0);
                    tc::mma_bf16(tmem + g.nb, av, bl, idesc, true);
                }
            }
            tc::mma_commit(bar);
        }
        const bool ok = tc::mbar_wait(bar, phase, kWaitPolls);
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        phase ^= 1u;
        tc::fence_after_sync();
        const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
        if (g.combined) {
            for (int c0 = 0; c0 < g.ncols; c0 += 8) {
                float vs[8];
                tc::tmem_ld8(lane_base + c0, vs);
                tc::tmem_wait_ld();
                if (in) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (c0 + i < g.ncols) g.out[(long long)(c0 + i) * g.px + p] = vs[i];
                }
            }
        } else {
            for (int c0 = 0; c0 < g.ncols; c0 += 8) {
                float vs[8], vv[8];
                tc::tmem_ld8(lane_base + c0, vs);
                tc::tmem_ld8(lane_base + g.nb + c0, vv);
                tc::tmem_wait_ld();
                if (in) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (c0 + i < g.ncols) {
                            g.out[(long long)(c0 + i) * g.px + p] = vs[i];
                            g.out[(long long)(g.ncols + c0 + i) * g.px + p] = vv[i];
                        }
                    }
                }
            }
        }
        tc::fence_before_sync();
        __syncthreads();
    }
    if (failed) {
        if (tid == 0) raise_day_flag(g.error, 1);
        // let the MMAs of the abandoned tile finish before freeing their columns
        tc::mbar_wait(bar, phase, kWaitPolls);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, ncols_tmem);
    }
}

// Pipelined form of the combined contraction (the batched day's): two A
// stages in shared memory and two accumulators in tensor memory, 256
// threads.  While the tensor cores multiply tile i, the threads expand tile
// i + 1 into the other stage (threads 0-127 the sky masks, 128-255 the
// vegetation masks of the same 128 pixels; the mask words of tile i + 2 are
// already loading), then wait for tile i and store its sums from tensor
// memory (warp w: lanes 32 (w % 4) .. + 31, every other 8-column group from
// 8 (w / 4)).  Thread 0 issues each tile's MMAs once both of its operands
// are in shared memory and the stage's accumulator has been read out.
constexpr int kPipeThreads = 2 * kARows;

size_t gemm_pipe_smem_bytes(int nb) { return (size_t)4 * kABytes + (size_t)4 * nb * kK * 2 + 32; }

__global__ void __launch_bounds__(kPipeThreads, 1) patch_gemm_pipe_kernel(GemmArgs g) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* b_ops = smem + 4 * kABytes;  // hi, lo, c * w hi, c * w lo
    const int bbytes = g.nb * kK * 2;
    uint64_t* bar = reinterpret_cast<uint64_t*>(b_ops + 4 * bbytes);  // one per stage
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = tid & (kARows - 1);
    const bool veg_half = tid >= kARows;
    uint32_t ncols_tmem = 32;
    while (ncols_tmem < (uint32_t)(2 * g.nb)) ncols_tmem <<= 1;
    {  // weights: global -> shared, 16 bytes per copy
        const uint4* src = reinterpret_cast<const uint4*>(g.b);
        uint4* dst = reinterpret_cast<uint4*>(b_ops);
        for (int i = tid; i < 4 * bbytes / 16; i += blockDim.x) dst[i] = src[i];
    }
    if (tid == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        tc::fence_mbar_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, ncols_tmem);
        tc::tmem_relinquish();
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const uint32_t idesc = tc::idesc_bf16_f32(kARows, g.nb);
    const uint32_t b_hi_addr = tc::smem_addr(b_ops);
    uint32_t valid[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const int nbits = g.patches - 32 * w;
        valid[w] = nbits >= 32 ? 0xffffffffu : (nbits <= 0 ? 0u : ((1u << nbits) - 1u));
    }
    const long long ntiles = (g.px + kARows - 1) / kARows;
    const long long first = blockIdx.x, stride = gridDim.x;
    const long long my = first < ntiles ? (ntiles - 1 - first) / stride + 1 : 0;  // tiles of this CTA

    uint32_t sw[SOLWEIG_MASK_WORDS], vw[SOLWEIG_MASK_WORDS];
    auto load = [&](long long t) {
        const long long p = t * kARows + row;
        const bool in = p < g.px;
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            sw[w] = in ? __ldg(&g.masks[(long long)w * g.px + p]) : 0u;
            vw[w] = in ? __ldg(&g.masks[(long long)(SOLWEIG_MASK_WORDS + w) * g.px + p]) : 0u;
        }
    };
    auto expand = [&](int st) {
        unsigned char* a = smem + (2 * st + (veg_half ? 1 : 0)) * kABytes;
        unsigned char* rowp = a + (row >> 3) * kSBO + (row & 7) * 16;
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            const uint32_t m = (veg_half ? (sw[w] & vw[w]) : (sw[w] & ~vw[w])) & valid[w];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<uint4*>(rowp + (w * 4 + j) * 128) = expand8((m >> (8 * j)) & 0xFFu);
        }
    };
    auto issue = [&](int st) {  // thread 0: sky x (hi, lo) and vegetation x (c hi, c lo) into stage st
        tc::fence_after_sync();
        const uint32_t acc = tmem + (uint32_t)(st * g.nb);
        const uint32_t as0 = tc::smem_addr(smem + 2 * st * kABytes), av0 = as0 + kABytes;
#pragma unroll 1
        for (int k = 0; k < kK / 16; ++k) {
            const uint64_t bh = tc::smem_desc(b_hi_addr + k * 256, 128, kSBO);
            const uint64_t bl = tc::smem_desc(b_hi_addr + bbytes + k * 256, 128, kSBO);
            const uint64_t ch = tc::smem_desc(b_hi_addr + 2 * bbytes + k * 256, 128, kSBO);
            const uint64_t cl = tc::smem_desc(b_hi_addr + 3 * bbytes + k * 256, 128, kSBO);
            const uint64_t as = tc::smem_desc(as0 + k * 256, 128, kSBO);
            const uint64_t av = tc::smem_desc(av0 + k * 256, 128, kSBO);
            tc::mma_bf16(acc, as, bh, idesc, k > 0);
            tc::mma_bf16(acc, as, bl, idesc, true);
            tc::mma_bf16(acc, av, ch, idesc, true);
            tc::mma_bf16(acc, av, cl, idesc, true);
        }
        tc::mma_commit(&bar[st]);
    };

    uint32_t parity[2] = {0u, 0u};
    int pending = 0;  // stages with committed MMAs not yet waited for
    bool failed = false;
    if (my > 0) {
        load(first);
        expand(0);
        if (my > 1) load(first + stride);
        tc::fence_async_smem();
        __syncthreads();
        if (tid == 0) issue(0);
        pending = 1;
    }
    for (long long i = 0; i < my; ++i) {
        const int st = (int)(i & 1);
        const long long t = first + i * stride;
        if (i + 1 < my) {
            expand(st ^ 1);  // its masks were loaded one iteration ago
            if (i + 2 < my) load(t + 2 * stride);
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();  // stage st ^ 1 expanded; its accumulator read out last iteration
        if (i + 1 < my) {
            if (tid == 0) issue(st ^ 1);
            pending |= 1 << (st ^ 1);
        }
        const bool ok = tc::mbar_wait(&bar[st], parity[st], kWaitPolls);
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        parity[st] ^= 1u;
        pending &= ~(1 << st);
        tc::fence_after_sync();
        const int q = warp & 3;
        const uint32_t lane_base = tmem + (uint32_t)(st * g.nb) + ((uint32_t)(q * 32) << 16);
        const long long p = t * kARows + q * 32 + lane;
        const bool in = p < g.px;
        for (int c0 = 8 * (warp >> 2); c0 < g.ncols; c0 += 16) {
            float v[8];
            tc::tmem_ld8(lane_base + c0, v);
            tc::tmem_wait_ld();
            if (in) {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (c0 + k < g.ncols) g.out[(long long)(c0 + k) * g.px + p] = v[k];
            }
        }
    }
    if (failed) {
        if (tid == 0) raise_day_flag(g.error, 1);
        // let committed MMAs finish before their columns are freed
        for (int st = 0; st < 2; ++st)
            if (pending & (1 << st)) tc::mbar_wait(&bar[st], parity[st], kWaitPolls);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, ncols_tmem);
    }
}

// ------------------------------------------------------------------ kernel 7

struct DayRadArgs {
    const SolweigSkyLayout* layout;
    const SolweigHour* hours;
    int nhours;
    const DayTable* tables;
    const float* gvf;   // [H][3][px]
    const float* nosh;  // [px]
    const float* sums;  // [ncols][px]: sky + 0.03 x vegetation sums (luminance, luminance*cos*omega)
    int ncols;
    SolweigState state;
    SolweigOutputs out;  // base pointers; hour h at + h * hour_stride
    long long hour_stride;
    int chunk;           // hours per block (grid.y); all of them when a state or ground temperature is kept
};


__device__ __forceinline__ float* hour_plane(float* base, int hr, long long stride) {
    return base ? base + hr * stride : nullptr;
}

// Flux arithmetic of the hour loop in float32 (the hour's scalars are rounded
// once from the float64 host plan); the building split keeps its exact float64
// thresholds.  Against the per-hour form (float64 fluxes) Tmrt differs by <
// 1e-3 K (tested).
//
// What bounds it: instruction issue (77 % of the cycles) and the load/store
// unit (73 %: the hour's scalars, read through L1 without a barrier, and
// spills).  A building patch that is not sunlit is shaded, so one pass of
// popcounts over the sunlit patches serves both sums and both tests (POPC runs
// at an eighth of the issue rate), and patches exactly on a limit take a branch.
// 2000^2 day: 2.86 -> 1.90 ms.  Full occupancy (2048 resident threads per SM,
// 32 registers, spills) against 40 / 48 registers at 1536 / 1280 threads: 2.00
// against 2.08 / 2.17 ms; the scalars and mask rows as 16-byte loads, which
// live longer: 2.14 to 2.35 ms.
template <int OPT, int THREADS>
__global__ void __launch_bounds__(THREADS, 2048 / THREADS) day_radiation_kernel(SolweigScene S, DayRadArgs a) {
    __shared__ float wcos[SOLWEIG_MAX_BANDS], wsin[SOLWEIG_MAX_BANDS];
    const SolweigSkyLayout& L = *a.layout;
    if (threadIdx.x < SOLWEIG_MAX_BANDS) {
        const int b = threadIdx.x;
        const int k0 = Bands<OPT>::off(b < 8 ? b : 0);
        wcos[b] = b < L.nbands ? L.omega[k0] * L.cos_alt[k0] : 0.f;
        wsin[b] = b < L.nbands ? L.omega[k0] * L.sin_alt[k0] : 0.f;
    }
    __syncthreads();  // wcos, wsin
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)blockIdx.x * THREADS + threadIdx.x;
    const bool in = p < n;
    const long long q = in ? p : 0;  // a valid pixel for the loads of idle threads
    const SolweigOutputs& o = a.out;
    const bool need_tg = o.tg || o.tg_out || a.state.tgout1;

    // --- per-pixel static data, loaded once for the day
    uint32_t bld[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const int nbits = S.patches - 32 * w;
        const uint32_t valid = nbits >= 32 ? 0xffffffffu : (nbits <= 0 ? 0u : ((1u << nbits) - 1u));
        bld[w] = ~S.masks[(long long)w * n + q] & ~S.masks[(long long)(SOLWEIG_MASK_WORDS + w) * n + q] & valid;
    }
    uint32_t cnt_lo = 0, cnt_hi = 0;  // sky patches per band, 8 bits each
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        cnt_lo |= (uint32_t)S.sky_band_counts[(long long)b * n + q] << (8 * b);
        cnt_hi |= (uint32_t)(b + 4 < S.nbands ? S.sky_band_counts[(long long)(b + 4) * n + q] : 0) << (8 * b);
    }
    const uint8_t fl = S.flags[q];
    const bool ground = fl & 1;
    const bool water = S.has_water && (fl & 4);
    const float emis = S.emis[q];
    const float svfbuveg = S.svfbuveg[q];
    const float tan_alfa = (float)tan(S.svfalfa[q]);
    const double tan_asvf = S.tan_asvf[q];
    const int tbucket = tan_bucket(tan_asvf);
    const float oc = S.veg_sums[2 * n + q], os = S.veg_sums[3 * n + q];
    const float g_nosh = a.nosh[q];
    constexpr float ewall = 0.9f, albedo_b = 0.2f;
    constexpr float absK = 0.7f, absL = 0.95f, Fside = 0.22f, Fup = 0.06f, Fcyl = 0.28f;
    constexpr float sbc = (float)kSBC, inv_pi = (float)(1.0 / kPi);

    // sums over the vegetation and building patches: those not sunlit emit as shaded walls
    float shd_c, shd_s;
    {
        float all_c;
        band_sums<OPT>(bld, bld, wcos, wsin, all_c, shd_c, shd_s);
        shd_c += S.veg_sums[q];
        shd_s += S.veg_sums[n + q];
    }
    float st_lup = a.state.tgmap1 ? a.state.tgmap1[q] : 0.f;
    float st_tg = a.state.tgout1 ? a.state.tgout1[q] : 0.f;

    // hours of this block (blockIdx.y); the wave-delay state of the hours before them
    const int h0 = blockIdx.y * a.chunk, h1 = min(h0 + a.chunk, a.nhours);
    for (int hr = 0; hr < h0; ++hr) {
        const HourLoop& hs = a.tables[hr].loop;
        if (!(hs.flags & kHourDay)) continue;
        const float g_lup = a.gvf[(3LL * hr) * n + q];
        const float prev = (hs.flags & kHourFirst) ? g_lup : st_lup;
        st_lup = (hs.flags & kHourUpdate) ? g_lup * (1.f - hs.wave_w) + prev * hs.wave_w : prev;
    }
    for (int hr = h0; hr < h1; ++hr) {
        // the hour's table and scalars, read through L1 by every thread (no
        // shared staging, so the hour loop needs no barrier)
        const DayTable& T = a.tables[hr];
        const HourLoop& hs = T.loop;  // scalars are read where they are used: registers are short
        const uint32_t flags = hs.flags;
        const bool day = flags & kHourDay;

        // Building patches, sunlit (ref) and sunlit within the longwave's sun
        // test (hs.lw_sun): the other ones are shaded.
        float ref_c = 0.f, none_c = 0.f, lw_sun_c = 0.f, lw_sun_s = 0.f, lw_shd_c = shd_c, lw_shd_s = shd_s;
        if (day) {
            const int isun = count_le_from(T.tsun, S.patches, T.sun_start[tbucket], tan_asvf);
            // every shaded threshold is at or above its patch's sunlit one, so
            // at most isun of them are <= t, nearly always all of them
            int ishd = isun;
            while (ishd > 0 && T.vshade[ishd - 1] > tan_asvf) --ishd;
            uint32_t m[SOLWEIG_MASK_WORDS], mt[SOLWEIG_MASK_WORDS];
#pragma unroll
            for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
                m[w] = bld[w] & T.suf[isun][w];
                mt[w] = m[w] & hs.test[w];
            }
            band_sums<OPT>(m, mt, wcos, wsin, ref_c, lw_sun_c, lw_sun_s);
            lw_shd_c -= lw_sun_c;
            lw_shd_s -= lw_sun_s;
            if (ishd < isun) {  // patches exactly on the limit are neither
                float t_c, t_s;
#pragma unroll
                for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
                    m[w] = bld[w] & ~m[w] & ~T.pre[ishd][w];
                    mt[w] = m[w] & hs.test[w];
                }
                band_sums<OPT>(m, mt, wcos, wsin, none_c, t_c, t_s);
                lw_shd_c -= t_c;
                lw_shd_s -= t_s;
            }
        }
        float ld_sky = 0.f, ls_sky = 0.f;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const float cnt = (float)(((b < 4 ? cnt_lo : cnt_hi) >> (8 * (b & 3))) & 0xFFu);
            ld_sky = fmaf(hs.band_down[b], cnt, ld_sky);
            ls_sky = fmaf(hs.band_side[b], cnt, ls_sky);
        }

        float shadow = 0.f, tg = 0.f, tg_out = hs.ta;
        float kup_all = 0.f, lup_all;
        float kdown = 0.f, kside = 0.f, kside_i = 0.f, kside_d = 0.f, d_rad = 0.f;
        if (day) {
            const long long g0 = (3LL * hr) * n + q;
            const float g_lup = a.gvf[g0];
            const float g_alb = a.gvf[g0 + n];
            shadow = a.gvf[g0 + 2 * n];
            const float fsh = wedge_fsh_tan(tan_alfa, hs.tan_zen);
            const float reflected = albedo_b * (1.f - svfbuveg) * (hs.rad_g * (1.f - fsh) + hs.rad_d * fsh);
            const float base_up = hs.rad_d * svfbuveg + reflected;
            kup_all = g_alb * hs.rad_i_sin + base_up * g_nosh;
            const float prev = (flags & kHourFirst) ? g_lup : st_lup;
            lup_all = g_lup * (1.f - hs.wave_w) + prev * hs.wave_w;
            st_lup = (flags & kHourUpdate) ? lup_all : prev;
            if (need_tg) {
                // ground temperature (TsWaveDelay of Tg * shadow + Ta); not part of Tmrt
                const SolweigHour& h = a.hours[hr];
                const double amp = (double)S.tgk[q] * h.altmax + (double)S.tstart[q];
                const double phase = ((h.dectime_frac - h.snup / 24.0) /
                                      ((double)S.tmaxlst[q] / 24.0 - h.snup / 24.0)) * kPi / 2.0;
                double tgd = amp * sin(phase) * h.ci_tgg;
                if (S.landcover == 1 && tgd < 0.0) tgd = 0.0;
                if (water) tgd = h.twater - h.ta;
                tg = (float)tgd;
                const float cur = tg * shadow + hs.ta;
                const float prv = (flags & kHourFirst) ? cur : st_tg;
                tg_out = cur * (1.f - hs.wave_w) + prv * hs.wave_w;
                st_tg = (flags & kHourUpdate) ? tg_out : prv;
            }
            // the contraction already added the vegetation patches at their
            // diffuse transmissivity: sky + 0.03 x vegetation sums
            const long long s0 = 2LL * hr * n + q;
            const float lum = a.sums[s0], cw = a.sums[s0 + n];
            d_rad = hs.rad_d * lum;
            kdown = hs.rad_i_sin * shadow + d_rad + reflected;
            kside_i = shadow * hs.rad_i_cos;
            kside_d = hs.rad_ratio * cw;
            kside = kside_i + kside_d + hs.sw_sun * ref_c + hs.sw_shade * (shd_c - ref_c - none_c);
        } else {
            float lup = emis * hs.night_lup;
            if (S.landcover == 1 && (fl & 4)) lup = hs.night_lup_water;
            lup_all = lup;
        }
        const float refl = (ld_sky + lup_all) * ((1.f - ewall) * 0.5f * inv_pi);
        const float ldown = ld_sky + hs.lw_shade * lw_shd_s + hs.lw_sun * lw_sun_s + refl * os;
        const float lside = ls_sky + hs.lw_shade * lw_shd_c + hs.lw_sun * lw_sun_c + refl * oc;
        // E+S+W+N of Kup and Lup are 4x the all-direction values (see the file header).
        const float sstr = absK * (kside * Fcyl + (kdown + kup_all) * Fup + 2.f * kup_all * Fside) +
                           absL * ((ldown + lup_all) * Fup + lside * Fcyl + 2.f * lup_all * Fside);
        const float tmrt = sqrtf(sqrtf(sstr * (1.f / (absL * sbc)))) - 273.2f;
        if (in) {
            const long long at = hr * a.hour_stride + p;
            if (o.tmrt) o.tmrt[at] = tmrt;
            if (o.utci) {
                float u = __int_as_float(0x7fc00000);
                if (ground) {
                    u = utci_eval(hs.utci, (double)tmrt, hs.utci[7], flags & kHourUtci);
                }
                o.utci[at] = u;
            }
            if (o.kdown) o.kdown[at] = kdown;
            if (o.kup) o.kup[at] = kup_all;
            if (o.ldown) o.ldown[at] = ldown;
            if (o.lup) o.lup[at] = lup_all;
            if (o.lside) o.lside[at] = lside;
            if (o.kside_i) o.kside_i[at] = kside_i;
            if (o.kside_d) o.kside_d[at] = kside_d;
            if (o.kside) o.kside[at] = kside;
            if (o.d_rad) o.d_rad[at] = d_rad;
            if (o.shadow) o.shadow[at] = shadow;
            if (o.tg) o.tg[at] = tg;
            if (o.tg_out) o.tg_out[at] = tg_out;
        }
    }
    if (in) {
        if (a.state.tgmap1) a.state.tgmap1[p] = st_lup;
        if (a.state.tgout1) a.state.tgout1[p] = st_tg;
    }
}

// ------------------------------------------------------------------ host side

inline long long align256(long long x) { return (x + 255) & ~255LL; }

struct DayWork {
    long long quads, lup_first, gvf, nosh, sums, wf32, bw, tables, error, tilemax, walks, dict, exits, rec, total;
};

DayWork day_work_layout(int rows, int cols, int nhours, bool water) {
    DayWork w{};
    const long long px = (long long)rows * cols;
    const int ncols = 2 * nhours;
    const int nb = (ncols + 15) / 16 * 16;
    long long o = 0;
    // the error flag pair first: the same place for every raster size, so the
    // days of differently sized tiles sharing one buffer share its sticky word
    w.error = o; o = align256(o + 16);
    w.quads = o; o = align256(o + 16LL * px * nhours);
    w.lup_first = o; o = align256(o + (water ? 4LL * px * nhours : 0));
    w.gvf = o; o = align256(o + 12LL * px * nhours);
    w.nosh = o; o = align256(o + 4LL * px);
    w.sums = o; o = align256(o + 4LL * px * 2 * ncols);
    w.wf32 = o; o = align256(o + 4LL * ncols * kK);
    w.bw = o; o = align256(o + 2LL * 4 * nb * kK);
    w.tables = o; o = align256(o + (long long)sizeof(DayTable) * nhours);
    // per 16 x 16 tile maxima of the heights (ceil(rows/16) * ceil(cols/16)
    // floats, bounded here from the pixel count alone: <= px/256 + (rows + cols)/16 + 1)
    w.tilemax = o; o = align256(o + 4LL * (px / 256 + (px + 1) / 16 + 4));
    // GVF walk words, for scenes that come without them: in the patch-sum region
    // behind the samples' codes, free until the contraction (72 bytes per pixel that
    // most scenes bring along); days too short for that (four hours and less) keep a
    // region of their own
    const long long words = water ? 0 : 4LL * walk_words(rows, cols);
    const long long codes = align256(4LL * px * ((nhours + kWkHours - 1) / kWkHours));
    w.walks = w.sums + codes;
    if (codes + words > 4LL * px * 2 * ncols) { w.walks = o; o = align256(o + words); }
    // the tiles' distinct samples
    w.dict = o;
    o = align256(o + (water ? 0 : walk_words(rows, cols) / kWkTileWords * 8 * kWkDictKeys * ((nhours + 3) / kWkHours)));
    // per hour the first-outside steps of the rows and columns, and the ray's step records
    w.exits = o; o = align256(o + 4LL * (rows + cols) * nhours);
    w.rec = o; o = align256(o + 8LL * record_pitch(std::max(rows, cols) + 2) * nhours);
    w.total = o;
    return w;
}

// For kernels that always take the same size (allow_shared for the others).
void set_smem_attr(const void* kernel, size_t bytes) {
    // Not a stream operation; cheap after the first call.
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int TABLE>
void fill_day_table(GvfTable<TABLE>& tab, const int32_t* dxdy, int second, int pitch) {
    for (int i = 0; i < SOLWEIG_GVF_DIRECTIONS * second; ++i) {
        tab.offs[i] = make_int2(dxdy[2 * i], dxdy[2 * i + 1]);
        tab.delta[i] = dxdy[2 * i] * pitch + dxdy[2 * i + 1];
    }
}

int launch_gvf_walks(const SolweigScene& S, const int32_t* gvf_dxdy, int second, uint32_t* hits, uint32_t* walks,
                     float* nosh, cudaStream_t st) {
    GvfTable<kWkMaxSteps> tab;
    fill_day_table(tab, gvf_dxdy, second, kWkMaxWidth);
    const size_t smem = gvf_walks_smem_bytes();
    set_smem_attr((const void*)gvf_walks_kernel, smem);
    dim3 grid(blocks_for(S.cols, kWkTile), blocks_for(S.rows, kWkTile));
    gvf_walks_kernel<<<grid, kWkPixels, smem, st>>>(S, second, tab, hits, walks, nosh);
    SOLWEIG_CHECK_LAUNCH("gvf_walks_kernel");
    return SOLWEIG_OK;
}

// Arguments of the walk-word kernels for a table of walks; false unless every
// walk starts at its pixel.
bool day_walk_args(const int32_t* gvf_dxdy, int second, DayWalkArgs* wa) {
    wa->second = second;
    wa->halo = second - 1;
    wa->width = kWkTile + 2 * wa->halo;
    wa->magic = (uint32_t)((0x100000000ull + wa->width - 1) / wa->width);
    return walk_offsets(gvf_dxdy, second, wa->width, &wa->at);
}

// The GVF planes of every daytime hour from the walk words in wa: codes takes
// 4 bytes per pixel and pass of four hours.
int launch_day_walk(const SolweigScene& S, const SolweigHour* hours, int nhours, DayWalkArgs& wa, const float4* quads,
                    uint32_t* codes, unsigned long long* dict, float* gvf, const float* nosh_in, float* nosh,
                    cudaStream_t st) {
    wa.codes = codes;
    wa.dict = dict;
    const dim3 grid(blocks_for(S.cols, kWkTile), blocks_for(S.rows, kWkTile), (nhours + kWkHours - 1) / kWkHours);
    gvf_codes_kernel<<<grid, kWkCodeThreads, 0, st>>>(S.rows, S.cols, hours, nhours, quads, codes, dict, gvf, nosh_in,
                                                      nosh);
    SOLWEIG_CHECK_LAUNCH("gvf_codes_kernel");
    const size_t smem = day_walk_smem_bytes(wa.width);
    allow_shared((const void*)day_gvf_walk_kernel);
    day_gvf_walk_kernel<<<grid, kWkThreads, smem, st>>>(S, hours, nhours, wa, quads, gvf);
    SOLWEIG_CHECK_LAUNCH("day_gvf_walk_kernel");
    return SOLWEIG_OK;
}

template <int TY, int FIRST, int SECOND, int TABLE>
void launch_day_gvf_ty(const SolweigScene& S, const SolweigHour* hours, int nhours, const DayGvfArgs& ga,
                       const GvfTable<TABLE>& tab, const float4* quads, const float* lup_first, float* gvf,
                       float* nosh, cudaStream_t st) {
    const size_t smem = sizeof(float4) * (size_t)(32 + 2 * ga.halo) * (TY + 2 * ga.halo);
    dim3 grid(blocks_for(S.cols, 32), blocks_for(S.rows, TY), nhours);
    if (S.has_water) {
        auto k = day_gvf_kernel<TY, FIRST, SECOND, TABLE, true>;
        allow_shared((const void*)k);
        k<<<grid, dim3(32, TY), smem, st>>>(S, hours, ga, tab, quads, lup_first, gvf, nosh);
    } else {
        auto k = day_gvf_kernel<TY, FIRST, SECOND, TABLE, false>;
        allow_shared((const void*)k);
        k<<<grid, dim3(32, TY), smem, st>>>(S, hours, ga, tab, quads, lup_first, gvf, nosh);
    }
}

template <int FIRST, int SECOND, int TABLE>
void launch_day_gvf(int ty, const SolweigScene& S, const SolweigHour* hours, int nhours, const DayGvfArgs& ga,
                    const GvfTable<TABLE>& tab, const float4* quads, const float* lup_first, float* gvf,
                    float* nosh, cudaStream_t st) {
    if (ty == 4) launch_day_gvf_ty<4, FIRST, SECOND, TABLE>(S, hours, nhours, ga, tab, quads, lup_first, gvf, nosh, st);
    else if (ty == 16) launch_day_gvf_ty<16, FIRST, SECOND, TABLE>(S, hours, nhours, ga, tab, quads, lup_first, gvf, nosh, st);
    else launch_day_gvf_ty<8, FIRST, SECOND, TABLE>(S, hours, nhours, ga, tab, quads, lup_first, gvf, nosh, st);
}

int launch_gemm(const uint32_t* masks, long long px, int patches, const __nv_bfloat16* b, int ncols, int nb,
                float* out, int* error, cudaStream_t st, int ctas_per_sm = 0, bool combined = false) {
    if (combined && gemm_pipe_smem_bytes(nb) <= 227 * 1024) {
        // the pipelined kernel: one CTA per SM (its shared memory)
        const size_t smem = gemm_pipe_smem_bytes(nb);
        allow_shared((const void*)patch_gemm_pipe_kernel);
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const long long ntiles = (px + kARows - 1) / kARows;
        long long grid = sms > 0 ? sms : 1;
        if (grid > ntiles) grid = ntiles;
        GemmArgs g{masks, px, patches, b, ncols, nb, out, error, 1};
        patch_gemm_pipe_kernel<<<(unsigned)grid, kPipeThreads, smem, st>>>(g);
        SOLWEIG_CHECK_LAUNCH("patch_gemm_pipe_kernel");
        return SOLWEIG_OK;
    }
    const size_t smem = gemm_smem_bytes(nb, combined);
    SOLWEIG_CHECK_ARG(smem <= 227 * 1024, "patch contraction: %d weight columns need %zu bytes of shared memory",
                      ncols, smem);
    allow_shared((const void*)patch_gemm_kernel);
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, patch_gemm_kernel, kARows, smem);
    if (per_sm < 1) per_sm = 1;
    if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
    const long long ntiles = (px + kARows - 1) / kARows;
    long long grid = (long long)sms * per_sm;
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) grid = 1;
    GemmArgs g{masks, px, patches, b, ncols, nb, out, error, combined ? 1 : 0};
    patch_gemm_kernel<<<(unsigned)grid, kARows, smem, st>>>(g);
    SOLWEIG_CHECK_LAUNCH("patch_gemm_kernel");
    return SOLWEIG_OK;
}

}  // namespace

}  // namespace solweig
