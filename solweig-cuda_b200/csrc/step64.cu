// The hourly SOLWEIG step with float64 radiation: the reference's
// `--dtype float64` switch (run.py:27), which recompiles its gvf.cu,
// shortwave.cu, longwave.cu and flux.cu kernels with Real = double
// (src/runtime.py:43-49, src/model.py:382-620, :731).
//
// Hours in launches of their own (grid.z) as far as the scratch reaches; only
// the wave delay runs through them in order.
//
//  K1 step64_fields_kernel     shadow sweep (the float32 step's walk: the same
//                              masks) and the per-pixel GVF inputs in float64:
//                              shadow, Lup excess (before and after the water
//                              override), albedo * shadow, the sunlit-wall bits
//  K2 step64_gvf_kernel        the 18 search directions of gvf_2018a /
//                              sunonsurface_2018a (src/umep_solweig.py:583-663,
//                              :1400-1600)
//  K3 step64_wave_kernel       wave delay of the ground planes, hour by hour
//  K4 step64_radiation_kernel  F_sh, Kup, Kdown, Kside and the anisotropic
//                              longwave (Kside_veg_v2022a :666-911,
//                              Lcyl_v2022a :946-1028), Tmrt (:345-360) and UTCI
//
// Everything per pixel is float64, with products grouped as the reference's
// expressions group them.  Two regroupings save most of the work and add
// fewer roundings than they replace: the steps after a walk's end, which all
// add the same, come as one product, and sums of solid-angle weights over a
// set of patches, equal within an altitude band, are band counts times the
// band's weight.  The means over a walk's steps are products with rounded
// reciprocals (true divisions: 2.00 instead of 1.67 ms per day of 300 x 280 px).
// Against longer precision the sum of a pixel's 18 walks has an rms error of 1.05
// to 1.15e-16 for 22 steps (1.13 to 1.78e-16 with one addition per step and
// divisions), 1.08 to 1.15 for 11 steps (1.06 to 1.15), 1.08 to 1.16 for 6 (1.04
// to 1.15).  This file is compiled with --fmad=false (as the reference
// compiles its kernels, src/runtime.py:11), so no multiply-add is contracted.
// UTCI is evaluated from the float32-rounded Tmrt and air temperature, as
// utci_calculator casts its inputs (src/utci.py:8-12).
#include "gvf_words.cuh"
#include "hour.cuh"
#include "radiation.cuh"

namespace solweig {

constexpr int kStep64BX = 32, kStep64BY = 4;
static_assert(SOLWEIG_SCRATCH64_PLANES % 2 == 0, "an hour's planes keep the next hour's sample pairs aligned");

// Scratch planes of an hour [SOLWEIG_SCRATCH64_PLANES][pixels] float64.
enum Scratch64 : int {
    kS64Sample = 0,    // 2 planes as pairs: Lup excess after the water override, albedo * shadow
    kS64Shadow = 2,    // sh - (1 - vegsh)(1 - psi)
    kS64LupFirst = 3,  // Lup excess before the override (first search direction)
    kS64Bits = 4,      // one byte per pixel: 1 = sunlit wall
    kS64Gvf = 5,       // 15 planes: Lup, albedo, albedo without shadow x (all, E, S, W, N); the last
                       // five of a launch's first daytime hour serve all its hours
};

struct GvfOffsets64 {
    int2 offs[SOLWEIG_GVF_DIRECTIONS * SOLWEIG_GVF_MAX_STEPS];
    long long ahead[SOLWEIG_GVF_DIRECTIONS * SOLWEIG_GVF_MAX_STEPS];  // pixels from the walking one
};

__device__ __forceinline__ double* hour_scratch(double* sc, long long n) {
    return sc + (long long)blockIdx.z * SOLWEIG_SCRATCH64_PLANES * n;
}

// First daytime hour of a launch, whose scratch holds the albedo-without-shadow
// planes of all of them.
__device__ __forceinline__ int first_day_hour(const SolweigHour* __restrict__ hours) {
    int z = 0;
    while (!hours[z].daytime) ++z;
    return z;
}

__global__ void __launch_bounds__(kStep64BX* kStep64BY) step64_fields_kernel(
    SolweigScene S, const SolweigHour* __restrict__ hours, double* __restrict__ scratch, bool pairs) {
    const SolweigHour& h = hours[blockIdx.z];
    if (!h.daytime) return;
    const int c = blockIdx.x * kStep64BX + threadIdx.x;
    const int r = blockIdx.y * kStep64BY + threadIdx.y;
    if (r >= S.rows || c >= S.cols) return;
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)r * S.cols + c;
    double* sc = hour_scratch(scratch, n);
    const double a = S.dsm[p];
    const double wall = S.walls[p];
    const uint8_t fl = S.flags[p];
    const int2* ray = reinterpret_cast<const int2*>(h.ray_dxdy);
    // the packed geometry, where the scene has it, gives the same masks from one load per step
    const ShadowResult s =
        S.geo32 ? shadow_walk_geo(GeoF32x4{reinterpret_cast<const float4*>(S.geo32)}, S.rows, S.cols, r, c, a,
                                  S.vegdem[p], (fl & 2) != 0, wall, ray, h.ray_dz, h.steps, S.hmax, true)
                : shadow_walk_geo(GeoF64{S.dsm, S.vegdem, S.vegdem2}, S.rows, S.cols, r, c, a, S.vegdem[p],
                                  (fl & 2) != 0, wall, ray, h.ray_dz, h.steps, S.hmax, true);
    // Wall planes of shadowingfunction_wallheight_23 (only the sunlit-wall
    // test of the GVF reads them); see quad_from_walk for the no-division test.
    const double wallbol = wall > 0.0 ? 1.0 : 0.0;
    const double facesh = self_shadow_face(S.aspect[p], wallbol, h.ray_low, h.ray_high, h.ray_middle);
    double wallsun = wall - (s.f - a);
    if (wallsun < 0.0) wallsun = 0.0;
    if (facesh == 1.0) wallsun = 0.0;
    const double wallsh = wall - wallsun;
    double wallshve = (s.topmax - a) * (s.veg ? 1.0 : 0.0) * wallbol - wallsh;
    if (wallshve < 0.0) wallshve = 0.0;
    if (wallshve > wall) wallshve = wall;
    wallsun = wallsun - wallshve;
    if (wallsun < 0.0) wallsun = 0.0;
    const bool sunwall = (fl & 1) && wall > 0.0 && wallsun == wall;
    const double sh = s.shadowed ? 0.0 : 1.0;
    const double vegsh = s.veg ? 0.0 : 1.0;
    const double shadow = sh - (1.0 - vegsh) * (1.0 - h.psi);
    double tg = ground_tg(S, h, p);
    const double emis = S.emis[p];
    if (S.has_water) {
        sc[kS64LupFirst * n + p] = lup_excess(emis, tg, shadow, h.ta);
        if (fl & 4) tg = h.twater - h.ta;
    }
    sc[kS64Shadow * n + p] = shadow;
    const double2 v = make_double2(lup_excess(emis, tg, shadow, h.ta), (double)S.alb[p] * shadow);
    double* sample = sc + kS64Sample * n + 2 * p;
    if (pairs) {
        *reinterpret_cast<double2*>(sample) = v;
    } else {
        sample[0] = v.x;
        sample[1] = v.y;
    }
    reinterpret_cast<uint8_t*>(sc + kS64Bits * n)[p] = sunwall;
}

// Ground view factors of the daytime hours into the scratch GVF planes (the
// step reads no gvfSum / gvfNorm, so the shadow sums are not kept).  A walk
// adds its samples in order up to the first building; past it (or past the
// raster's edge, where the last sample repeats) every step adds the same
// terms, which come as one product.  WALK: the scene's walk words (kWalkWords)
// give the walk's length and the wall pixels it meets, so a step only reads its
// sample; its walk lengths (kWalkHits) leave a sunlit-wall byte per step; else
// the ground bits are read first.  The albedo without shadow is the same in
// every hour of a launch: NOSH (the first daytime hour) sums its five planes.
// PAIRS: a sample is one 16-byte load, else (scratch on an odd multiple of 8
// bytes, with the ground bits alone) two.
// What bounds it: the latency of the samples' loads through L1 and the FP64
// pipe; 64 registers (8 blocks per SM).  17 hours of 300 x 280 pixels: 1.13 ->
// 0.68 ms against lengths, a byte and an albedo per step and hour (5 or 6 blocks
// per SM: 0.78, 0.76 against 0.75 before the offsets came ready).
enum Walk64 { kWalkGround, kWalkHits, kWalkWords };

template <int WALK, bool NOSH, bool PAIRS>
__device__ __forceinline__ void gvf64_pixel(const SolweigScene& S, const SolweigHour& h, const GvfOffsets64& tab,
                                            int first, int second, int r, int c, double* __restrict__ sc) {
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)r * S.cols + c;
    const double* samples = sc + kS64Sample * n + 2 * p;
    auto sample = [&](long long ahead) {
        const double* at = samples + 2 * ahead;
        return PAIRS ? *reinterpret_cast<const double2*>(at) : make_double2(at[0], at[1]);
    };
    const double* lup1p = sc + kS64LupFirst * n + p;
    const uint8_t* sunp = reinterpret_cast<const uint8_t*>(sc + kS64Bits * n) + p;
    const uint8_t* flagp = S.flags + p;
    const float* albp = S.alb + p;
    const double ta = h.ta;
    constexpr double ewall = 0.9, albedo_b = 0.2;
    const double lwall = kSBC * ewall * pow4(h.tgwall + ta + 273.15) - kSBC * ewall * pow4(ta + 273.15);
    const bool own_ground = *flagp & 1;
    const double own_b = own_ground ? 1.0 : 0.0, ground = 1.0 - own_b;
    const double own_sh = sc[kS64Shadow * n + p], own_alb = (double)*albp;
    const double own_lup = sample(0).x;
    const uint32_t face = S.gvf_face[p];
    const double dfirst = first, dsecond = second;
    const double by_first = 1.0 / dfirst, by_first1 = 1.0 / (dfirst + 1.0);
    const double by_second = 1.0 / dsecond, by_second1 = 1.0 / (dsecond + 1.0);
    double lup[5] = {0, 0, 0, 0, 0}, alb[5] = {0, 0, 0, 0, 0}, nosh[5] = {0, 0, 0, 0, 0};
    uint32_t code = 0u;
    const uint32_t* words = WALK == kWalkWords ? S.gvf_walks + walk_word_at(r, c, S.cols) : nullptr;
    for (int j = 0; j < SOLWEIG_GVF_DIRECTIONS; ++j) {
        const int2* o = tab.offs + j * second;
        const long long* ahead = tab.ahead + j * second;
        // lim samples are read; hit = first step with a building (second: none)
        int lim, hit;
        uint32_t walls = 0u;
        if (WALK == kWalkWords) {
            const uint32_t word = __ldg(words + j * kWkPixels);
            lim = min((int)((word >> kWkLimShift) & 31u), second);
            hit = word & kWkFrozen ? second : lim;
            walls = word & kWkWallBits;
        } else if (!own_ground) {
            lim = hit = 0;
        } else if (WALK == kWalkHits) {
            if (j % 5 == 0) code = S.gvf_hits[(long long)(j / 5) * n + p];
            lim = min((int)(code & 31u), second);
            hit = code & 32u ? second : lim;
            code >>= 6;
        } else {
            lim = hit = second;
            for (int k = 0; k < second; ++k) {
                if (!in_raster(r + o[k].x, c + o[k].y, S.rows, S.cols)) {
                    lim = k;
                    if (k == 0) hit = 0;  // nothing seen: no ground
                    break;
                }
                if (!(__ldg(flagp + ahead[k]) & 1)) {
                    lim = hit = k;
                    break;
                }
            }
        }
        double s_lup = 0.0, s_albsh = 0.0, s_alb = 0.0, n_lup = 0.0, n_albsh = 0.0, n_alb = 0.0;
        double2 t = make_double2(0.0, 0.0);
        double t_alb = 0.0;
        int sun = second;  // first step showing a sunlit wall
        if (WALK == kWalkWords) {
            for (; walls; walls &= walls - 1u) {
                const int k = __ffs((int)walls) - 1;
                if (sunp[ahead[k]]) {
                    sun = k;
                    break;
                }
            }
        }
        for (int k = 0; k < lim; ++k) {
            const long long q = ahead[k];
            t = sample(q);
            if (WALK != kWalkWords) {
                if (j == 0 && S.has_water) t.x = lup1p[q];
                if (sunp[q] && sun == second) sun = k;
            }
            s_lup += t.x;
            s_albsh += t.y;
            if (NOSH) {
                t_alb = (double)__ldg(albp + q);
                s_alb += t_alb;
            }
            if (k + 1 <= first) {
                n_lup = s_lup; n_albsh = s_albsh; n_alb = s_alb;
            }
        }
        if (hit > lim) {  // the walk left the raster: its last sample repeats
            const double rest = hit - lim;
            s_lup += rest * t.x;
            s_albsh += rest * t.y;
            s_alb += rest * t_alb;
            if (first > lim) {
                const double near = first - lim;
                n_lup += near * t.x; n_albsh += near * t.y; n_alb += near * t_alb;
            }
        }
        const int n_wall = second - hit, n_wall_near = first > hit ? first - hit : 0;   // steps behind a building
        const int n_sun = second - sun, n_sun_near = first > sun ? first - sun : 0;     // steps with a sunlit wall seen
        const bool sun_near = n_sun_near > 0, wall_near = n_wall_near > 0;
        const bool sun_far = n_sun > 0, wall_far = n_wall > 0;
        // keep == 1 of the reference: every step saw a sunlit wall and the
        // wall face is turned away from this direction.
        const double w_sun = n_sun == second && ((face >> j) & 1u) ? 0.0 : (double)n_sun;
        const double lup1 = sun_near ? (n_sun_near * lwall + n_lup) * by_first1 : n_lup * by_first;
        const double lup2 = sun_far ? (w_sun * lwall + s_lup) * by_second1 : s_lup * by_second;
        const double alb1 = sun_near ? (n_sun_near * albedo_b + n_albsh) * by_first1 : n_albsh * by_first;
        const double alb2 = sun_far ? (w_sun * albedo_b + s_albsh) * by_second1 : s_albsh * by_second;
        const double d_lup = (lup1 * 0.5 + lup2 * 0.4) / 0.9 + own_lup * ground;
        const double d_alb = (alb1 * 0.5 + alb2 * 0.4) / 0.9 + own_alb * ground * own_sh;
        double d_nosh = 0.0;
        if (NOSH) {
            const double nosh1 = wall_near ? (n_wall_near * albedo_b + n_alb) * by_first1 : n_alb * by_first;
            const double nosh2 = wall_far ? (n_wall * albedo_b + s_alb) * by_second : s_alb * by_second;
            d_nosh = ((nosh1 * 0.5 + nosh2 * 0.4) / 0.9) * own_b + own_alb * ground;
        }
        const unsigned groups = gvf_direction_groups(j);
#pragma unroll
        for (int g = 0; g < 5; ++g)
            if (groups & (1u << g)) {
                lup[g] += d_lup;
                alb[g] += d_alb;
                if (NOSH) nosh[g] += d_nosh;
            }
    }
    const double ambient = kSBC * (double)S.emis[p] * pow4(ta + 273.15);
    double* gvf = sc + kS64Gvf * n;
#pragma unroll
    for (int g = 0; g < 5; ++g) {
        const double div = g == 0 ? 18.0 : 9.0;
        gvf[(long long)g * n + p] = lup[g] / div + ambient;
        gvf[(long long)(5 + g) * n + p] = alb[g] / div;
        if (NOSH) gvf[(long long)(10 + g) * n + p] = nosh[g] / div;
    }
}

template <int WALK, bool PAIRS>
__global__ void __launch_bounds__(kStep64BX* kStep64BY, 8) step64_gvf_kernel(
    SolweigScene S, const SolweigHour* __restrict__ hours, const __grid_constant__ GvfOffsets64 tab, int first,
    int second, double* __restrict__ scratch) {
    const SolweigHour& h = hours[blockIdx.z];
    if (!h.daytime) return;
    const int c = blockIdx.x * kStep64BX + threadIdx.x;
    const int r = blockIdx.y * kStep64BY + threadIdx.y;
    if (r >= S.rows || c >= S.cols) return;
    double* sc = hour_scratch(scratch, (long long)S.rows * S.cols);
    if (first_day_hour(hours) == (int)blockIdx.z) gvf64_pixel<WALK, true, PAIRS>(S, h, tab, first, second, r, c, sc);
    else gvf64_pixel<WALK, false, PAIRS>(S, h, tab, first, second, r, c, sc);
}

// Per-patch and per-band values of one hour (float64), staged in shared memory.
struct PatchSmem64 {
    double lum[SOLWEIG_MAX_PATCHES];      // Perez luminance (diffuse sum)
    double lum_chi[SOLWEIG_MAX_PATCHES];  // lum * radD / rad_tot * cos(alt) * omega (side diffuse)
    double x_off[SOLWEIG_MAX_PATCHES], lo[SOLWEIG_MAX_PATCHES], hi[SOLWEIG_MAX_PATCHES];
    double lsky[SOLWEIG_MAX_PATCHES];     // sky emittance (cardinal planes)
    double card[4][SOLWEIG_MAX_PATCHES];  // omega * cos(alt) * cardinal cosine
    double wcos[SOLWEIG_MAX_BANDS], wsin[SOLWEIG_MAX_BANDS];      // omega * cos(alt), omega * sin(alt)
    double sky_down[SOLWEIG_MAX_BANDS], sky_side[SOLWEIG_MAX_BANDS];
    uint32_t band[SOLWEIG_MAX_BANDS][SOLWEIG_MASK_WORDS];         // patches of a band
    uint32_t valid[SOLWEIG_MASK_WORDS], test[SOLWEIG_MASK_WORDS]; // patches; longwave sun test
};

__device__ __forceinline__ double* state64_plane(const SolweigState64& st, int d) {
    return d == 0 ? st.tgmap1 : d == 1 ? st.tgmap1e : d == 2 ? st.tgmap1s : d == 3 ? st.tgmap1w : st.tgmap1n;
}

__device__ __forceinline__ double* kside64_plane(const SolweigOutputs64& o, int d) {
    return d == 1 ? o.keast : d == 2 ? o.ksouth : d == 3 ? o.kwest : o.knorth;
}

__device__ __forceinline__ double* lcard64_plane(const SolweigOutputs64& o, int d) {
    return d == 1 ? o.least : d == 2 ? o.lsouth : d == 3 ? o.lwest : o.lnorth;
}

// TsWaveDelay_2015a (src/umep_solweig.py:1633-1652) of one pixel: returns the
// delayed value and updates the carried state.
__device__ __forceinline__ double wave_delay64(const SolweigHour& h, double current, double& state) {
    const double prev = h.firstdaytime ? current : state;
    const double w = h.wave_weight;
    const double out = current * (1.0 - w) + prev * w;
    state = h.wave_update ? out : prev;
    return out;
}

__device__ __forceinline__ void stage_patches64(PatchSmem64& sm, const SolweigSkyLayout& L, const SolweigSky64& K,
                                                const SolweigHour& h, const SolweigHour64& h64) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int nt = blockDim.x * blockDim.y;
    for (int k = tid; k < SOLWEIG_MAX_PATCHES; k += nt) {
        const bool ok = k < L.patches;
        const bool lit = ok && h.daytime;
        sm.lum[k] = lit ? h64.lum[k] : 0.0;
        sm.lum_chi[k] = lit ? (h64.lum[k] * h.rad_d) / h.rad_tot * K.cos_alt[k] * K.omega[k] : 0.0;
        sm.x_off[k] = ok ? h.yi[k] : 0.0;
        sm.lo[k] = ok ? L.sunlit_below[k] : 0.0;
        sm.hi[k] = ok ? L.shaded_above[k] : 0.0;
        sm.lsky[k] = ok ? h64.band_lsky[L.band_of_patch[k]] : 0.0;
        for (int d = 0; d < 4; ++d) sm.card[d][k] = ok ? K.omega[k] * K.cos_alt[k] * K.cardinal[d][k] : 0.0;
    }
    for (int i = tid; i < (SOLWEIG_MAX_BANDS + 2) * SOLWEIG_MASK_WORDS; i += nt) {
        const int b = i / SOLWEIG_MASK_WORDS, w = i % SOLWEIG_MASK_WORDS;
        uint32_t m = 0u;
        for (int k = 0; k < 32 && 32 * w + k < L.patches; ++k) {
            const int q = 32 * w + k;
            const bool in = b < SOLWEIG_MAX_BANDS ? L.band_of_patch[q] == b
                            : b == SOLWEIG_MAX_BANDS ? true : h.daytime && h.lw_sun_test[q];
            m |= (in ? 1u : 0u) << k;
        }
        if (b < SOLWEIG_MAX_BANDS) sm.band[b][w] = m;
        else if (b == SOLWEIG_MAX_BANDS) sm.valid[w] = m;
        else sm.test[w] = m;
    }
    for (int b = tid; b < SOLWEIG_MAX_BANDS; b += nt) {
        int k = 0;  // a patch of the band: its altitude and solid angle are the band's
        while (k < L.patches && L.band_of_patch[k] != b) ++k;
        const bool ok = k < L.patches;
        sm.wcos[b] = ok ? K.omega[k] * K.cos_alt[k] : 0.0;
        sm.wsin[b] = ok ? K.omega[k] * K.sin_alt[k] : 0.0;
        sm.sky_down[b] = ok ? (h64.band_lsky[b] * K.omega[k]) * K.sin_alt[k] : 0.0;
        sm.sky_side[b] = ok ? (h64.band_lsky[b] * K.omega[k]) * K.cos_alt[k] : 0.0;
    }
}

// Sums of omega * cos(alt) and omega * sin(alt) over the patches of m.
__device__ __forceinline__ double2 weight_sums(const PatchSmem64& sm, const uint32_t (&m)[SOLWEIG_MASK_WORDS]) {
    double2 s = make_double2(0.0, 0.0);
    for (int b = 0; b < SOLWEIG_MAX_BANDS; ++b) {
        int count = 0;
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w)
            if (sm.band[b][w]) count += __popc(m[w] & sm.band[b][w]);
        s.x += count * sm.wcos[b];
        s.y += count * sm.wsin[b];
    }
    return s;
}

// Wave delay of one pixel through `count` hours: the five Lup planes in place
// in the scratch, the ground temperature planes and the carried state.
__global__ void __launch_bounds__(128) step64_wave_kernel(SolweigScene S, const SolweigHour* __restrict__ hours,
                                                          int count, SolweigState64 st, SolweigOutputs64 out,
                                                          long long stride, double* __restrict__ scratch) {
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint8_t fl = S.flags[p];
    double state[5], tg_state = st.tgout1[p];
#pragma unroll
    for (int d = 0; d < 5; ++d) state[d] = state64_plane(st, d)[p];
    for (int i = 0; i < count; ++i) {
        const SolweigHour& h = hours[i];
        double tg = 0.0, tg_out = h.ta;
        if (h.daytime) {
            double* sc = scratch + (long long)i * SOLWEIG_SCRATCH64_PLANES * n;
            double* lup = sc + kS64Gvf * n + p;
#pragma unroll
            for (int d = 0; d < 5; ++d) lup[(long long)d * n] = wave_delay64(h, lup[(long long)d * n], state[d]);
            tg = ground_tg(S, h, p);
            if (S.has_water && (fl & 4)) tg = h.twater - h.ta;
            tg_out = wave_delay64(h, tg * sc[kS64Shadow * n + p] + h.ta, tg_state);
        }
        if (out.tg) out.tg[i * stride + p] = tg;
        if (out.tg_out) out.tg_out[i * stride + p] = tg_out;
    }
#pragma unroll
    for (int d = 0; d < 5; ++d) state64_plane(st, d)[p] = state[d];
    st.tgout1[p] = tg_state;
}

// One pixel-hour of the radiation epilogue in float64 (Lup already delayed).
// Expressions follow Kup_veg_2015a, Kside_veg_v2022a, Lcyl_v2022a and the Tmrt
// expression; a 0/1 mask factor of the reference is a branch or a patch set
// here.  Only the luminance sums and the sunlit / shaded tests go through the
// patches one by one; CARDINAL: also the E, S, W, N longwave planes.
template <bool CARDINAL>
__global__ void __launch_bounds__(kStep64BX* kStep64BY, 6) step64_radiation_kernel(
    SolweigScene S, const double* __restrict__ svfbuveg, const SolweigSkyLayout* __restrict__ Lp,
    const SolweigSky64* __restrict__ Kp, const SolweigHour* __restrict__ hours,
    const SolweigHour64* __restrict__ hours64, SolweigOutputs64 out, long long stride, double* __restrict__ scratch) {
    const SolweigHour& h = hours[blockIdx.z];
    const SolweigSkyLayout& L = *Lp;
    __shared__ PatchSmem64 sm;
    stage_patches64(sm, L, *Kp, h, hours64[blockIdx.z]);
    __syncthreads();
    const int c = blockIdx.x * kStep64BX + threadIdx.x;
    const int r = blockIdx.y * kStep64BY + threadIdx.y;
    if (r >= S.rows || c >= S.cols) return;
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)r * S.cols + c;
    const double* sc = hour_scratch(scratch, n);
    const bool day = h.daytime != 0;
    const uint8_t fl = S.flags[p];
    const double ta = h.ta;
    const double emis = S.emis[p];
    constexpr double ewall = 0.9, albedo_b = 0.2;
    constexpr double absK = 0.7, absL = 0.95, Fside = 0.22, Fup = 0.06, Fcyl = 0.28;
    // patches: sky, vegetation (in front or behind), building; building ones sunlit / shaded
    uint32_t sky[SOLWEIG_MASK_WORDS], veg[SOLWEIG_MASK_WORDS], bld[SOLWEIG_MASK_WORDS], open[SOLWEIG_MASK_WORDS];
    uint32_t sun[SOLWEIG_MASK_WORDS], shd[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const uint32_t s = S.masks[(long long)w * n + p] & sm.valid[w];
        const uint32_t v = S.masks[(long long)(SOLWEIG_MASK_WORDS + w) * n + p] & sm.valid[w];
        open[w] = s;
        sky[w] = s & ~v;
        veg[w] = v;
        bld[w] = ~s & ~v & sm.valid[w];
        sun[w] = shd[w] = 0u;
    }
    const double tan_asvf = S.tan_asvf[p];
    const int P = L.patches;
    // Diffuse sky: diffsh is 1 for sky patches, the float32 value of
    // 1 - (1 - transmissivity) for vegetation in front of the sky, 0 behind buildings.
    const double dveg = Kp->diffsh_veg;
    double lum = 0.0, chi = 0.0;
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const int kn = min(32, P - 32 * w);
        if (day && open[w]) {
            for (int k = 0; k < kn; ++k) {
                const double f = (open[w] >> k) & 1u ? ((veg[w] >> k) & 1u ? dveg : 1.0) : 0.0;
                lum += f * sm.lum[32 * w + k];
                chi += f * sm.lum_chi[32 * w + k];
            }
        }
        // in the night the tests only matter where the longwave looks at the sun, which is nowhere
        if (day && bld[w]) {
            for (int k = 0; k < kn; ++k) {
                const double x = tan_asvf + sm.x_off[32 * w + k];
                sun[w] |= (x < sm.lo[32 * w + k] ? 1u : 0u) << k;
                shd[w] |= (x > sm.hi[32 * w + k] ? 1u : 0u) << k;
            }
            sun[w] &= bld[w];
            shd[w] &= bld[w];
        }
    }
    const double2 c_veg = weight_sums(sm, veg);

    double shadow = 0.0;
    double kup[5] = {0, 0, 0, 0, 0}, lup[5];
    double kdown = 0.0, kside_i = 0.0, kside_d = 0.0, kside = 0.0, d_rad = 0.0;
    if (day) {
        shadow = sc[kS64Shadow * n + p];
        const double fsh = wedge_fsh(S.svfalfa[p], h.tan_zen);
        const double svb = svfbuveg[p];
        const double reflected = albedo_b * (1.0 - svb) * (h.rad_g * (1.0 - fsh) + h.rad_d * fsh);
        const double base = h.rad_d * svb + reflected;
        const double* gvf = sc + kS64Gvf * n;
        const double* nosh =
            scratch + ((long long)first_day_hour(hours) * SOLWEIG_SCRATCH64_PLANES + kS64Gvf + 10) * n;
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            kup[d] = gvf[(long long)(5 + d) * n + p] * h.rad_i * h.sin_alt + base * nosh[(long long)d * n + p];
            lup[d] = gvf[(long long)d * n + p];
        }
        d_rad = lum * h.rad_d;
        kdown = h.rad_i * shadow * h.sin_alt + d_rad + reflected;
        kside_i = shadow * h.rad_i * h.cos_alt;
        kside_d = chi;
        const double sun_surf = (albedo_b * (h.rad_i * h.cos_alt) + (h.rad_d * 0.5)) / kPi;
        const double shade_surf = (albedo_b * h.rad_d * 0.5) / kPi;
        kside = kside_i + kside_d + sun_surf * weight_sums(sm, sun).x + shade_surf * weight_sums(sm, shd).x +
                shade_surf * c_veg.x;
    } else {
        double l = kSBC * emis * pow4(0.0 + ta + 0.0 + 273.15);
        if (S.landcover == 1 && (fl & 4)) l = kSBC * 0.98 * pow4(h.twater + 273.15);
#pragma unroll
        for (int d = 0; d < 5; ++d) lup[d] = l;
    }

    // Anisotropic longwave (Lcyl_v2022a with define_patch_characteristics):
    // a building patch the sun test does not reach is shaded.
    const double tk4 = pow4(ta + 273.15);
    const double veg_surf = (ewall * kSBC * tk4) / kPi;
    const double sun_surf = (ewall * kSBC * pow4(ta + h.tgwall + 273.15)) / kPi;
    const double shade_surf = veg_surf;
    uint32_t obst[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        sun[w] &= sm.test[w];
        shd[w] = (shd[w] & sm.test[w]) | (bld[w] & ~sm.test[w]);
        obst[w] = sm.valid[w] & ~sky[w];
    }
    const double2 c_sun = weight_sums(sm, sun), c_shd = weight_sums(sm, shd), c_obst = weight_sums(sm, obst);
    double d_sky = 0.0, s_sky = 0.0;
    for (int b = 0; b < SOLWEIG_MAX_BANDS; ++b) {
        int count = 0;
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w)
            if (sm.band[b][w]) count += __popc(sky[w] & sm.band[b][w]);
        d_sky += count * sm.sky_down[b];
        s_sky += count * sm.sky_side[b];
    }
    const double refl = ((d_sky + lup[0]) * (1.0 - ewall) * 0.5) / kPi;
    const double lside = s_sky + veg_surf * c_veg.x + shade_surf * c_shd.x + sun_surf * c_sun.x + refl * c_obst.x;
    const double ldown = d_sky + veg_surf * c_veg.y + shade_surf * c_shd.y + sun_surf * c_sun.y + refl * c_obst.y;
    double card[4] = {0, 0, 0, 0};
    if (CARDINAL) {
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            const int kn = min(32, P - 32 * w);
            for (int k = 0; k < kn; ++k) {
                const uint32_t bit = 1u << k;
                double l;  // what the patch emits and reflects
                if (sky[w] & bit) l = sm.lsky[32 * w + k];
                else l = ((veg[w] & bit) ? veg_surf : (sun[w] & bit) ? sun_surf : (shd[w] & bit) ? shade_surf : 0.0) +
                         refl;
#pragma unroll
                for (int d = 0; d < 4; ++d) card[d] += l * sm.card[d][32 * w + k];
            }
        }
    }

    // Tmrt, cylinder with anisotropic sky: Keast.. = KupE..*0.5 and
    // Least.. = LupE..*0.5 enter the sums before the patch terms are added.
    const double ksum = kup[4] * 0.5 + kup[1] * 0.5 + kup[2] * 0.5 + kup[3] * 0.5;
    const double lsum = lup[4] * 0.5 + lup[1] * 0.5 + lup[2] * 0.5 + lup[3] * 0.5;
    const double sstr = absK * (kside * Fcyl + (kdown + kup[0]) * Fup + ksum * Fside) +
                        absL * ((ldown + lup[0]) * Fup + lside * Fcyl + lsum * Fside);
    const double tmrt = sqrt(sqrt(sstr / (absL * kSBC))) - 273.2;
    const long long at = blockIdx.z * stride + p;
    if (out.tmrt) out.tmrt[at] = tmrt;
    if (out.utci)
        out.utci[at] = (fl & 1) ? utci_eval(h.utci, (double)(float)tmrt, (double)(float)ta, h.utci_valid)
                                : __int_as_float(0x7fc00000);
    if (out.kdown) out.kdown[at] = kdown;
    if (out.kup) out.kup[at] = kup[0];
    if (out.ldown) out.ldown[at] = ldown;
    if (out.lup) out.lup[at] = lup[0];
    if (out.shadow) out.shadow[at] = shadow;
    // Cardinal planes: E, S, W, N = direction 1..4 of the GVF; the longwave
    // patch terms are accumulated as E, S, W, N (card[0..3]).
#pragma unroll
    for (int d = 1; d < 5; ++d) {
        double* ko = kside64_plane(out, d);
        if (ko) ko[at] = kup[d] * 0.5;
        double* lo = lcard64_plane(out, d);
        if (CARDINAL && lo) lo[at] = lup[d] * 0.5 + card[d - 1];
    }
    if (out.kside_i) out.kside_i[at] = kside_i;
    if (out.kside_d) out.kside_d[at] = kside_d;
    if (out.kside) out.kside[at] = kside;
    if (out.lside) out.lside[at] = lside;
    if (out.d_rad) out.d_rad[at] = d_rad;
}

}  // namespace solweig

using namespace solweig;

extern "C" int solweig_step64_hours(const SolweigScene* scene, const double* svfbuveg, const SolweigSkyLayout* layout,
                                    const SolweigSky64* sky, const SolweigHour* hours, const SolweigHour64* hours64,
                                    int hour, int count, const SolweigState64* state, const SolweigOutputs64* out,
                                    int64_t hour_stride, const int32_t* gvf_dxdy, int first_steps, int second_steps,
                                    double* scratch, void* stream) {
    SOLWEIG_CHECK_ARG(scene && svfbuveg && layout && sky && hours && hours64 && hour >= 0 && state && out &&
                          gvf_dxdy && scratch,
                      "solweig_step64: null argument");
    SOLWEIG_CHECK_ARG(count >= 1 && count <= 65535, "solweig_step64: %d hours", count);
    const SolweigScene& S = *scene;
    SOLWEIG_CHECK_ARG(S.rows > 0 && S.cols > 0 && S.rows < (1 << 20) && S.cols < (1 << 20),
                      "solweig_step64: bad scene shape %dx%d", S.rows, S.cols);
    SOLWEIG_CHECK_ARG(S.dsm && S.vegdem && S.vegdem2 && S.walls && S.aspect && S.flags && S.alb && S.emis &&
                          S.tgk && S.tstart && S.tmaxlst && S.svfalfa && S.tan_asvf && S.masks && S.gvf_face,
                      "solweig_step64: scene has a null array");
    SOLWEIG_CHECK_ARG(state->tgmap1 && state->tgmap1e && state->tgmap1s && state->tgmap1w && state->tgmap1n &&
                          state->tgout1,
                      "solweig_step64: state has a null plane");
    SOLWEIG_CHECK_ARG(second_steps >= 1 && second_steps <= SOLWEIG_GVF_MAX_STEPS && first_steps >= 1 &&
                          first_steps <= second_steps,
                      "solweig_step64: GVF steps first=%d second=%d", first_steps, second_steps);
    GvfOffsets64 tab;
    for (int i = 0; i < SOLWEIG_GVF_DIRECTIONS * second_steps; ++i) {
        tab.offs[i] = make_int2(gvf_dxdy[2 * i], gvf_dxdy[2 * i + 1]);
        tab.ahead[i] = (long long)gvf_dxdy[2 * i] * S.cols + gvf_dxdy[2 * i + 1];
    }
    // the scene's walk lengths and words, if they are those of this table
    const bool hits = S.gvf_hits && first_steps == 1 && second_steps <= 22 && !S.has_water &&
                      S.gvf_table == gvf_table_key(gvf_dxdy, first_steps, second_steps);
    const bool words = hits && S.gvf_walks && ((uintptr_t)S.gvf_walks & 3) == 0;
    const bool pairs = ((uintptr_t)scratch & 15) == 0;  // an hour's planes are an even number of doubles
    cudaStream_t st = as_stream(stream);
    const SolweigHour* hr = hours + hour;
    dim3 block(kStep64BX, kStep64BY);
    dim3 grid(blocks_for(S.cols, kStep64BX), blocks_for(S.rows, kStep64BY), count);
    step64_fields_kernel<<<grid, block, 0, st>>>(S, hr, scratch, pairs);
    SOLWEIG_CHECK_LAUNCH("step64_fields_kernel");
    auto gvf = !pairs ? step64_gvf_kernel<kWalkGround, false>
               : words ? step64_gvf_kernel<kWalkWords, true>
               : hits  ? step64_gvf_kernel<kWalkHits, true>
                       : step64_gvf_kernel<kWalkGround, true>;
    gvf<<<grid, block, 0, st>>>(S, hr, tab, first_steps, second_steps, scratch);
    SOLWEIG_CHECK_LAUNCH("step64_gvf_kernel");
    step64_wave_kernel<<<blocks_for((long long)S.rows * S.cols, 128), 128, 0, st>>>(S, hr, count, *state, *out,
                                                                                   hour_stride, scratch);
    SOLWEIG_CHECK_LAUNCH("step64_wave_kernel");
    if (out->least || out->lsouth || out->lwest || out->lnorth)
        step64_radiation_kernel<true><<<grid, block, 0, st>>>(S, svfbuveg, layout, sky, hr, hours64 + hour, *out,
                                                              hour_stride, scratch);
    else
        step64_radiation_kernel<false><<<grid, block, 0, st>>>(S, svfbuveg, layout, sky, hr, hours64 + hour, *out,
                                                               hour_stride, scratch);
    SOLWEIG_CHECK_LAUNCH("step64_radiation_kernel");
    return SOLWEIG_OK;
}

extern "C" int solweig_step64(const SolweigScene* scene, const double* svfbuveg, const SolweigSkyLayout* layout,
                              const SolweigSky64* sky, const SolweigHour* hours, const SolweigHour64* hours64,
                              int hour, const SolweigState64* state, const SolweigOutputs64* out,
                              const int32_t* gvf_dxdy, int first_steps, int second_steps, double* scratch,
                              void* stream) {
    return solweig_step64_hours(scene, svfbuveg, layout, sky, hours, hours64, hour, 1, state, out, 0, gvf_dxdy,
                                first_steps, second_steps, scratch, stream);
}
