// Per-pixel radiation epilogue of one hour: patch sums, fluxes, Tmrt, UTCI.
//
// Restates the cyl = 1, anisotropic-sky path of Solweig_2022a_calc
// (src/umep_solweig.py:50-372) with Kside_veg_v2022a (:666-911),
// Lcyl_v2022a / define_patch_characteristics (:946-1028, :1205-1356),
// Kup_veg_2015a (:915-927), TsWaveDelay_2015a (:1633-1652),
// cylindric_wedge (:383-426) and the Tmrt expression (:345-360); the UTCI
// polynomial of src/kernels/utci.cu evaluated in (Tmrt - Ta) with the seven
// hourly coefficients computed on the host.
//
// Patch sums use the packed visibility words.  Within one altitude band the
// solid angle and cos/sin of the altitude are the same for every patch, so
// every static sum is a per-band popcount (computed once after the SVF); only
// the Perez luminance weights (sky / vegetation patches) and the sunlit/shaded
// split of building patches change every hour.
#pragma once
#include "common.cuh"

namespace solweig {

// One patch of an hour, read by a whole warp at once (four 16-byte loads).
struct alignas(16) PatchRow {
    float lum, lum_cw;    // Perez luminance; times cos(alt) * omega
    float wcos, wsin;     // omega * cos(alt), omega * sin(alt)
    float card[4];        // longwave E,S,W,N cosines (0 = not in that half)
    float lsky_side;      // sky longwave of the patch on a vertical surface
    uint32_t lw_test;     // longwave sun test
    double x_off;         // yi (added to tan(asvf))
    double lo, hi;        // sunlit below, shaded above
};

// Values of one hour staged in shared memory.
struct PatchSmem {
    PatchRow row[SOLWEIG_MAX_PATCHES];
    float band_down[SOLWEIG_MAX_BANDS];  // sky longwave per visible patch, horizontal
    float band_side[SOLWEIG_MAX_BANDS];  // sky longwave per visible patch, vertical
    int patches;
};

__device__ __forceinline__ void stage_patches(PatchSmem& sm, const SolweigSkyLayout& L,
                                              const SolweigHour& h) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int nt = blockDim.x * blockDim.y;
    for (int k = tid; k < L.patches; k += nt) {
        PatchRow& row = sm.row[k];
        row.lum = h.lum[k];
        row.lum_cw = h.lum[k] * L.cos_alt[k] * L.omega[k];
        row.wcos = L.omega[k] * L.cos_alt[k];
        row.wsin = L.omega[k] * L.sin_alt[k];
        for (int d = 0; d < 4; ++d) row.card[d] = L.cardinal[d][k];
        const int b = L.band_of_patch[k];
        row.lsky_side = h.band_lsky[b] * L.band_omega[b] * L.band_cos[b];
        row.lw_test = h.lw_sun_test[k];
        row.x_off = h.yi[k];
        row.lo = L.sunlit_below[k];
        row.hi = L.shaded_above[k];
    }
    if (tid < SOLWEIG_MAX_BANDS) {
        const bool ok = tid < L.nbands;
        sm.band_down[tid] = ok ? h.band_lsky[tid] * L.band_omega[tid] * L.band_sin[tid] : 0.f;
        sm.band_side[tid] = ok ? h.band_lsky[tid] * L.band_omega[tid] * L.band_cos[tid] : 0.f;
    }
    if (tid == 0) sm.patches = L.patches;
}

// Results of the per-pixel patch loop (weights, before hour scaling).
struct PatchSums {
    float lum_sky, lum_veg;        // sum of luminance over sky / vegetation patches
    float cw_sky, cw_veg;          // same, times cos(alt)*omega
    float sw_sun, sw_shade;        // omega*cos over building patches sunlit / shaded (shortwave)
    float lw_sun_c, lw_shade_c;    // omega*cos, building patches sunlit / shaded (longwave)
    float lw_sun_s, lw_shade_s;    // omega*sin, same
    float card_sky[4], card_veg[4], card_sun[4], card_shade[4], card_obst[4];
};

// Every lane takes the patches in the same order, so a patch's values are four
// broadcast loads and the sums conditional additions.  A loop per class over
// each pixel's own bits (sky, vegetation, building, obstruction), with a load
// per value and lanes at different patches, took 155 us of an hour of 400 x 360
// pixels with the cardinal terms; this takes 70 us (four blocks per SM; three:
// 74, five: 86).  What bounds it is instruction issue.
template <bool Cardinal>
__device__ __forceinline__ PatchSums patch_loop(const PatchSmem& sm, const uint32_t* S,
                                                const uint32_t* V, double tan_asvf, bool daytime) {
    PatchSums ps{};
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const int kn = min(32, sm.patches - 32 * w);
#pragma unroll 1
        for (int i = 0; i < kn; ++i) {
            const PatchRow& row = sm.row[32 * w + i];
            const float4 l = *reinterpret_cast<const float4*>(&row.lum);
            const bool s = (S[w] >> i) & 1u, v = (V[w] >> i) & 1u;
            const bool sky = s && !v, veg = s && v, bld = !s && !v;
            if (sky) {
                ps.lum_sky += l.x;
                ps.cw_sky += l.y;
            }
            if (veg) {
                ps.lum_veg += l.x;
                ps.cw_veg += l.y;
            }
            const float4 c = *reinterpret_cast<const float4*>(row.card);
            const float card[4] = {c.x, c.y, c.z, c.w};
            if (bld) {
                const double x = tan_asvf + row.x_off;
                const bool sunlit = x < row.lo, shaded = x > row.hi;
                const bool test = row.lw_test != 0;
                const bool lsun = test && sunlit, lshade = !test || shaded;
                if (sunlit) ps.sw_sun += l.z;
                if (shaded) ps.sw_shade += l.z;
                if (lsun) {
                    ps.lw_sun_c += l.z;
                    ps.lw_sun_s += l.w;
                }
                if (lshade) {
                    ps.lw_shade_c += l.z;
                    ps.lw_shade_s += l.w;
                }
                if (Cardinal) {
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        if (lsun) ps.card_sun[d] += l.z * card[d];
                        if (lshade) ps.card_shade[d] += l.z * card[d];
                    }
                }
            }
            if (Cardinal) {
                const float side = row.lsky_side;
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    if (sky) ps.card_sky[d] += side * card[d];
                    if (v) ps.card_veg[d] += l.z * card[d];
                    if (!sky) ps.card_obst[d] += l.z * card[d];
                }
            }
        }
    }
    if (!daytime) ps.lum_sky = ps.cw_sky = ps.lum_veg = ps.cw_veg = ps.sw_sun = ps.sw_shade = 0.f;
    return ps;
}

__device__ __forceinline__ float utci_eval(const double* c, double tmrt, double ta, int valid) {
    if (!valid || tmrt <= -999.0) return -999.0f;
    const double d = tmrt - ta;
    double u = c[6];
#pragma unroll
    for (int i = 5; i >= 0; --i) u = u * d + c[i];
    return (float)u;
}

// Fraction of shaded wall, cylindric_wedge (NaN -> 0.5), from ta = tan(svfalfa).
// With h = 2 / (tan(svfalfa) tan(zenith)) the wedge's b and q satisfy b / q = h,
// so the angle of its arc, above h = 1, is atan(t) with t^2 = h^2 - 1/4, the
// arc's (sin - phi cos) / (1 - cos) is (t - phi) (1 + sqrt(1 + t^2)) / t^2, and
// b drops out of the ratio: one arc tangent, two divisions and two roots
// instead of six divisions, three roots and trigonometric functions of phi.
// Radiation of a 2000^2 day (float32): 2.00 -> 1.90 ms; reverse pass of 500 x 500
// pixels (float64): 2.26 -> 2.10 ms.  Its error against longer precision is no
// larger in either type.
template <typename T>
__device__ __forceinline__ T wedge_fsh_tan(T ta, T tan_zen) {
    const T h = T(2) / (ta * tan_zen);
    T arc = T(0);
    if (h > T(1)) {
        const T tt = h * h - T(0.25), t = sqrt(tt);
        arc = (T(1) - h) * ((t - atan(t)) * (T(1) + sqrt(tt + T(1))) / tt);
    }
    const T fsh = T(1) - (h + arc) * T(1.0 / kPi);
    return isnan(fsh) ? T(0.5) : fsh;
}

__device__ __forceinline__ double wedge_fsh(double svfalfa, double tan_zen) {
    return wedge_fsh_tan(tan(svfalfa), tan_zen);
}

}  // namespace solweig
