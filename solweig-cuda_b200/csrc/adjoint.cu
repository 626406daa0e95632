// Gradient of a day's mean UTCI (or Tmrt) with the shadow and SVF masks held
// fixed: a hand-written reverse pass of the batched day.
//
// Parameters (per pixel): ground albedo a, ground emissivity e and the
// direct-beam transmissivity t of vegetation, which replaces the hour's psi
// in shadow = sh - (1 - vegsh)(1 - t) (src/umep_solweig.py:171 of the step;
// the diffuse-sky transmissivity 0.03 of the SVF stays fixed).  Forcing: the
// kernels return the partials of the objective with respect to the per-hour
// scalars the device consumes (Ta, direct and diffuse radiation, their
// normaliser, CI_TgG, the wall temperature, the 8 band sky emittances, the 7
// UTCI coefficients and, through the contraction, the Perez luminances);
// the host chains them with the Jacobian of its FP64 hour plan.
//
//  forward (also re-run by the backward: per-hour recomputation, nothing is
//  kept from the forward call)
//    the day's sweep stage    masks of every hour (shadow sweep, psi of the hour)
//    param_quads_kernel       GVF field quads from the parameters: shadow with t,
//                             Lup with e, albedo a
//    gvf_walks_kernel         walk words and the albedo-without-shadow plane
//    day_gvf_walk_kernel      all-direction GVF of every hour (scene copy with e, a)
//    contraction              luminance sums (mask-only, parameter-free)
//    grad_radiation_kernel    per pixel: forward over the hours (states kept),
//                             objective, then backward over the hours, each
//                             hour's fluxes recomputed from its inputs
//  backward
//    gvf_transpose_kernel     transpose of the GVF walk: every pixel gathers the
//                             adjoints of the GVF planes of the pixels whose
//                             walks read it (of Lup, albedo*shadow and albedo)
//    param_grad_kernel        per pixel: chain to a, e, t; Ta / CI_TgG partials
//    lum_grad_kernel          mask-transpose sums for the Perez luminances
#include "day_kernels.cuh"

namespace solweig {
namespace {

enum HourField {
    kGTa = 0,
    kGRadI,
    kGRadD,
    kGRadTot,
    kGCiTgg,
    kGTgwall,
    kGBand0,                   // 8 band sky emittances
    kGUtci0 = kGBand0 + 8,     // 7 UTCI coefficients
    kGFields = kGUtci0 + 7
};
static_assert(kGFields == SOLWEIG_GRAD_HOUR_FIELDS, "hour field count");

constexpr double kEwall = 0.9, kAlbB = 0.2;
constexpr double kVegTransmissivity = 0.03;  // of the canopy for diffuse radiation
constexpr double kAbsK = 0.7, kAbsL = 0.95, kFside = 0.22, kFup = 0.06, kFcyl = 0.28;

struct GradPtrs {
    const float* alb;
    const float* emis;
    const float* tau;
    const uint8_t* sv;      // [H][px] bit0 sh (sunlit of buildings), bit1 vegsh (no canopy shade)
    const float4* quads;    // [H][px] parameter quads
    const float* gvf;       // [H][3][px]
    const float* nosh;      // [px]
    const float* sums;      // [2 * ncols][px]
    int ncols;
    // adjoint outputs of the radiation pass
    float* lam_gl;          // [H][px]
    float* lam_ga;          // [H][px]
    float* lam_gn;          // [px], summed over the hours
    float* lam_s;           // [H][px]  own shadow
    float* lam_sums;        // [H][2][px] of the sky's sums (the canopy's: times kVegTransmissivity)
    float* d_emis_direct;   // [px]
    double* hour_grad;      // [H][kGFields]
    double* daily;          // [px] objective per pixel (forward)
    const float* weights;   // [px] dJ/d daily (backward)
    int objective;          // 0 UTCI, 1 Tmrt
};

// ------------------------------------------------------------------ quads

// Decode the building / canopy masks from the forward quads (shadow value with
// the hour's psi) and rebuild the quads with the parameters.
__global__ void param_quads_kernel(SolweigScene S, const SolweigHour* __restrict__ hours, int nhours,
                                   const float4* __restrict__ q0, float4* __restrict__ q1,
                                   uint8_t* __restrict__ sv, const float* __restrict__ alb,
                                   const float* __restrict__ emis, const float* __restrict__ tau,
                                   const int* __restrict__ error) {
    const long long n = (long long)S.rows * S.cols;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n * nhours) return;
    const int hr = (int)(idx / n);
    const long long p = idx - (long long)hr * n;
    const SolweigHour& h = hours[hr];
    if (!h.daytime) return;
    const float4 q = q0[idx];
    const float s0 = q.x;
    if (*error) {  // a ray longer than the sweep's records: no result rather than a wrong one
        const float nan = __int_as_float(0x7fffffff);
        sv[idx] = 0;
        q1[idx] = make_float4(nan, nan, nan, q.w);
        return;
    }
    // shadow = (float)(sh - (1 - vegsh)(1 - psi)): 1, psi, 0 or psi - 1
    int sh, vegsh;
    if (s0 == 1.0f) { sh = 1; vegsh = 1; }
    else if (s0 == 0.0f) { sh = 0; vegsh = 1; }
    else if (s0 == (float)(1.0 - (1.0 - h.psi))) { sh = 1; vegsh = 0; }
    else { sh = 0; vegsh = 0; }
    sv[idx] = (uint8_t)(sh | (vegsh << 1));
    const double t = tau[p];
    const double shadow = (double)(float)((double)sh - (1.0 - vegsh) * (1.0 - t));
    const double tg = ground_tg(S, h, p);
    const float lup = (float)lup_excess((double)emis[p], tg, shadow, h.ta);
    q1[idx] = make_float4((float)shadow, lup, alb[p], q.w);
}

// ------------------------------------------------------------------ radiation

struct HourIn {
    bool day;
    double s, gl, ga;
    double Ls, Cs, Lv, Cv;
};

// What the passes read of one hour, from the plan once per block.
struct HourTerms {
    double sky_down[8], sky_side[8];  // band radiances times omega sin, omega cos
    double direct_up, beam;           // direct radiation on the ground, on a wall
    double ratio;                     // diffuse radiation over its normaliser
    double sw_shade, sw_sun, lw_shade, lw_sun;
    double ambient, d_ambient;        // SBC Tk^4 and its derivative
    double d_shade, d_sun;            // derivatives of lw_shade, lw_sun
};

__device__ void hour_terms(const SolweigHour& h, const SolweigSkyLayout& L, HourTerms& t) {
    const double ta = h.ta, tk = ta + 273.15, tw = ta + h.tgwall + 273.15;
    for (int b = 0; b < 8; ++b) {
        const double bl = b < L.nbands ? (double)h.band_lsky[b] * L.band_omega[b] : 0.0;
        t.sky_down[b] = bl * L.band_sin[b];
        t.sky_side[b] = bl * L.band_cos[b];
    }
    t.direct_up = h.rad_i * h.sin_alt;
    t.beam = h.rad_i * h.cos_alt;
    t.ratio = h.rad_d / h.rad_tot;
    t.sw_shade = (kAlbB * h.rad_d * 0.5) / kPi;
    t.sw_sun = (kAlbB * t.beam + h.rad_d * 0.5) / kPi;
    t.ambient = kSBC * pow4(tk);
    t.d_ambient = kSBC * 4.0 * tk * tk * tk;
    t.lw_shade = (kEwall * kSBC * pow4(tk)) / kPi;
    t.lw_sun = h.daytime ? (kEwall * kSBC * pow4(tw)) / kPi : 0.0;
    t.d_shade = kEwall * kSBC * 4.0 * tk * tk * tk / kPi;
    t.d_sun = kEwall * kSBC * 4.0 * tw * tw * tw / kPi;
}

// Everything of one pixel-hour the reverse pass needs beyond the state.
struct PixelStatics {
    uint32_t bld[SOLWEIG_MASK_WORDS];
    uint32_t cnt_lo, cnt_hi;  // sky patches per band, 8 bits each
    uint32_t bld_lo, bld_hi;  // building patches per band
    bool ground;
    int tbucket;
    double emis, svfbuveg, tan_alfa, tan_asvf, vc, vs, oc, os, gn;
    __device__ double cnt(int b) const {
        // exact: the byte in the last place of 2^52
        const int n = (int)(((b < 4 ? cnt_lo : cnt_hi) >> (8 * (b & 3))) & 0xFFu);
        return __hiloint2double(0x43300000, n) - __hiloint2double(0x43300000, 0);
    }
};

// Patches of m and of mt in band b.
template <int OPT>
__device__ __forceinline__ void band_counts(const uint32_t (&m)[SOLWEIG_MASK_WORDS],
                                            const uint32_t (&mt)[SOLWEIG_MASK_WORDS], int b, int& n, int& nt) {
    const int lo = Bands<OPT>::off(b), hi = Bands<OPT>::off(b + 1);
    n = nt = 0;
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
}

struct BuildingTerms {
    float sws, swh, lsu_c, lsu_s, lsh_c, lsh_s;
};

// Sums over the building patches of a daytime hour: sunlit (sws) and shaded
// (swh) ones, and those with the longwave's sun test (lsu, lsh).  One pass of
// popcounts over the sunlit patches: the others are shaded, except patches
// exactly on a limit, which take a branch.
template <int OPT>
__device__ __forceinline__ BuildingTerms building_terms(const DayTable& T, const PixelStatics& ps, int P, bool day,
                                                        const float* wcos, const float* wsin) {
    const int isun = day ? count_le_from(T.tsun, P, T.sun_start[ps.tbucket], ps.tan_asvf) : P;
    int ishd = isun;  // every shaded threshold is at or above its patch's sunlit one
    while (day && ishd > 0 && T.vshade[ishd - 1] > ps.tan_asvf) --ishd;
    uint32_t m[SOLWEIG_MASK_WORDS], mt[SOLWEIG_MASK_WORDS], none[SOLWEIG_MASK_WORDS], nonet[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        m[w] = day ? ps.bld[w] & T.suf[isun][w] : 0u;
        mt[w] = m[w] & T.loop.test[w];
        none[w] = nonet[w] = 0u;
    }
    const bool limits = ishd < isun;
    if (limits) {
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            none[w] = ps.bld[w] & ~m[w] & ~T.pre[ishd][w];
            nonet[w] = none[w] & T.loop.test[w];
        }
    }
    BuildingTerms t{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        int n, nt, off = 0, offt = 0;
        band_counts<OPT>(m, mt, b, n, nt);
        if (limits) band_counts<OPT>(none, nonet, b, off, offt);
        const int all = (int)(((b < 4 ? ps.bld_lo : ps.bld_hi) >> (8 * (b & 3))) & 0xFFu);
        const float wc = wcos[b], ws = wsin[b];
        t.sws = fmaf((float)n, wc, t.sws);
        t.swh = fmaf((float)(all - n - off), wc, t.swh);
        t.lsu_c = fmaf((float)nt, wc, t.lsu_c);
        t.lsu_s = fmaf((float)nt, ws, t.lsu_s);
        t.lsh_c = fmaf((float)(all - nt - offt), wc, t.lsh_c);
        t.lsh_s = fmaf((float)(all - nt - offt), ws, t.lsh_s);
    }
    return t;
}

struct HourOut {
    double sstr, lup;
    double fsh, base_up;  // daytime
};

// Forward of one pixel-hour given the incoming state; returns sstr and Lup
// and the outgoing state.
__device__ __forceinline__ HourOut hour_forward(const SolweigHour& h, const HourTerms& t, const PixelStatics& ps,
                                                const HourIn& in, const BuildingTerms& bt, double state_in,
                                                double& state_out) {
    HourOut o;
    double kup = 0.0, lup, kdown = 0.0, kside = 0.0;
    state_out = state_in;
    o.fsh = o.base_up = 0.0;
    if (in.day) {
        o.fsh = wedge_fsh_tan(ps.tan_alfa, h.tan_zen);
        const double reflK = kAlbB * (1.0 - ps.svfbuveg) * (h.rad_g * (1.0 - o.fsh) + h.rad_d * o.fsh);
        o.base_up = h.rad_d * ps.svfbuveg + reflK;
        kup = in.ga * t.direct_up + o.base_up * ps.gn;
        const double prev = h.firstdaytime ? in.gl : state_in;
        lup = in.gl * (1.0 - h.wave_weight) + prev * h.wave_weight;
        state_out = h.wave_update ? lup : prev;
        const double d_rad = h.rad_d * (in.Ls + kVegTransmissivity * in.Lv);
        kdown = t.direct_up * in.s + d_rad + reflK;
        const double kside_d = t.ratio * (in.Cs + kVegTransmissivity * in.Cv);
        kside = in.s * t.beam + kside_d + t.sw_sun * bt.sws + t.sw_shade * bt.swh + t.sw_shade * ps.vc;
    } else {
        lup = ps.emis * t.ambient;
    }
    double ld_sky = 0.0, ls_sky = 0.0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const double cnt = ps.cnt(b);
        ld_sky += t.sky_down[b] * cnt;
        ls_sky += t.sky_side[b] * cnt;
    }
    const double refl = (ld_sky + lup) * ((1.0 - kEwall) * 0.5 / kPi);
    const double ldown = ld_sky + t.lw_shade * (ps.vs + bt.lsh_s) + t.lw_sun * bt.lsu_s + refl * ps.os;
    const double lside = ls_sky + t.lw_shade * (ps.vc + bt.lsh_c) + t.lw_sun * bt.lsu_c + refl * ps.oc;
    o.sstr = kAbsK * (kside * kFcyl + (kdown + kup) * kFup + 2.0 * kup * kFside) +
             kAbsL * ((ldown + lup) * kFup + lside * kFcyl + 2.0 * lup * kFside);
    o.lup = lup;
    return o;
}

// Reverse of one pixel-hour.  lam_state: adjoint of the outgoing state in,
// of the incoming state out.  Hour-scalar partials are added to acc[].
__device__ __forceinline__ void hour_backward(const SolweigHour& h, const HourTerms& t, const SolweigSkyLayout& L,
                                              const PixelStatics& ps, const HourIn& in, const BuildingTerms& bt,
                                              double state_in, double lam_obj, int objective, double& lam_state,
                                              double* acc, double& d_emis, double& lam_gl, double& lam_ga,
                                              double& lam_gn, double& lam_s, double* lam_sum) {
    const double ta = h.ta;
    double st_out;
    const HourOut o = hour_forward(h, t, ps, in, bt, state_in, st_out);
    const double root = sqrt(sqrt(o.sstr / (kAbsL * kSBC)));
    const double tmrt = root - 273.2;
    double lam_tmrt = 0.0;
    if (objective == 0) {
        if (ps.ground && h.utci_valid && tmrt > -999.0) {
            const double D = tmrt - ta;
            double dpoly = 0.0, pw = 1.0;
#pragma unroll
            for (int i = 1; i <= 6; ++i) {
                dpoly += i * h.utci[i] * pw;
                pw *= D;
            }
            double pw2 = lam_obj;
#pragma unroll
            for (int i = 0; i <= 6; ++i) {
                acc[kGUtci0 + i] += pw2;
                pw2 *= D;
            }
            lam_tmrt = lam_obj * dpoly;
            acc[kGTa] -= lam_tmrt;
        }
    } else {
        lam_tmrt = lam_obj;
    }
    const double lam_sstr = lam_tmrt * 0.25 * root / o.sstr;
    const double lam_kside = kAbsK * kFcyl * lam_sstr;
    const double lam_kdown = kAbsK * kFup * lam_sstr;
    const double lam_kup = kAbsK * (kFup + 2.0 * kFside) * lam_sstr;
    const double lam_ldown = kAbsL * kFup * lam_sstr;
    const double lam_lside = kAbsL * kFcyl * lam_sstr;
    double lam_lup = kAbsL * (kFup + 2.0 * kFside) * lam_sstr;
    const double lam_refl = lam_ldown * ps.os + lam_lside * ps.oc;
    const double crefl = (1.0 - kEwall) * 0.5 / kPi;
    lam_lup += lam_refl * crefl;
    const double lam_ldsky = lam_ldown + lam_refl * crefl;
    const double lam_lssky = lam_lside;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (b < L.nbands)
            acc[kGBand0 + b] += ((double)L.band_omega[b]) * ps.cnt(b) *
                                (lam_ldsky * L.band_sin[b] + lam_lssky * L.band_cos[b]);
    }
    const double lam_lw_shade = lam_ldown * (ps.vs + bt.lsh_s) + lam_lside * (ps.vc + bt.lsh_c);
    acc[kGTa] += lam_lw_shade * t.d_shade;
    lam_gl = lam_ga = lam_gn = lam_s = 0.0;
    lam_sum[0] = lam_sum[1] = 0.0;
    if (in.day) {
        const double lam_lw_sun = (lam_ldown * bt.lsu_s + lam_lside * bt.lsu_c) * t.d_sun;
        acc[kGTa] += lam_lw_sun;
        acc[kGTgwall] += lam_lw_sun;
        // Kside
        acc[kGRadI] += lam_kside * bt.sws * (kAlbB / kPi) * h.cos_alt;
        acc[kGRadD] += lam_kside * (bt.sws * (0.5 / kPi) + (bt.swh + ps.vc) * (kAlbB * 0.5 / kPi));
        const double csum = (in.Cs + kVegTransmissivity * in.Cv) / h.rad_tot;
        acc[kGRadD] += lam_kside * csum;
        acc[kGRadTot] -= lam_kside * t.ratio * csum;
        lam_sum[1] = lam_kside * t.ratio;
        lam_s += lam_kside * t.beam;
        acc[kGRadI] += lam_kside * in.s * h.cos_alt;
        // Kdown
        lam_s += lam_kdown * t.direct_up;
        acc[kGRadI] += lam_kdown * in.s * h.sin_alt;
        acc[kGRadD] += lam_kdown * (in.Ls + kVegTransmissivity * in.Lv);
        lam_sum[0] = lam_kdown * h.rad_d;
        double lam_reflK = lam_kdown;
        // Kup
        lam_ga = lam_kup * t.direct_up;
        lam_gn = lam_kup * o.base_up;
        acc[kGRadI] += lam_kup * in.ga * h.sin_alt;
        const double lam_base = lam_kup * ps.gn;
        acc[kGRadD] += lam_base * ps.svfbuveg;
        lam_reflK += lam_base;
        acc[kGRadD] += lam_reflK * kAlbB * (1.0 - ps.svfbuveg) * o.fsh;
        // wave delay of the GVF Lup
        const double lam_lup_total = lam_lup + (h.wave_update ? lam_state : 0.0);
        const double lam_prev = lam_lup_total * h.wave_weight + (h.wave_update ? 0.0 : lam_state);
        lam_gl = lam_lup_total * (1.0 - h.wave_weight) + (h.firstdaytime ? lam_prev : 0.0);
        lam_state = h.firstdaytime ? 0.0 : lam_prev;
        // ambient term of the GVF Lup plane: SBC * e * Tk^4
        d_emis += lam_gl * t.ambient;
        acc[kGTa] += lam_gl * ps.emis * t.d_ambient;
    } else {
        d_emis += lam_lup * t.ambient;
        acc[kGTa] += lam_lup * ps.emis * t.d_ambient;
        // the state passes through a night hour unchanged
    }
}

// Sums v[i] over the warp and leaves sum i in lane i: every exchange halves the
// number of values, 31 of them instead of five per value.
__device__ __forceinline__ double warp_sums(double (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool up = lane & o;
            const double give = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}

constexpr int kGradThreads = 128;
constexpr int kMaxGradHours = 32;

// One thread per pixel, all hours.  BACK: the states of the hours (which take
// the GVF alone), then every hour's fluxes and their reverse from the last hour
// on; else the objective.  What bounds it is the latency of float64 chains and
// of the plane loads (16 warps per SM in the reverse, issue 0.55 per cycle).
// 500 x 500 pixels, 24 hours: forward 0.65 -> 0.25 ms, reverse 1.45 -> 0.51 ms
// against one kernel that ran the objective before the reverse, with binary
// searches and a pass of popcounts per building sum, the hour's terms and
// divisions per pixel, a power function and five shuffles per reduced value.
template <int OPT, bool BACK>
__global__ void __launch_bounds__(kGradThreads, BACK ? 4 : 6) grad_radiation_kernel(SolweigScene S, const SolweigSkyLayout* Lp,
                                                                      const SolweigHour* __restrict__ hours,
                                                                      int nhours, const DayTable* __restrict__ tables,
                                                                      GradPtrs g) {
    __shared__ float wcos[8], wsin[8];
    __shared__ double red[kGradThreads / 32][kGFields];
    __shared__ HourTerms terms[kMaxGradHours];
    const SolweigSkyLayout& L = *Lp;
    if (threadIdx.x < 8) {
        const int b = threadIdx.x;
        const int k0 = Bands<OPT>::off(b);
        wcos[b] = b < L.nbands ? L.omega[k0] * L.cos_alt[k0] : 0.f;
        wsin[b] = b < L.nbands ? L.omega[k0] * L.sin_alt[k0] : 0.f;
    }
    if (threadIdx.x < nhours) hour_terms(hours[threadIdx.x], L, terms[threadIdx.x]);
    __syncthreads();
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)blockIdx.x * kGradThreads + threadIdx.x;
    const bool in_range = p < n;
    const long long q = in_range ? p : 0;
    PixelStatics ps;
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        const int nbits = S.patches - 32 * w;
        const uint32_t valid = nbits >= 32 ? 0xffffffffu : (nbits <= 0 ? 0u : ((1u << nbits) - 1u));
        ps.bld[w] = ~S.masks[(long long)w * n + q] & ~S.masks[(long long)(SOLWEIG_MASK_WORDS + w) * n + q] & valid;
    }
    ps.cnt_lo = ps.cnt_hi = ps.bld_lo = ps.bld_hi = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        ps.cnt_lo |= (uint32_t)S.sky_band_counts[(long long)b * n + q] << (8 * b);
        ps.cnt_hi |= (uint32_t)(b + 4 < S.nbands ? S.sky_band_counts[(long long)(b + 4) * n + q] : 0) << (8 * b);
        int lo, hi, same;
        band_counts<OPT>(ps.bld, ps.bld, b, lo, same);
        band_counts<OPT>(ps.bld, ps.bld, b + 4, hi, same);
        ps.bld_lo |= (uint32_t)lo << (8 * b);
        ps.bld_hi |= (uint32_t)hi << (8 * b);
    }
    ps.ground = (S.flags[q] & 1) != 0;
    ps.emis = g.emis[q];
    ps.svfbuveg = S.svfbuveg[q];
    ps.tan_alfa = tan(S.svfalfa[q]);
    ps.tan_asvf = S.tan_asvf[q];
    ps.tbucket = tan_bucket(ps.tan_asvf);
    ps.vc = S.veg_sums[q];
    ps.vs = S.veg_sums[n + q];
    ps.oc = S.veg_sums[2 * n + q];
    ps.os = S.veg_sums[3 * n + q];
    ps.gn = g.nosh[q];

    auto hour_in = [&](int hr) {
        HourIn in;
        in.day = hours[hr].daytime != 0;
        in.s = in.gl = in.ga = in.Ls = in.Cs = in.Lv = in.Cv = 0.0;
        if (in.day) {
            const long long g0 = 3LL * hr * n + q;
            in.gl = g.gvf[g0];
            in.ga = g.gvf[g0 + n];
            in.s = g.gvf[g0 + 2 * n];
            const long long s0 = 2LL * hr;
            in.Ls = g.sums[s0 * n + q];
            in.Cs = g.sums[(s0 + 1) * n + q];
            in.Lv = g.sums[(g.ncols + s0) * n + q];
            in.Cv = g.sums[(g.ncols + s0 + 1) * n + q];
        }
        return in;
    };

    if constexpr (!BACK) {
        double st = 0.0, obj = 0.0;
        for (int hr = 0; hr < nhours; ++hr) {
            const SolweigHour& h = hours[hr];
            const HourIn in = hour_in(hr);
            const BuildingTerms bt = building_terms<OPT>(tables[hr], ps, S.patches, in.day, wcos, wsin);
            double st2;
            const HourOut o = hour_forward(h, terms[hr], ps, in, bt, st, st2);
            st = st2;
            const double tmrt = sqrt(sqrt(o.sstr / (kAbsL * kSBC))) - 273.2;
            if (g.objective == 0) {
                obj += ps.ground ? (double)utci_eval(h.utci, tmrt, h.ta, h.utci_valid) : 0.0;
            } else {
                obj += tmrt;
            }
        }
        const double daily = obj / (double)nhours;
        if (in_range) g.daily[p] = (g.objective == 0 && !ps.ground) ? __longlong_as_double(0x7ff8000000000000ll) : daily;
    } else {
        double state_in[kMaxGradHours];  // incoming state of every hour
        double st = 0.0;
        for (int hr = 0; hr < nhours; ++hr) {
            const SolweigHour& h = hours[hr];
            state_in[hr] = st;
            if (!h.daytime) continue;
            const double gl = g.gvf[3LL * hr * n + q];
            const double prev = h.firstdaytime ? gl : st;
            st = h.wave_update ? gl * (1.0 - h.wave_weight) + prev * h.wave_weight : prev;
        }
        const double w = in_range ? (double)g.weights[p] : 0.0;
        const double lam_obj = (g.objective == 0 && !ps.ground) ? 0.0 : w / (double)nhours;
        double lam_state = 0.0, d_emis = 0.0, lam_gn = 0.0;
        for (int hr = nhours - 1; hr >= 0; --hr) {
            const SolweigHour& h = hours[hr];
            const HourIn in = hour_in(hr);
            const BuildingTerms bt = building_terms<OPT>(tables[hr], ps, S.patches, in.day, wcos, wsin);
            double acc[32];
#pragma unroll
            for (int f = 0; f < 32; ++f) acc[f] = 0.0;
            double lgl, lga, lgn, ls, lsum[2];
            hour_backward(h, terms[hr], L, ps, in, bt, state_in[hr], lam_obj, g.objective, lam_state, acc, d_emis, lgl,
                          lga, lgn, ls, lsum);
            lam_gn += lgn;
            if (in_range) {
                g.lam_gl[hr * n + p] = (float)lgl;
                g.lam_ga[hr * n + p] = (float)lga;
                g.lam_s[hr * n + p] = (float)ls;
                for (int i = 0; i < 2; ++i) g.lam_sums[(2LL * hr + i) * n + p] = (float)lsum[i];
            }
            // block reduction of the hour-scalar partials
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            if (!in_range) {
#pragma unroll
                for (int f = 0; f < kGFields; ++f) acc[f] = 0.0;
            }
            const double sum = warp_sums(acc);
            if (lane < kGFields) red[warp][lane] = sum;
            __syncthreads();
            if (threadIdx.x < kGFields) {
                double v = 0.0;
                for (int i = 0; i < kGradThreads / 32; ++i) v += red[i][threadIdx.x];
                atomicAdd(&g.hour_grad[hr * kGFields + threadIdx.x], v);
            }
            __syncthreads();
        }
        if (in_range) {
            g.d_emis_direct[p] = (float)d_emis;
            g.lam_gn[p] = (float)lam_gn;
        }
    }
}

// ------------------------------------------------------------------ GVF transpose

struct GvfAdjPtrs {
    const float* lam_gl;   // [H][px]
    const float* lam_ga;   // [H][px]
    const float* lam_gn;   // [px], summed over the hours
    float* lam_lup;        // [H][px] scatter target
    float* lam_albsh;      // [H][px]
    float* lam_alb;        // [px]
    double* hour_grad;     // [H][kGFields]
};

// For tables whose walks don't start at their pixel, which have no walk words:
// every pixel p and hour takes the 18 walks of the forward (first = 1,
// second = 22, the fixed 1 m case) with the coefficient of every walked
// sample in p's all-direction GVF planes; the adjoints are scattered onto the
// samples.  Samples outside the raster repeat the last in-raster sample.
template <int TY>
__global__ void __launch_bounds__(32 * TY) gvf_adjoint_kernel(SolweigScene S, const SolweigHour* __restrict__ hours,
                                                             GvfTable<22> tab, const float4* __restrict__ quads,
                                                             GvfAdjPtrs a) {
    constexpr int FIRST = 1, SECOND = 22, H = SECOND - 1;
    const int z = blockIdx.z;
    const SolweigHour& h = hours[z];
    if (!h.daytime) return;
    const long long n = (long long)S.rows * S.cols;
    const float4* quad = quads + z * n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int pitch = 32 + 2 * H;
    float4* tile = reinterpret_cast<float4*>(smem_raw);
    const int row0 = blockIdx.y * TY - H, col0 = blockIdx.x * 32 - H;
    load_quad_tile(tile, pitch, TY + 2 * H, quad, S.rows, S.cols, row0, col0);
    __syncthreads();
    const int c = blockIdx.x * 32 + threadIdx.x;
    const int r = blockIdx.y * TY + threadIdx.y;
    if (r >= S.rows || c >= S.cols) return;
    const long long p = (long long)r * S.cols + c;
    const float4 own = tile[(threadIdx.y + H) * pitch + threadIdx.x + H];
    const bool own_ground = (__float_as_int(own.w) & kQuadGround) != 0;
    const float ob = own_ground ? 1.f : 0.f;
    const double lgl = a.lam_gl[z * n + p] / 18.0;
    const double lga = a.lam_ga[z * n + p] / 18.0;
    bool first_day = true;  // the albedo's adjoint is of all hours
    for (int k = 0; k < z; ++k) first_day = first_day && !hours[k].daytime;
    const double lgn = first_day ? a.lam_gn[p] / 18.0 : 0.0;
    float* lup_t = a.lam_lup + z * n;
    float* albsh_t = a.lam_albsh + z * n;
    // own-pixel corrections (non-ground pixels)
    if (!own_ground) {
        atomicAdd(&lup_t[p], (float)(18.0 * lgl));
        atomicAdd(&albsh_t[p], (float)(18.0 * lga));
        atomicAdd(&a.lam_alb[p], (float)(18.0 * lgn));
    }
    double lwall_coef = 0.0;
    const uint32_t face = S.gvf_face[p];
    if (own_ground) {
        for (int j = 0; j < SOLWEIG_GVF_DIRECTIONS; ++j) {
            const int2* offs = tab.offs + j * SECOND;
            // pass 1: walk length, sunlit-wall statistics, frozen tail
            int hit = SECOND, n_sun = 0, n_sun_first = 0, last = -1, frozen_at = -1;
            bool seen_sun = false;
            for (int s = 0; s < SECOND; ++s) {
                const int rr = r + offs[s].x, cc = c + offs[s].y;
                const bool inside = in_raster(rr, cc, S.rows, S.cols);
                int bits;
                if (inside) {
                    bits = __float_as_int(tile[(rr - row0) * pitch + (cc - col0)].w);
                    last = s;
                } else {
                    bits = last >= 0 ? __float_as_int(tile[(r + offs[last].x - row0) * pitch + (c + offs[last].y - col0)].w) : 0;
                }
                if (!(bits & kQuadGround)) {
                    hit = s;
                    break;
                }
                seen_sun = seen_sun || (bits & kQuadSunwall);
                if (!inside) {
                    // frozen from here on: every remaining step repeats this sample
                    frozen_at = s;
                    n_sun += seen_sun ? SECOND - s : 0;
                    if (s < FIRST) n_sun_first = n_sun - (seen_sun ? SECOND - FIRST : 0);
                    break;
                }
                n_sun += seen_sun ? 1 : 0;
                if (s + 1 == FIRST) n_sun_first = n_sun;
            }
            if (hit < SECOND) {
                if (hit < FIRST) n_sun_first = n_sun + (seen_sun ? FIRST - hit : 0);
                n_sun += seen_sun ? SECOND - hit : 0;
            }
            const bool sun_near = n_sun_first > 0, sun_far = n_sun > 0;
            const int n_wall = SECOND - hit;
            const bool wall_near = FIRST > hit, wall_far = n_wall > 0;
            const bool face_drop = (n_sun == SECOND) && ((face >> j) & 1u);
            const double c1 = 0.5 / 0.9 * (sun_near ? 1.0 / (FIRST + 1) : 1.0 / FIRST);
            const double c2 = 0.4 / 0.9 * (sun_far ? 1.0 / (SECOND + 1) : 1.0 / SECOND);
            const double n1 = 0.5 / 0.9 * (wall_near ? 1.0 / (FIRST + 1) : 1.0 / FIRST);
            const double n2 = 0.4 / 0.9 * (1.0 / SECOND);
            (void)wall_far;
            // d(d_lup)/d(lwall) = c1' * n_sun_first + c2' * n_sun (when counted)
            lwall_coef += (sun_near ? 0.5 / 0.9 / (FIRST + 1) * n_sun_first : 0.0) +
                          (sun_far && !face_drop ? 0.4 / 0.9 / (SECOND + 1) * n_sun : 0.0);
            // pass 2: scatter onto the walked samples
            const int steps = frozen_at >= 0 ? frozen_at + 1 : hit;
            for (int s = 0; s < steps; ++s) {
                int rr = r + offs[s].x, cc = c + offs[s].y;
                int mult = 1;
                if (s == frozen_at) {
                    rr = r + offs[last].x;
                    cc = c + offs[last].y;
                    mult = SECOND - s;
                }
                // steps s .. s + mult - 1 all read this sample
                double k_lup = 0.0, k_nosh = 0.0;
                for (int t = s; t < s + mult; ++t) {
                    k_lup += (t < FIRST ? c1 : 0.0) + c2;
                    k_nosh += (t < FIRST ? n1 : 0.0) + n2;
                }
                const long long qq = (long long)rr * S.cols + cc;
                atomicAdd(&lup_t[qq], (float)(k_lup * lgl));
                atomicAdd(&albsh_t[qq], (float)(k_lup * lga));
                atomicAdd(&a.lam_alb[qq], (float)(k_nosh * lgn * ob));
            }
        }
    }
    if (lwall_coef != 0.0 && lgl != 0.0) {
        const double ta = h.ta, tk = ta + 273.15, tw = h.tgwall + ta + 273.15;
        const double v = lgl * lwall_coef;
        atomicAdd(&a.hour_grad[z * kGFields + kGTa], v * kSBC * 0.9 * 4.0 * (tw * tw * tw - tk * tk * tk));
        atomicAdd(&a.hour_grad[z * kGFields + kGTgwall], v * kSBC * 0.9 * 4.0 * tw * tw * tw);
    }
}

// Transpose of the GVF of every daytime hour by walk words, in two kernels.
//
// A pixel p adds to its planes, per direction j, the samples s < lim(p, j) at
// p + off(j, s) times c2 = 0.4 / 0.9 / (22 or, when it met a sunlit wall, 23).
// So pixel q gathers, from every (j, s) with lim(p, j) > s at p = q - off(j, s),
// p's adjoint times that c2: no atomics, a fixed order, and the length test is
// the same for all hours.  gvf_transpose_words_kernel packs lim and the sunlit
// bits of two hours into one byte per (pixel, direction), four directions to a
// word, and sums the wall terms; gvf_transpose_kernel stages the adjoints of two
// hours (16 bytes a pixel) and one word of a 32 x 32 tile and its halo (two
// blocks per SM) and gathers both.  The adjoint of the albedo alone doesn't
// depend on the hour's sun, so the hours' sum is gathered once (last slice).
//
// One thread per pixel and hour scattering its walks by three atomics a sample,
// and two float64 atomics on the hour's partials, took 5.59 ms for 17 hours of
// 500 x 500 pixels; the two kernels take 0.16 + 0.93 ms.  What bounds
// the gather is instruction issue (65 % of the cycles) and shared-memory
// wavefronts (57 %).
constexpr int kTrSteps = kWkMaxSteps, kTrHalo = kTrSteps - 1, kTrWidth = kWkTile + 2 * kTrHalo;
constexpr int kTrCells = kTrWidth * kTrWidth, kTrThreads = 512;
constexpr int kTrGroups = (kWkDirs + 3) / 4;  // words of four directions
constexpr double kNear = 0.5 / 0.9, kFar = 0.4 / 0.9;

struct TransposeOffsets {
    int2 back[kWkDirs][kTrSteps / 2];  // -16 (bytes of a staged pixel) times the cells of samples 2 i + 1 and 2 i + 2
    int8_t dr[kWkDirs][kTrSteps], dc[kWkDirs][kTrSteps];
    int reach;  // pixels between neighbouring samples, at most
};

__global__ void __launch_bounds__(256) gvf_transpose_words_kernel(SolweigScene S, const SolweigHour* __restrict__ hours,
                                                                  int nhours,
                                                                  const __grid_constant__ TransposeOffsets off,
                                                                  const uint32_t* __restrict__ walks,
                                                                  const uint32_t* __restrict__ codes,
                                                                  const float* __restrict__ lam_gl,
                                                                  uint32_t* __restrict__ words,
                                                                  double* __restrict__ hour_grad) {
    __shared__ int sample_at[kWkDirs][kTrSteps];
    __shared__ int day_hour[64], days;
    __shared__ double red[8][kWkHours];
    const int tid = threadIdx.x;
    const long long n = (long long)S.rows * S.cols;
    for (int i = tid; i < kWkDirs * kTrSteps; i += blockDim.x)
        (&sample_at[0][0])[i] = (&off.dr[0][0])[i] * S.cols + (&off.dc[0][0])[i];
    if (tid < 32) days = day_hours(hours, nhours, day_hour);
    __syncthreads();
    const int nd = days, g0 = blockIdx.y * kWkHours;
    if (g0 >= nd) return;
    const long long p = (long long)blockIdx.x * blockDim.x + tid;
    double v[kWkHours] = {0.0, 0.0, 0.0, 0.0};
    if (p < n) {
        const int r = (int)(p / S.cols), c = (int)(p - (long long)r * S.cols);
        const uint32_t* walk = walks + walk_word_at(r, c, S.cols);
        const uint32_t* code = codes + blockIdx.y * n + p;
        uint32_t* out = words + (long long)blockIdx.y * 2 * kTrGroups * n + p;
        int wall_steps[kWkHours] = {0, 0, 0, 0};
#pragma unroll 1
        for (int g = 0; g < kTrGroups; ++g) {
            uint32_t word[2] = {0u, 0u};
            for (int d = 0; d < 4 && 4 * g + d < kWkDirs; ++d) {
                const int j = 4 * g + d;
                const uint32_t w = walk[j * kWkPixels];
                const uint32_t lim = min((w >> kWkLimShift) & 31u, (uint32_t)kTrSteps);
                uint32_t seen = 0u;
                for (uint32_t walls = w & kWkWallBits; walls; walls &= walls - 1u) {
                    const int m = __ffs((int)walls) - 1;
                    const uint32_t b = code[sample_at[j][m]];
#pragma unroll
                    for (int k = 0; k < kWkHours; ++k) {
                        if (((b >> (5 * k + 4)) & 1u) && !((seen >> k) & 1u)) {
                            seen |= 1u << k;
                            if (m > 0 || !(w & kWkFace)) wall_steps[k] += kTrSteps - m;
                        }
                    }
                }
                word[0] |= ((lim << 2) | (seen & 3u)) << (8 * d);
                word[1] |= ((lim << 2) | (seen >> 2)) << (8 * d);
            }
            out[g * n] = word[0];
            out[(kTrGroups + g) * n] = word[1];
        }
        const uint32_t own = *code;
#pragma unroll
        for (int k = 0; k < kWkHours; ++k) {
            const bool near = (own >> (5 * k + 4)) & 1u;
            const double coef = (near ? kWkDirs * (kNear / 2) : 0.0) + kFar / (kTrSteps + 1) * wall_steps[k];
            if (g0 + k < nd && coef != 0.0) v[k] = (double)lam_gl[day_hour[g0 + k] * n + p] / 18.0 * coef;
        }
    }
    // the wall's Lup: partials of the hour's Ta and wall temperature
#pragma unroll
    for (int k = 0; k < kWkHours; ++k) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if ((tid & 31) == 0) red[tid >> 5][k] = v[k];
    }
    __syncthreads();
    if (tid < kWkHours && g0 + tid < nd) {
        double sum = 0.0;
        for (int w = 0; w < 8; ++w) sum += red[w][tid];
        if (sum == 0.0) return;
        const int hr = day_hour[g0 + tid];
        const SolweigHour& h = hours[hr];
        const double ta = h.ta, tk = ta + 273.15, tw = h.tgwall + ta + 273.15;
        atomicAdd(&hour_grad[hr * kGFields + kGTa], sum * kSBC * 0.9 * 4.0 * (tw * tw * tw - tk * tk * tk));
        atomicAdd(&hour_grad[hr * kGFields + kGTgwall], sum * kSBC * 0.9 * 4.0 * tw * tw * tw);
    }
}

struct TransposePtrs {
    const uint32_t* words;  // of gvf_transpose_words_kernel
    const uint32_t* codes;  // of gvf_codes_kernel
    const float* lam_gl;    // [H][px]
    const float* lam_ga;    // [H][px]
    const float* lam_gn;    // [px]
    float* lam_lup;         // [H][px]
    float* lam_albsh;       // [H][px]
    float* lam_alb;         // [px]
};

// Adds a staged pixel's adjoints (the hours' Lup, then their albedos) where its
// byte says that its walk reads the sample, times `sun` in the hours in which it
// met a sunlit wall, else `plain`.  Predicated: nearly every warp has a lane
// that adds.
__device__ __forceinline__ void gather_where(float4& sum, uint32_t at, uint32_t byte, uint32_t least, float sun,
                                             float plain) {
    const float w0 = byte & 1u ? sun : plain, w1 = byte & 2u ? sun : plain;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .f32 a, b, c, d;\n\t"
        "setp.ge.u32 p, %5, %6;\n\t"
        "@p ld.shared.v4.f32 {a, b, c, d}, [%4];\n\t"
        "@p fma.rn.f32 %0, %7, a, %0;\n\t@p fma.rn.f32 %1, %8, b, %1;\n\t"
        "@p fma.rn.f32 %2, %7, c, %2;\n\t@p fma.rn.f32 %3, %8, d, %3;\n\t}"
        : "+f"(sum.x), "+f"(sum.y), "+f"(sum.z), "+f"(sum.w)
        : "r"(at), "r"(byte), "r"(least), "f"(w0), "f"(w1));
}

__global__ void __launch_bounds__(kTrThreads, 2) gvf_transpose_kernel(SolweigScene S,
                                                                      const SolweigHour* __restrict__ hours, int nhours,
                                                                      const __grid_constant__ TransposeOffsets off,
                                                                      TransposePtrs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4* plane = reinterpret_cast<float4*>(smem_raw);
    uint32_t* word = reinterpret_cast<uint32_t*>(plane + kTrCells);
    __shared__ int day_hour[64], days;
    const int tid = threadIdx.x;
    const long long n = (long long)S.rows * S.cols;
    if (tid < 32) days = day_hours(hours, nhours, day_hour);
    __syncthreads();
    const int nd = days;
    const bool albedo = blockIdx.z + 1 == gridDim.z;
    const int z = albedo ? 0 : blockIdx.z;  // the hours 2 z and 2 z + 1
    if (2 * z >= nd) return;
    const int ha = day_hour[2 * z], hb = day_hour[min(2 * z + 1, nd - 1)];
    const uint32_t* words = a.words + (long long)z * kTrGroups * n;
    const int row0 = blockIdx.y * kWkTile - kTrHalo, col0 = blockIdx.x * kWkTile - kTrHalo;
    for (int i = tid; i < kTrCells; i += kTrThreads) {
        const int rr = row0 + i / kTrWidth, cc = col0 + i % kTrWidth;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in_raster(rr, cc, S.rows, S.cols)) {
            const long long p = (long long)rr * S.cols + cc;
            if (albedo) v.x = __ldg(a.lam_gn + p);
            else v = make_float4(__ldg(a.lam_gl + ha * n + p), __ldg(a.lam_gl + hb * n + p), __ldg(a.lam_ga + ha * n + p),
                                 __ldg(a.lam_ga + hb * n + p));
        }
        plane[i] = v;
    }
    // c2 in units of 0.4 / 0.9 / (22 * 23), exact
    constexpr float plain = kTrSteps + 1;
    const float sun = albedo ? plain : (float)kTrSteps;
    // two pixels a thread, 16 rows apart: one address and offset for both
    constexpr int kOwn = 2, kOwnRows = kWkTile / kOwn, kOwnCells = kOwnRows * kTrWidth;
    static_assert(kOwn * kTrThreads == kWkPixels, "two pixels a thread");
    int ty, tx;
    walk_pixel(tid, ty, tx);
    const int r = blockIdx.y * kWkTile + ty, c = blockIdx.x * kWkTile + tx;
    const int own = (ty + kTrHalo) * kTrWidth + tx + kTrHalo;
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(plane + own);
    float4 acc[kOwn];
    bool ground[kOwn], edge[kOwn];
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
        const int ri = r + i * kOwnRows;
        acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        ground[i] = ri < S.rows && c < S.cols && (S.flags[(long long)ri * S.cols + c] & 1);
        edge[i] = ground[i] && (ri < off.reach || c < off.reach || ri >= S.rows - off.reach || c >= S.cols - off.reach);
    }
#pragma unroll 1
    for (int g = 0; g < kTrGroups; ++g) {
        __syncthreads();
        for (int i = tid; i < kTrCells; i += kTrThreads) {
            const int rr = row0 + i / kTrWidth, cc = col0 + i % kTrWidth;
            word[i] = in_raster(rr, cc, S.rows, S.cols) ? __ldg(words + g * n + (long long)rr * S.cols + cc) : 0u;
        }
        __syncthreads();
        if (!ground[0] && !ground[1]) continue;  // no walk reads other pixels: their bytes say so too
#pragma unroll 1
        for (int d = 0; d < 4 && 4 * g + d < kWkDirs; ++d) {
            const int j = 4 * g + d;
            // a pixel's byte of this direction: 4 lim + the hours' sunlit bits
            const uint8_t* byte = reinterpret_cast<const uint8_t*>(word + own) + d;
            float4 sum[kOwn];
#pragma unroll
            for (int i = 0; i < kOwn; ++i) {
                sum[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                gather_where(sum[i], at + 16 * i * kOwnCells, byte[4 * i * kOwnCells], 4u, sun, plain);
            }
            uint32_t least = 8u;  // 4 (m + 1)
#pragma unroll 1
            for (int m = 0; m < kTrSteps / 2; ++m) {
                const int2 o = off.back[j][m];
                const uint8_t *byte0 = byte + (o.x >> 2), *byte1 = byte + (o.y >> 2);
                uint32_t b0[kOwn], b1[kOwn];
#pragma unroll
                for (int i = 0; i < kOwn; ++i) {
                    b0[i] = byte0[4 * i * kOwnCells];
                    b1[i] = byte1[4 * i * kOwnCells];
                }
#pragma unroll
                for (int i = 0; i < kOwn; ++i) {
                    gather_where(sum[i], at + o.x + 16 * i * kOwnCells, b0[i], least, sun, plain);
                    // lim is at most 22: nothing for the step after the last
                    gather_where(sum[i], at + o.y + 16 * i * kOwnCells, b1[i], least + 4u, sun, plain);
                }
                least += 8u;
            }
#pragma unroll
            for (int i = 0; i < kOwn; ++i) {
                if (edge[i]) {
                    // walks that leave the raster behind this pixel repeat it to their end
#pragma unroll 1
                    for (int m = 0; m + 1 < kTrSteps; ++m) {
                        const int nr = r + i * kOwnRows + off.dr[j][m + 1] - off.dr[j][m];
                        const int nc = c + off.dc[j][m + 1] - off.dc[j][m];
                        if (in_raster(nr, nc, S.rows, S.cols)) continue;
                        const int cell = i * kOwnCells - off.dr[j][m] * kTrWidth - off.dc[j][m];
                        const uint32_t b = byte[4 * cell];
                        const float times = (float)(kTrSteps - 1 - m);
                        if ((b >> 2) == (uint32_t)(m + 1)) gather_where(sum[i], at + 16 * cell, b, 0u, times * sun, times * plain);
                    }
                }
                acc[i].x += sum[i].x;
                acc[i].y += sum[i].y;
                acc[i].z += sum[i].z;
                acc[i].w += sum[i].w;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
        const int ri = r + i * kOwnRows;
        if (ri >= S.rows || c >= S.cols) continue;
        const long long p = (long long)ri * S.cols + c;
        const float4 v = plane[own + i * kOwnCells];
        // the pixel's own sample also is the near term of its 18 walks, half of it
        // when it is a sunlit wall; off the ground it is the pixel's plane
        auto total = [&](float far, float self, bool near) {
            return (float)(ground[i] ? (double)far * (kFar / (kTrSteps * (kTrSteps + 1)) / 18.0) + (near ? kNear / 2 : kNear) * self
                                     : (double)self);
        };
        if (albedo) {
            a.lam_alb[p] = total(acc[i].x, v.x, false);
            continue;
        }
        const uint32_t code = a.codes[(z >> 1) * n + p] >> (10 * (z & 1));
        a.lam_lup[ha * n + p] = total(acc[i].x, v.x, code & 16u);
        a.lam_albsh[ha * n + p] = total(acc[i].z, v.z, code & 16u);
        if (2 * z + 1 < nd) {
            a.lam_lup[hb * n + p] = total(acc[i].y, v.y, code & 512u);
            a.lam_albsh[hb * n + p] = total(acc[i].w, v.w, code & 512u);
        }
    }
}

int launch_gvf_transpose(const SolweigScene& S, const SolweigHour* hours, int nhours, const int32_t* dxdy,
                         const DayWalkArgs& wa, uint32_t* words, const GvfAdjPtrs& g, cudaStream_t st) {
    TransposeOffsets off;
    off.reach = 1;
    for (int j = 0; j < kWkDirs; ++j)
        for (int m = 0; m < kTrSteps; ++m) {
            const int32_t* o = dxdy + 2 * (j * kTrSteps + m);
            const int back = -16 * (o[0] * kTrWidth + o[1]);
            if (m & 1) off.back[j][m >> 1] = make_int2(back, 0);
            else if (m > 0) off.back[j][(m - 1) >> 1].y = back;
            off.dr[j][m] = (int8_t)o[0];
            off.dc[j][m] = (int8_t)o[1];
            if (m > 0) off.reach = std::max(off.reach, std::max(std::abs(o[0] - o[-2]), std::abs(o[1] - o[-1])));
        }
    const int passes = (nhours + kWkHours - 1) / kWkHours;
    const long long px = (long long)S.rows * S.cols;
    gvf_transpose_words_kernel<<<dim3(blocks_for(px, 256), passes), 256, 0, st>>>(
        S, hours, nhours, off, wa.walks, wa.codes, g.lam_gl, words, g.hour_grad);
    SOLWEIG_CHECK_LAUNCH("gvf_transpose_words_kernel");
    const size_t smem = (sizeof(float4) + 4) * (size_t)kTrCells;
    set_smem_attr((const void*)gvf_transpose_kernel, smem);
    const dim3 grid(blocks_for(S.cols, kWkTile), blocks_for(S.rows, kWkTile), (nhours + 1) / 2 + 1);
    gvf_transpose_kernel<<<grid, kTrThreads, smem, st>>>(
        S, hours, nhours, off,
        TransposePtrs{words, wa.codes, g.lam_gl, g.lam_ga, g.lam_gn, g.lam_lup, g.lam_albsh, g.lam_alb});
    SOLWEIG_CHECK_LAUNCH("gvf_transpose_kernel");
    return SOLWEIG_OK;
}

// ------------------------------------------------------------------ parameters

__global__ void param_grad_kernel(SolweigScene S, const SolweigHour* __restrict__ hours, int nhours,
                                  const float4* __restrict__ quads, const uint8_t* __restrict__ sv,
                                  const float* __restrict__ alb, const float* __restrict__ emis,
                                  const float* __restrict__ lam_lup, const float* __restrict__ lam_albsh,
                                  const float* __restrict__ lam_alb, const float* __restrict__ lam_s,
                                  const float* __restrict__ d_emis_direct, float* __restrict__ d_alb,
                                  float* __restrict__ d_emis, float* __restrict__ d_tau, double* __restrict__ hour_grad) {
    __shared__ double red[8][2];
    const long long n = (long long)S.rows * S.cols;
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = p < n;
    const long long q = in ? p : 0;
    double da = in ? lam_alb[q] : 0.0, de = in ? d_emis_direct[q] : 0.0, dt = 0.0;
    const double e = emis[q], a_ = alb[q];
    for (int hr = 0; hr < nhours; ++hr) {
        const SolweigHour& h = hours[hr];
        double g_ta = 0.0, g_ci = 0.0;
        if (h.daytime && in) {
            const long long i = hr * n + q;
            const double s = quads[i].x;
            const int vegsh = (sv[i] >> 1) & 1;
            const double ll = lam_lup[i], la = lam_albsh[i];
            const double amp = (double)S.tgk[q] * h.altmax + (double)S.tstart[q];
            const double phase =
                ((h.dectime_frac - h.snup / 24.0) / ((double)S.tmaxlst[q] / 24.0 - h.snup / 24.0)) * kPi / 2.0;
            const double wave = amp * sin(phase);
            double tg = wave * h.ci_tgg;
            const bool clamped = S.landcover == 1 && tg < 0.0;
            if (clamped) tg = 0.0;
            const double T = h.ta + 273.15, X = tg * s + T;
            const double X3 = X * X * X;
            de += ll * kSBC * (pow4(X) - pow4(T));
            da += la * s;
            dt += (ll * kSBC * e * 4.0 * X3 * tg + la * a_ + (double)lam_s[i]) * (1.0 - vegsh);
            g_ta = ll * kSBC * e * 4.0 * (X3 - T * T * T);
            g_ci = clamped ? 0.0 : ll * kSBC * e * 4.0 * X3 * s * wave;
        }
        for (int o = 16; o > 0; o >>= 1) {
            g_ta += __shfl_xor_sync(0xffffffffu, g_ta, o);
            g_ci += __shfl_xor_sync(0xffffffffu, g_ci, o);
        }
        if ((threadIdx.x & 31) == 0) {
            red[threadIdx.x >> 5][0] = g_ta;
            red[threadIdx.x >> 5][1] = g_ci;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            double v = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[w][threadIdx.x];
            if (v != 0.0) atomicAdd(&hour_grad[hr * kGFields + (threadIdx.x == 0 ? kGTa : kGCiTgg)], v);
        }
        __syncthreads();
    }
    if (in) {
        d_alb[p] = (float)da;
        d_emis[p] = (float)de;
        d_tau[p] = (float)dt;
    }
}

// lum_grad[h][4][k]: sums over pixels of (sky, sky, veg, veg) mask bits times
// the adjoints of (luminance sum, luminance*cos*omega sum) of each mask.  The
// canopy's adjoints are the sky's times its transmissivity, so the pixels are
// summed once per mask and the factor is applied to the sums.
//
// A warp sums four daytime hours (grid.y) over its pixels, each lane five
// patches in registers: a pixel's adjoints and mask words are broadcast from
// shared memory and a set bit takes eight predicated additions, so a NaN stays
// with the patches that see it.  What bounds it is instruction issue, 80
// additions per pixel and pass.  One shared-memory atomic per set bit and sum
// took 4.99 ms for 17 hours of 500 x 500 pixels, this takes 0.14 ms.
// kLumPixels bounds the float32 chain of a sum (it was px / 148 per block);
// beyond it the sums are float64.
constexpr int kLumHours = 4, kLumWarps = 8, kLumPixels = 512, kLumPitch = 20, kLumLanePatches = kK / 32;
static_assert(kLumLanePatches == SOLWEIG_MASK_WORDS, "one patch of every mask word per lane");

__device__ __forceinline__ void add_where(uint32_t bit, float (&acc)[2 * kLumHours], const float (&v)[2 * kLumHours]) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %16, 0;\n\t"
        "@p add.f32 %0, %0, %8;\n\t@p add.f32 %1, %1, %9;\n\t@p add.f32 %2, %2, %10;\n\t@p add.f32 %3, %3, %11;\n\t"
        "@p add.f32 %4, %4, %12;\n\t@p add.f32 %5, %5, %13;\n\t@p add.f32 %6, %6, %14;\n\t@p add.f32 %7, %7, %15;\n\t}"
        : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3]), "+f"(acc[4]), "+f"(acc[5]), "+f"(acc[6]), "+f"(acc[7])
        : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "r"(bit));
}

__global__ void __launch_bounds__(32 * kLumWarps, 2) lum_grad_kernel(SolweigScene S,
                                                                     const SolweigHour* __restrict__ hours, int nhours,
                                                                     const float* __restrict__ lam_sums,
                                                                     int warp_pixels, double* __restrict__ lum_grad) {
    // a warp's 32 pixels: eight adjoints, five sky and five canopy words each; afterwards the block's sums
    __shared__ __align__(16) unsigned char smem[kLumWarps * 32 * kLumPitch * 4];
    __shared__ int day_hour[64], days;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n = (long long)S.rows * S.cols;
    if (warp == 0) days = day_hours(hours, nhours, day_hour);
    __syncthreads();
    const int nd = days, g0 = blockIdx.y * kLumHours;
    if (g0 >= nd) return;
    float* buf = reinterpret_cast<float*>(smem) + warp * 32 * kLumPitch;
    float acc[2][kLumLanePatches][2 * kLumHours];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int w = 0; w < kLumLanePatches; ++w)
#pragma unroll
            for (int i = 0; i < 2 * kLumHours; ++i) acc[m][w][i] = 0.f;
    const long long p0 = ((long long)blockIdx.x * kLumWarps + warp) * warp_pixels;
    const long long p1 = min(n, p0 + warp_pixels);
    const uint32_t own = 1u << lane;
    for (long long q0 = p0; q0 < p1; q0 += 32) {
        const int count = (int)min(32ll, p1 - q0);
        if (lane < count) {
            const long long p = q0 + lane;
            float v[kLumPitch];
#pragma unroll
            for (int i = 0; i < kLumHours; ++i) {
                const long long at = 2LL * day_hour[min(g0 + i, nd - 1)] * n + p;
                v[2 * i] = lam_sums[at];
                v[2 * i + 1] = lam_sums[at + n];
            }
#pragma unroll
            for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
                const int nbits = S.patches - 32 * w;
                const uint32_t valid = nbits >= 32 ? 0xffffffffu : (nbits <= 0 ? 0u : ((1u << nbits) - 1u));
                const uint32_t sky = S.masks[(long long)w * n + p] & valid;
                const uint32_t veg = S.masks[(long long)(SOLWEIG_MASK_WORDS + w) * n + p];
                v[8 + w] = __uint_as_float(sky & ~veg);
                v[13 + w] = __uint_as_float(sky & veg);
            }
            v[18] = v[19] = 0.f;
            float4* row = reinterpret_cast<float4*>(buf + lane * kLumPitch);
#pragma unroll
            for (int i = 0; i < kLumPitch / 4; ++i) row[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
        __syncwarp();
        for (int t = 0; t < count; ++t) {
            const float4* row = reinterpret_cast<const float4*>(buf + t * kLumPitch);
            const float4 a = row[0], b = row[1], c = row[2], d = row[3];
            const float2 e = *reinterpret_cast<const float2*>(row + 4);
            const float v[2 * kLumHours] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            const float word[2 * kLumLanePatches] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w, e.x, e.y};
#pragma unroll
            for (int w = 0; w < kLumLanePatches; ++w) {
                add_where(__float_as_uint(word[w]) & own, acc[0][w], v);
                add_where(__float_as_uint(word[kLumLanePatches + w]) & own, acc[1][w], v);
            }
        }
        __syncwarp();
    }
    // the block's sums, one mask and hour at a time: [sum][warp][patch]
    float* part = reinterpret_cast<float*>(smem);
    static_assert(2 * kLumWarps * kK * 4 <= (int)sizeof(smem), "partial sums of an hour fit");
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int i = 0; i < kLumHours; ++i) {
            __syncthreads();
#pragma unroll
            for (int w = 0; w < kLumLanePatches; ++w) {
#pragma unroll
                for (int c = 0; c < 2; ++c) part[(c * kLumWarps + warp) * kK + 32 * w + lane] = acc[m][w][2 * i + c];
            }
            __syncthreads();
            if (g0 + i >= nd) continue;
            double* out = lum_grad + ((long long)day_hour[g0 + i] * 4 + 2 * m) * kK;
            for (int k = threadIdx.x; k < 2 * kK; k += blockDim.x) {
                const int c = k / kK, patch = k - c * kK;
                double v = 0.0;
#pragma unroll
                for (int w = 0; w < kLumWarps; ++w) v += (double)part[(c * kLumWarps + w) * kK + patch];
                if (v != 0.0) atomicAdd(out + k, m ? kVegTransmissivity * v : v);
            }
        }
    }
}

// ------------------------------------------------------------------ host

struct GradWork {
    long long day_total;  // the batched-day work (quads0 = its quads)
    long long quads1, sv, gvf, lam_gl, lam_ga, lam_gn, lam_s, lam_sums, lam_lup, lam_albsh, lam_alb, d_emis_direct;
    long long walks, codes, words;  // of the GVF walks: walk words (read until the transpose), samples' codes, the transpose's words
    long long total;
};

GradWork grad_work_layout(int rows, int cols, int nhours) {
    GradWork g{};
    const long long px = (long long)rows * cols;
    const DayWork d = day_work_layout(rows, cols, nhours, false);
    long long o = d.total;
    g.day_total = d.total;
    g.quads1 = o; o = align256(o + 16LL * px * nhours);
    g.sv = o; o = align256(o + 1LL * px * nhours);
    g.gvf = o; o = align256(o + 12LL * px * nhours);
    g.lam_gl = o; o = align256(o + 4LL * px * nhours);
    g.lam_ga = o; o = align256(o + 4LL * px * nhours);
    g.lam_gn = o; o = align256(o + 4LL * px);
    g.lam_s = o; o = align256(o + 4LL * px * nhours);
    g.lam_sums = o; o = align256(o + 8LL * px * nhours);
    g.lam_lup = o; o = align256(o + 4LL * px * nhours);
    g.lam_albsh = o; o = align256(o + 4LL * px * nhours);
    g.lam_alb = o; o = align256(o + 4LL * px);
    g.d_emis_direct = o; o = align256(o + 4LL * px);
    const long long passes = (nhours + kWkHours - 1) / kWkHours;
    g.walks = o; o = align256(o + 4LL * walk_words(rows, cols));
    g.codes = o; o = align256(o + 4LL * px * passes);
    g.words = o; o = align256(o + 4LL * 2 * kTrGroups * px * passes);
    g.total = o;
    return g;
}

}  // namespace
}  // namespace solweig

using namespace solweig;

extern "C" int64_t solweig_day_grad_work_bytes(int rows, int cols, int nhours) {
    if (rows <= 0 || cols <= 0 || nhours <= 0) return 0;
    return grad_work_layout(rows, cols, nhours).total;
}

// Shared forward of the gradient entry points: masks, parameter quads, GVF,
// contraction, tables.
static int grad_prepare(const SolweigScene* scene, const SolweigSkyLayout* layout, const SolweigHour* hours,
                        int nhours, const int32_t* gvf_dxdy, int first_steps, int second_steps,
                        const SolweigGradParams* prm, void* work, int64_t work_bytes, cudaStream_t st,
                        SolweigScene& Sp, GradWork& gw, DayWork& dw, DayWalkArgs& wa, bool& walk_words) {
    SOLWEIG_CHECK_ARG(scene && layout && hours && prm && work, "solweig_day_grad: null argument");
    SOLWEIG_CHECK_ARG(prm->albedo && prm->emissivity && prm->transmissivity, "solweig_day_grad: null parameter");
    const SolweigScene& S = *scene;
    SOLWEIG_CHECK_ARG(nhours > 0 && nhours <= kMaxGradHours, "solweig_day_grad: nhours %d outside 1..%d", nhours,
                      kMaxGradHours);
    SOLWEIG_CHECK_ARG(!S.has_water, "solweig_day_grad: scenes with water pixels are not supported");
    SOLWEIG_CHECK_ARG(S.patches == 153 || S.patches == 145, "solweig_day_grad: %d patches", S.patches);
    SOLWEIG_CHECK_ARG(first_steps == 1 && second_steps == 22 && gvf_dxdy,
                      "solweig_day_grad: only the 1 m GVF walk (first=1, second=22)");
    const long long px = (long long)S.rows * S.cols;
    gw = grad_work_layout(S.rows, S.cols, nhours);
    dw = day_work_layout(S.rows, S.cols, nhours, false);
    SOLWEIG_CHECK_ARG(work_bytes >= gw.total, "solweig_day_grad: work buffer of %lld bytes, need %lld",
                      (long long)work_bytes, gw.total);
    SOLWEIG_CHECK_ARG(((uintptr_t)work & 255) == 0, "solweig_day_grad: work buffer not 256-byte aligned");
    for (int i = 0; i < 2 * SOLWEIG_GVF_DIRECTIONS * 22; ++i)
        SOLWEIG_CHECK_ARG(gvf_dxdy[i] >= -21 && gvf_dxdy[i] <= 21, "solweig_day_grad: GVF offset outside the halo");
    char* wb = static_cast<char*>(work);
    float4* quads0 = reinterpret_cast<float4*>(wb + dw.quads);
    float4* quads1 = reinterpret_cast<float4*>(wb + gw.quads1);
    uint8_t* sv = reinterpret_cast<uint8_t*>(wb + gw.sv);
    float* gvf = reinterpret_cast<float*>(wb + gw.gvf);
    float* nosh = reinterpret_cast<float*>(wb + dw.nosh);
    float* sums = reinterpret_cast<float*>(wb + dw.sums);
    float* wf32 = reinterpret_cast<float*>(wb + dw.wf32);
    __nv_bfloat16* bw = reinterpret_cast<__nv_bfloat16*>(wb + dw.bw);
    DayTable* tables = reinterpret_cast<DayTable*>(wb + dw.tables);
    int* err = reinterpret_cast<int*>(wb + dw.error);
    // The batched day's sweep stage (ray ceilings, step records and the sweep,
    // which also clears the error flag) in the same work regions: 0.58 -> 0.25 ms
    // for 17 hours of 500 x 500 pixels against the sweep alone.
    const SolweigOutputs none{};
    int rc = solweig_day_batched_part(scene, layout, hours, nhours, nullptr, &none, 0, gvf_dxdy, first_steps,
                                      second_steps, work, work_bytes, nullptr, 0, 0, nhours, st);
    if (rc) return rc;
    param_quads_kernel<<<blocks_for(px * nhours, 256), 256, 0, st>>>(S, hours, nhours, quads0, quads1, sv,
                                                                      prm->albedo, prm->emissivity,
                                                                      prm->transmissivity, err);
    SOLWEIG_CHECK_LAUNCH("param_quads_kernel");
    Sp = S;
    Sp.emis = prm->emissivity;
    Sp.alb = prm->albedo;
    // Walks that start at their pixel go by walk words: the scene's own hold its
    // lengths, but the albedo-without-shadow plane is of these parameters, so
    // one launch makes both (500 x 500 pixels: 0.10 ms, and the GVF of 17 hours
    // 0.60 ms instead of 1.22 ms with one block per tile and hour).
    walk_words = day_walk_args(gvf_dxdy, second_steps, &wa);
    if (walk_words) {
        uint32_t* walks = reinterpret_cast<uint32_t*>(wb + gw.walks);
        rc = launch_gvf_walks(Sp, gvf_dxdy, second_steps, nullptr, walks, nosh, st);
        if (rc) return rc;
        wa.walks = walks;
        rc = launch_day_walk(Sp, hours, nhours, wa, quads1, reinterpret_cast<uint32_t*>(wb + gw.codes),
                             reinterpret_cast<unsigned long long*>(wb + dw.dict), gvf, nullptr, nosh, st);
        if (rc) return rc;
    } else {
        cudaMemsetAsync(nosh, 0, 4 * px, st);
        GvfTable<22> tab;
        fill_day_table(tab, gvf_dxdy, 22, 32 + 42);
        DayGvfArgs ga{1, 22, 21};
        launch_day_gvf<1, 22, 22>(16, Sp, hours, nhours, ga, tab, quads1, nullptr, gvf, nosh, st);
        SOLWEIG_CHECK_LAUNCH("day_gvf_kernel");
    }
    const int ncols = 2 * nhours;
    const int nb = (ncols + 15) / 16 * 16;
    day_weights_kernel<<<blocks_for((long long)ncols * kK, 256), 256, 0, st>>>(layout, hours, nhours, wf32);
    split_bf16_kernel<<<blocks_for((long long)nb * kK, 256), 256, 0, st>>>(wf32, ncols, nb, S.patches, bw);
    day_tables_kernel<<<nhours, kK, 0, st>>>(layout, hours, tables);
    SOLWEIG_CHECK_LAUNCH("day_tables_kernel");
    return launch_gemm(S.masks, px, S.patches, bw, ncols, nb, sums, err, st, 0);
}

static GradPtrs grad_ptrs(void* work, const GradWork& gw, const DayWork& dw, const SolweigGradParams* prm,
                          int nhours) {
    char* wb = static_cast<char*>(work);
    GradPtrs g{};
    g.alb = prm->albedo;
    g.emis = prm->emissivity;
    g.tau = prm->transmissivity;
    g.sv = reinterpret_cast<uint8_t*>(wb + gw.sv);
    g.quads = reinterpret_cast<float4*>(wb + gw.quads1);
    g.gvf = reinterpret_cast<float*>(wb + gw.gvf);
    g.nosh = reinterpret_cast<float*>(wb + dw.nosh);
    g.sums = reinterpret_cast<float*>(wb + dw.sums);
    g.ncols = 2 * nhours;
    g.lam_gl = reinterpret_cast<float*>(wb + gw.lam_gl);
    g.lam_ga = reinterpret_cast<float*>(wb + gw.lam_ga);
    g.lam_gn = reinterpret_cast<float*>(wb + gw.lam_gn);
    g.lam_s = reinterpret_cast<float*>(wb + gw.lam_s);
    g.lam_sums = reinterpret_cast<float*>(wb + gw.lam_sums);
    g.d_emis_direct = reinterpret_cast<float*>(wb + gw.d_emis_direct);
    return g;
}

template <bool BACK, typename... Args>
static void launch_grad_radiation(int patches, unsigned blocks, cudaStream_t st, Args... args) {
    if (patches == 153) grad_radiation_kernel<2, BACK><<<blocks, kGradThreads, 0, st>>>(args...);
    else grad_radiation_kernel<1, BACK><<<blocks, kGradThreads, 0, st>>>(args...);
}

extern "C" int solweig_day_grad_forward(const SolweigScene* scene, const SolweigSkyLayout* layout,
                                        const SolweigHour* hours, int nhours, const int32_t* gvf_dxdy,
                                        int first_steps, int second_steps, const SolweigGradParams* params,
                                        int objective, double* daily, void* work, int64_t work_bytes, void* stream) {
    SOLWEIG_CHECK_ARG(daily && (objective == 0 || objective == 1), "solweig_day_grad_forward: bad arguments");
    cudaStream_t st = as_stream(stream);
    SolweigScene Sp;
    GradWork gw;
    DayWork dw;
    DayWalkArgs wa;
    bool walk_words;
    int rc = grad_prepare(scene, layout, hours, nhours, gvf_dxdy, first_steps, second_steps, params, work,
                          work_bytes, st, Sp, gw, dw, wa, walk_words);
    if (rc) return rc;
    GradPtrs g = grad_ptrs(work, gw, dw, params, nhours);
    g.daily = daily;
    g.weights = nullptr;
    g.objective = objective;
    const long long px = (long long)scene->rows * scene->cols;
    DayTable* tables = reinterpret_cast<DayTable*>(static_cast<char*>(work) + dw.tables);
    launch_grad_radiation<false>(scene->patches, blocks_for(px, kGradThreads), st, Sp, layout, hours, nhours,
                          (const DayTable*)tables, g);
    SOLWEIG_CHECK_LAUNCH("grad_radiation_kernel");
    return SOLWEIG_OK;
}

extern "C" int solweig_day_grad_backward(const SolweigScene* scene, const SolweigSkyLayout* layout,
                                         const SolweigHour* hours, int nhours, const int32_t* gvf_dxdy,
                                         int first_steps, int second_steps, const SolweigGradParams* params,
                                         int objective, const float* weights, float* d_albedo,
                                         float* d_emissivity, float* d_transmissivity, double* hour_grad,
                                         double* lum_grad, void* work, int64_t work_bytes, void* stream) {
    SOLWEIG_CHECK_ARG(weights && d_albedo && d_emissivity && d_transmissivity && hour_grad && lum_grad &&
                          (objective == 0 || objective == 1),
                      "solweig_day_grad_backward: bad arguments");
    cudaStream_t st = as_stream(stream);
    SolweigScene Sp;
    GradWork gw;
    DayWork dw;
    DayWalkArgs wa;
    bool walk_words;
    int rc = grad_prepare(scene, layout, hours, nhours, gvf_dxdy, first_steps, second_steps, params, work,
                          work_bytes, st, Sp, gw, dw, wa, walk_words);
    if (rc) return rc;
    const long long px = (long long)scene->rows * scene->cols;
    char* wb = static_cast<char*>(work);
    GradPtrs g = grad_ptrs(work, gw, dw, params, nhours);
    g.daily = nullptr;
    g.weights = weights;
    g.objective = objective;
    g.hour_grad = hour_grad;
    cudaMemsetAsync(hour_grad, 0, sizeof(double) * kGFields * nhours, st);
    cudaMemsetAsync(lum_grad, 0, sizeof(double) * 4 * kK * nhours, st);
    cudaMemsetAsync(wb + gw.lam_alb, 0, 4LL * px, st);
    DayTable* tables = reinterpret_cast<DayTable*>(wb + dw.tables);
    launch_grad_radiation<true>(scene->patches, blocks_for(px, kGradThreads), st, Sp, layout, hours, nhours,
                          (const DayTable*)tables, g);
    SOLWEIG_CHECK_LAUNCH("grad_radiation_kernel");
    GvfAdjPtrs ap{g.lam_gl, g.lam_ga, g.lam_gn, reinterpret_cast<float*>(wb + gw.lam_lup),
                  reinterpret_cast<float*>(wb + gw.lam_albsh), reinterpret_cast<float*>(wb + gw.lam_alb), hour_grad};
    if (walk_words) {
        rc = launch_gvf_transpose(Sp, hours, nhours, gvf_dxdy, wa, reinterpret_cast<uint32_t*>(wb + gw.words), ap, st);
        if (rc) return rc;
    } else {
        cudaMemsetAsync(wb + gw.lam_lup, 0, 4LL * px * nhours, st);
        cudaMemsetAsync(wb + gw.lam_albsh, 0, 4LL * px * nhours, st);
        GvfTable<22> tab;
        fill_day_table(tab, gvf_dxdy, 22, 32 + 42);
        constexpr int TY = 8;
        const size_t smem = sizeof(float4) * (size_t)(32 + 42) * (TY + 42);
        set_smem_attr((const void*)gvf_adjoint_kernel<TY>, smem);
        dim3 grid(blocks_for(scene->cols, 32), blocks_for(scene->rows, TY), nhours);
        gvf_adjoint_kernel<TY><<<grid, dim3(32, TY), smem, st>>>(Sp, hours, tab, g.quads, ap);
        SOLWEIG_CHECK_LAUNCH("gvf_adjoint_kernel");
    }
    param_grad_kernel<<<blocks_for(px, 256), 256, 0, st>>>(
        Sp, hours, nhours, g.quads, g.sv, params->albedo, params->emissivity, ap.lam_lup, ap.lam_albsh,
        ap.lam_alb, g.lam_s, g.d_emis_direct, d_albedo, d_emissivity, d_transmissivity, hour_grad);
    SOLWEIG_CHECK_LAUNCH("param_grad_kernel");
    {
        // two blocks per SM if the pixels of all hours give them, at least 32 pixels a warp
        const int passes = (nhours + kLumHours - 1) / kLumHours;
        const long long spread = (px * passes + 148 * 2 * kLumWarps - 1) / (148 * 2 * kLumWarps);
        const int warp_pixels = (int)std::min<long long>(kLumPixels, std::max<long long>(32, (spread + 31) / 32 * 32));
        dim3 grid(blocks_for(px, kLumWarps * warp_pixels), passes);
        lum_grad_kernel<<<grid, 32 * kLumWarps, 0, st>>>(Sp, hours, nhours, g.lam_sums, warp_pixels, lum_grad);
        SOLWEIG_CHECK_LAUNCH("lum_grad_kernel");
    }
    return SOLWEIG_OK;
}
