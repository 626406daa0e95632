// Host plan of forcing hours: the FP64 scalars, per-patch weights and sun ray
// of every hour (src/umep_solweig.py:122-232, src/model.py:808-958), written
// straight into SolweigHour records.
//
// The sun positions and the trigonometry of the sun's angles come from the
// caller, because the digital ray has to round exactly as numpy's; the rest
// (clearness index, diffuse split, Perez luminance of every patch, sky
// emissivities, wave-delay clock, UTCI coefficients) is evaluated here.  A day
// of 24 hours takes 0.1 ms; interpreted hour by hour it took 3.8 ms, longer
// than the GPU needs for a day of 1000 x 1000 px.
#include <math.h>
#include <string.h>

#include "common.cuh"

namespace solweig {

namespace {

constexpr double kD2R = kPi / 180.0;

// Perez (1993) coefficients: rows a1..a4, b1..b4, c1..c4, d1..d4, e1..e4, columns the 8 clearness bins.
constexpr double kPerez[20][8] = {
    {1.3525, -1.2219, -1.1000, -0.5484, -0.6000, -1.0156, -1.0000, -1.0500},
    {-0.2576, -0.7730, -0.2515, -0.6654, -0.3566, -0.3670, 0.0211, 0.0289},
    {-0.2690, 1.4148, 0.8952, -0.2672, -2.5000, 1.0078, 0.5025, 0.4260},
    {-1.4366, 1.1016, 0.0156, 0.7117, 2.3250, 1.4051, -0.5119, 0.3590},
    {-0.7670, -0.2054, 0.2782, 0.7234, 0.2937, 0.2875, -0.3000, -0.3250},
    {0.0007, 0.0367, -0.1812, -0.6219, 0.0496, -0.5328, 0.1922, 0.1156},
    {1.2734, -3.9128, -4.5000, -5.6812, -5.6812, -3.8500, 0.7023, 0.7781},
    {-0.1233, 0.9156, 1.1766, 2.6297, 1.8415, 3.3750, -1.6317, 0.0025},
    {2.8000, 6.9750, 24.7219, 33.3389, 21.0000, 14.0000, 19.0000, 31.0625},
    {0.6004, 0.1774, -13.0812, -18.3000, -4.7656, -0.9999, -5.0000, -14.5000},
    {1.2375, 6.4477, -37.7000, -62.2500, -21.5906, -7.1406, 1.2438, -46.1148},
    {1.0000, -0.1239, 34.8438, 52.0781, 7.2492, 7.5469, -1.9094, 55.3750},
    {1.8734, -1.5798, -5.0000, -3.5000, -3.5000, -3.4000, -4.0000, -7.2312},
    {0.6297, -0.5081, 1.5218, 0.0016, -0.1554, -0.1078, 0.0250, 0.4050},
    {0.9738, -1.7812, 3.9229, 1.1477, 1.4062, -1.0750, 0.3844, 13.3500},
    {0.2809, 0.1080, -2.6204, 0.1062, 0.3988, 1.5702, 0.2656, 0.6234},
    {0.0356, 0.2624, -0.0156, 0.4659, 0.0032, -0.0672, 1.0468, 1.5000},
    {-0.1246, 0.0672, 0.1597, -0.3296, 0.0766, 0.4016, -0.3788, -0.6426},
    {-0.5718, -0.2190, 0.4199, -0.0876, -0.0656, 0.3017, -2.4517, 1.8564},
    {0.9938, -0.4285, -0.5562, -0.0329, -0.1294, -0.4844, 1.4656, 0.5636},
};

// Empirical precipitable-water exponent by latitude band (upper bound) and season.
struct WaterBand {
    double below;
    double g[4];
};
constexpr WaterBand kWaterBands[] = {
    {10., {3.37, 2.85, 2.80, 2.64}}, {20., {2.99, 3.02, 2.70, 2.93}}, {30., {3.60, 3.00, 2.98, 2.93}},
    {40., {3.04, 3.11, 2.92, 2.94}}, {50., {2.70, 2.95, 2.77, 2.71}}, {60., {2.52, 3.07, 2.67, 2.93}},
    {70., {1.76, 2.69, 2.61, 2.61}}, {80., {1.60, 1.67, 2.24, 2.63}}, {90., {1.11, 1.44, 1.94, 2.02}},
};

// Sunrise (hours), daylen of src/umep_solweig.py:430-448.
double sunrise(double doy, double latitude) {
    const double dec = -23.45 * cos(2.0 * kPi * (doy + 10.0) / 365.0);
    double soc = tan(kD2R * dec) * tan(kD2R * latitude);
    soc = soc > -1.0 ? soc : -1.0;
    soc = soc < 1.0 ? soc : 1.0;
    return 12.0 - (12.0 + 24.0 * asin(soc) / kPi) / 2.0;
}

struct Clearness {
    double i0, ci, kt;
};

// Crawford & Duchon clearness index (src/umep_solweig.py:1654-1734); g: the
// precipitable-water exponent of the latitude and season.
Clearness clearness_index(double zen, double jday, double ta, double rh_fraction, double rad_g, double g,
                          double p_kpa) {
    const double p = p_kpa == -999.0 ? 1013. : p_kpa * 10.;
    const double itoa = 1370.0;
    const double b = 2. * kPi * jday / 365.;
    const double d = sqrt(1.00011 + 0.034221 * cos(b) + 0.001280 * sin(b) + 0.000719 * cos(2. * b) +
                          0.000077 * sin(2. * b));
    const double cz = cos(zen);
    const double m = 35. * cz * pow(1224. * (cz * cz) + 1., -1. / 2.);
    const double trpg = 1.021 - 0.084 * pow(m * (0.000949 * p + 0.051), 0.5);
    const double a2 = 17.27, b2 = 237.7;
    const double x = ((a2 * ta) / (b2 + ta)) + log(rh_fraction);
    double td = (b2 * x) / (a2 - x);
    td = (td * 1.8) + 32;
    const double u = exp(0.1133 - log(g + 1) + 0.0393 * td);
    const double tw = 1 - 0.077 * pow(u * m, 0.3);
    const double tar = pow(0.935, m);
    Clearness c;
    c.i0 = itoa * cz * trpg * tw * d * tar;
    if (fabs(zen) > kPi / 2) c.i0 = 0;
    const double corr = 0.1473 * log(90 - (zen / kPi * 180)) + 0.3454;
    c.ci = rad_g / c.i0 + (1 - corr);
    c.kt = rad_g / (itoa * cz * d);
    if (isnan(c.ci)) c.ci = HUGE_VAL;
    return c;
}

// Reindl et al. (1990) direct / diffuse split (src/umep_solweig.py:1789-1832).
void diffuse_fraction(double rad_g, double altitude, double kt, double ta, double rh, double* rad_i, double* rad_d) {
    const double s = sin(altitude * (kPi / 180));
    double d;
    if (ta <= -999.00 || rh <= -999.00 || isnan(ta) || isnan(rh)) {
        if (kt <= 0.3) d = rad_g * (1.020 - 0.248 * kt);
        else if (kt < 0.78) d = rad_g * (1.45 - 1.67 * kt);
        else d = rad_g * 0.147;
    } else {
        const double rhf = rh / 100;
        if (kt <= 0.3) d = rad_g * (1 - 0.232 * kt + 0.0239 * s - 0.000682 * ta + 0.0195 * rhf);
        else if (kt < 0.78) d = rad_g * (1.329 - 1.716 * kt + 0.267 * s - 0.00357 * ta + 0.106 * rhf);
        else d = rad_g * (0.426 * kt - 0.256 * s + 0.00349 * ta + 0.0734 * rhf);
    }
    double i = (rad_g - d) / s;
    if (i < 0) i = 0;
    if (altitude < 1 && i > rad_g) i = rad_g;
    if (d > rad_g) d = rad_g;
    *rad_i = i;
    *rad_d = d;
}

// Perez clearness bin: strict on both sides of every edge, bin 0 on an edge.
int clearness_bin(double eps) {
    constexpr double edges[7] = {1.065, 1.230, 1.500, 1.950, 2.800, 4.500, 6.200};
    int b = 0;
    for (int i = 0; i < 6; ++i)
        if (edges[i] < eps && eps < edges[i + 1]) b = i + 1;
    if (eps > edges[6]) b = 7;
    return b;
}

// Perez relative luminance of every patch, normalised to sum 1 (src/model.py:808-958).
void perez(const SolweigPlanScene& s, double zen_deg, double azimuth, double rad_d, double rad_i, double jday,
           double* lum) {
    const double altitude = (90 - zen_deg) * kD2R, zen = zen_deg * kD2R, az = azimuth * kD2R;
    const double z3 = 1.041 * pow(zen, 3);
    const double eps = ((rad_d + rad_i) / (rad_d + z3)) / (1 + z3);
    const double day = jday * 2 * kPi / 365;
    const double i0 = 1367 * (1.00011 + 0.034221 * cos(day) + 0.00128 * sin(day) + 0.000719 * cos(2 * day) +
                              0.000077 * sin(2 * day));
    const double sa = sin(altitude), ca = cos(altitude);
    const double airmass =
        altitude >= 10 * kD2R ? 1 / sa : 1 / sa + 0.50572 * pow(180 * altitude / kPi + 6.07995, -1.6364);
    const double delta = rad_d <= 10 ? 0.0 : (airmass * rad_d) / i0;
    const int b = clearness_bin(eps);
    auto c = [&](int r) { return kPerez[r][b]; };
    auto coef = [&](int j) {
        return c(4 * j) + c(4 * j + 1) * zen + delta * (c(4 * j + 2) + c(4 * j + 3) * zen);
    };
    const double ma = coef(0), mb = coef(1), me = coef(4);
    const double mc = b > 0 ? coef(2) : exp(pow(delta * (c(8) + c(9) * zen), c(10))) - 1;
    const double md = b > 0 ? coef(3) : -exp(delta * (c(12) + c(13) * zen)) + c(14) + delta * c(15) * delta;
    double total = 0;
    for (int k = 0; k < s.patches; ++k) {
        double cs = s.sin_alt[k] * sa + ca * s.cos_alt[k] * cos(fabs(s.azimuth[k] * kD2R - az));
        cs = cs < -1.0 ? -1.0 : cs > 1.0 ? 1.0 : cs;
        lum[k] = (1 + ma * exp(mb / s.cos_zen[k])) * (1 + mc * exp(md * acos(cs)) + me * cs * cs);
        total += lum[k];
    }
    for (int k = 0; k < s.patches; ++k) lum[k] /= total;
}

// Steps of the sun ray up to and including the first one above `maximum` or
// outside the raster (src/umep_solweig.py:2289-2318); rint rounds half to
// even as numpy does.
int sun_ray(const SolweigPlanScene& s, const SolweigPlanRow& r, int capacity, int32_t* dxdy, double* dz) {
    if (s.amaxvalue < 0) return 0;
    const double az = r.azimuth * (kPi / 180.), q = kPi / 4;
    const bool ymajor = (q <= az && az < 3 * q) || (5 * q <= az && az < 7 * q);
    auto sign = [](double x) { return x > 0 ? 1.0 : x < 0 ? -1.0 : x; };
    const double sx = -sign(r.cos_az), sy = sign(r.sin_az);
    const double ds = fabs(1 / (ymajor ? r.sin_az : r.cos_az)), tanab = r.tan_alt / s.scale;
    const int n = (s.rows > s.cols ? s.rows : s.cols) + 2;
    int k = 0;
    while (k < n && k < capacity) {
        const double minor = fabs(rint(ymajor ? k / r.tan_az : k * r.tan_az));
        const double dx = sx * (ymajor ? minor : k), dy = sy * (ymajor ? k : minor), z = (ds * k) * tanab;
        dxdy[2 * k] = (int32_t)dx;
        dxdy[2 * k + 1] = (int32_t)dy;
        dz[k] = z;
        ++k;
        if (!(s.amaxvalue >= z) || fabs(dx) >= s.rows || fabs(dy) >= s.cols) break;
    }
    return k;
}

// Self-shadow azimuth window of the walls.
void sun_window(double az, SolweigHour* h) {
    double low = az - kPi / 2, high = az + kPi / 2;
    const bool middle = low >= 0 && high < 2 * kPi;
    if (!middle) {
        if (low < 0 && high <= 2 * kPi) low += 2 * kPi;
        else high -= 2 * kPi;
    }
    h->ray_low = low;
    h->ray_high = high;
    h->ray_middle = middle;
}

int plan_hour(const SolweigPlanScene& s, const SolweigPlanRow& r, double step, double twater, SolweigPlanState* st,
              SolweigHour* h, SolweigPlanScalars* out, int32_t* dxdy, double* dz, int capacity, double* lum) {
    memset(h, 0, sizeof(*h));
    memset(out, 0, sizeof(*out));
    if (r.new_day) st->ci = 1.;
    const double snup = sunrise(r.jday, s.latitude);
    const double ea = 6.107 * pow(10., (7.5 * r.ta) / (237.3 + r.ta)) * (r.rh / 100.);
    const double msteg = 46.5 * (ea / (r.ta + 273.15));
    double esky = 1 - (1 + msteg) * exp(-pow(1.2 + 3.0 * msteg, 0.5));
    const bool day = r.altitude > 0;
    double ci = st->ci, rad_i = r.rad_i, rad_d = r.rad_d;
    out->ci_tg = out->ci_tgg = ci;
    const double frac = r.dectime - floor(r.dectime);
    if (day) {
        const double* g4 = nullptr;
        for (const WaterBand& w : kWaterBands)
            if (s.latitude < w.below) {
                g4 = w.g;
                break;
            }
        SOLWEIG_CHECK_ARG(g4, "solweig_plan_hours: latitude %g is not below 90 degrees", s.latitude);
        const double g = (r.jday > 335 || r.jday <= 60) ? g4[0] : r.jday <= 152 ? g4[1] : r.jday <= 244 ? g4[2] : g4[3];
        const Clearness c = clearness_index(r.zen, r.jday, r.ta, r.rh / 100., r.rad_g, g, r.p_kpa);
        ci = c.ci > 1 ? 1. : c.ci;
        diffuse_fraction(r.rad_g, r.altitude, c.kt, r.ta, r.rh, &rad_i, &rad_d);
        perez(s, r.zen * (180 / kPi), r.azimuth, rad_d, rad_i, r.jday, lum);
        double tgwall = (s.tgk_wall * r.altmax + s.tstart_wall) *
                        sin(((frac - snup / 24) / (s.tmaxlst_wall / 24 - snup / 24)) * kPi / 2);
        if (tgwall < 0) tgwall = 0;
        double i1, d1;
        diffuse_fraction(c.i0, r.altitude, 1., r.ta, r.rh, &i1, &d1);
        const double corr = 0.1473 * log(90 - (r.zen / kPi * 180)) + 0.3454;
        out->i0 = c.i0;
        out->ci_tg = r.rad_g / i1 + (1 - corr);
        if (out->ci_tg > 1) out->ci_tg = 1;
        out->ci_tgg = r.rad_g / (i1 * r.sin_alt + d1) + (1 - corr);
        if (out->ci_tgg > 1) out->ci_tgg = 1;
        h->tgwall = tgwall * out->ci_tgg;
        h->steps = sun_ray(s, r, capacity, dxdy, dz);
        sun_window(r.azimuth * (kPi / 180.), h);
        // wave-delay flags (all six TsWaveDelay calls share them)
        h->firstdaytime = (int32_t)st->firstdaytime;
        if (st->timeadd >= 59. / 1440) {
            h->wave_weight = exp(-33.27 * st->timeadd);
            h->wave_update = 1;
            st->timeadd = step > 59. / 1440 ? step : 0;
        } else {
            st->timeadd += step;
            h->wave_weight = exp(-33.27 * st->timeadd);
        }
        st->firstdaytime = 0;
        double total = 0;  // in patch order, as the reference's loop
        for (int k = 0; k < s.patches; ++k) {
            total += lum[k] * s.steradian[k] * s.sin_alt[k];
            const double diff = fabs(r.azimuth - s.azimuth[k]);
            const double yi = 2 * cos(diff * (kPi / 180)) * r.tan_alt;
            h->lum[k] = (float)lum[k];
            h->yi[k] = yi > 0 ? 0. : yi;
            h->lw_sun_test[k] = diff > 90 && diff < 270;
        }
        h->rad_tot = total;
    } else {
        st->firstdaytime = 1;
        st->timeadd = 0;
        h->rad_tot = 1.;
        for (int k = 0; k < s.patches; ++k) lum[k] = 0.;
    }
    st->ci = ci;
    if (ci < 0.95) esky = ci * esky + (1 - ci) * 1.;
    h->daytime = day;
    h->altitude = r.altitude;
    h->azimuth = r.azimuth;
    h->zen = r.zen;
    h->ta = r.ta;
    h->rh = r.rh;
    h->ws = r.ws;
    h->rad_g = r.rad_g;
    h->rad_d = rad_d;
    h->rad_i = rad_i;
    h->psi = r.psi;
    h->cos_alt = r.cos_alt;
    h->sin_alt = r.sin_alt;
    h->tan_zen = r.tan_zen;
    h->esky = esky;
    h->ci_tgg = day ? out->ci_tgg : 0.0;
    h->altmax = r.altmax;
    h->dectime_frac = frac;
    h->snup = snup;
    h->twater = twater;
    const double tk = r.ta + 273.15, base = kSBC * ((tk * tk) * (tk * tk));
    for (int b = 0; b < s.nbands; ++b) {  // Martin & Berdahl sky emissivity of a band
        out->band_lsky[b] = ((1 - (1 - esky) * exp(0.308 * (1.7 - s.band_inv_cos[b]))) * base) / kPi;
        h->band_lsky[b] = (float)out->band_lsky[b];
    }
    const float ta = (float)r.ta, rh = (float)r.rh, ws = (float)r.ws;
    const int rc = solweig_utci_collapse(ta, rh, ws, h->utci);
    if (rc) return rc;
    h->utci_valid = !(ta <= -999 || rh <= -999 || ws <= -999);
    out->ea = ea;
    out->esky = esky;
    out->ci = ci;
    out->rad_i = rad_i;
    out->rad_d = rad_d;
    out->tgwall = h->tgwall;
    out->steps = h->steps;
    return SOLWEIG_OK;
}

}  // namespace

}  // namespace solweig

using namespace solweig;

extern "C" int solweig_plan_hours(const SolweigPlanScene* scene, const SolweigPlanRow* rows, int n, double timestepdec,
                                  double twater, SolweigPlanState* state, SolweigHour* hours,
                                  SolweigPlanScalars* scalars, int32_t* ray_dxdy, double* ray_dz, int ray_capacity,
                                  double* luminance) {
    SOLWEIG_CHECK_ARG(scene && rows && state && hours && scalars && ray_dxdy && ray_dz && luminance,
                      "solweig_plan_hours: null argument");
    SOLWEIG_CHECK_ARG(n >= 0 && ray_capacity >= 1, "solweig_plan_hours: %d hours, ray capacity %d", n, ray_capacity);
    SOLWEIG_CHECK_ARG(scene->patches > 0 && scene->patches <= SOLWEIG_MAX_PATCHES && scene->nbands > 0 &&
                          scene->nbands <= SOLWEIG_MAX_BANDS,
                      "solweig_plan_hours: %d patches, %d bands", scene->patches, scene->nbands);
    for (int i = 0; i < n; ++i) {
        const int rc = plan_hour(*scene, rows[i], timestepdec, twater, state, hours + i, scalars + i,
                                 ray_dxdy + 2LL * i * ray_capacity, ray_dz + 1LL * i * ray_capacity, ray_capacity,
                                 luminance + 1LL * i * SOLWEIG_MAX_PATCHES);
        if (rc) return rc;
    }
    return SOLWEIG_OK;
}
