"""The native host plan (``solweig_plan_hours``) against the numpy functions it
follows (``sun.clearness_index``, ``sun.diffuse_fraction``, ``sky.perez``,
``sky.band_emissivity``, ``rays.shadow_ray``, each pinned to the reference):
sun rays identical, scalars to float64 rounding."""
import types

import numpy as np
import pytest

RTOL = 1e-13  # chains of some tens of float64 operations


def _scene(shape, scale):
    from solweig_cuda_b200 import engine
    return types.SimpleNamespace(layout=engine.SkyLayout(2), tgk_wall=0.58, tstart_wall=-3.41, tmaxlst_wall=15.0,
                                 scale=scale, amaxvalue=37.5, shape=shape, landcover=1)


@pytest.mark.parametrize("doy,lat,shape,scale,missing", [
    (172, 53.0, (300, 250), 1.0, False), (20, 47.0, (60, 517), 0.5, False), (355, 66.0, (33, 40), 1.0, False),
    (80, 0.0, (2, 1500), 2.0, False), (250, -38.0, (700, 64), 1.0, True)])
def test_native_plan_matches_numpy(doy, lat, shape, scale, missing):
    from solweig_cuda_b200 import engine, rays, sky, sun, synthetic
    scene = _scene(shape, scale)
    L = scene.layout.host
    met = synthetic.make_met(doy=doy, latitude=lat, longitude=10.0, seed=doy)
    if missing:
        met[:, 12] = -999.0  # no pressure
        met[13, 14] = 5.0    # overcast noon: diffuse radiation at most 10 W/m2
    sol = sun.metdata(met, lat, 10.0, 3.0, 1.0)
    plan = engine.plan_day(scene, met, lat, 10.0, 3.0, 1.0)
    assert len(plan) == 24
    ci, seen = 1.0, set()
    for i, (h, ray, scal) in enumerate(plan):
        day = sol.altitude[i] > 0
        seen.add(bool(day))
        if sol.dectime[i] == np.floor(sol.dectime[i]):
            ci = 1.0
        assert h.daytime == int(day)
        if day:
            want = rays.shadow_ray(sol.azimuth[i], sol.altitude[i], scale, 37.5, shape)
            assert np.array_equal(ray.dxdy, want.dxdy) and np.array_equal(ray.dz, want.dz)
            assert (ray.low, ray.high, ray.middle) == (want.low, want.high, want.middle)
            i0, ci, kt, _, _ = sun.clearness_index(sol.zen[i], sol.jday[i], met[i, 11], met[i, 10] / 100., met[i, 14],
                                                   lat, met[i, 12])
            ci = min(float(ci), 1.0)
            rad_i, rad_d = sun.diffuse_fraction(met[i, 14], sol.altitude[i], kt, met[i, 11], met[i, 10])
            lv = sky.perez(sol.zen[i] * (180 / np.pi), sol.azimuth[i], rad_d, rad_i, sol.jday[i], L)
            np.testing.assert_allclose(scal.lv, lv, rtol=RTOL)
            np.testing.assert_allclose([scal.I0, scal.radI, scal.radD], [i0, rad_i, rad_d], rtol=RTOL, atol=1e-9)
            yi = 2 * np.cos(np.abs(sol.azimuth[i] - L.azimuth) * (np.pi / 180)) * np.tan(sol.altitude[i] * (np.pi / 180))
            np.testing.assert_allclose(np.ctypeslib.as_array(h.yi)[:L.count], np.minimum(yi, 0), rtol=1e-12, atol=1e-12)
            np.testing.assert_allclose(h.rad_tot, np.sum(lv[:, 2] * L.steradian * L.sin_alt), rtol=1e-12)
        else:
            assert ray is None and scal.lv is None and h.rad_tot == 1.0
        ea = 6.107 * 10 ** ((7.5 * met[i, 11]) / (237.3 + met[i, 11])) * (met[i, 10] / 100.)
        m = 46.5 * (ea / (met[i, 11] + 273.15))
        esky = 1 - (1 + m) * np.exp(-((1.2 + 3.0 * m) ** 0.5))
        if ci < 0.95:
            esky = ci * esky + (1 - ci)
        np.testing.assert_allclose([scal.CI, scal.ea, scal.esky], [ci, ea, esky], rtol=RTOL)
        band = sky.band_emissivity(esky, L)[L.band_offsets[:-1]] * engine.SBC * (met[i, 11] + 273.15) ** 4 / np.pi
        np.testing.assert_allclose(scal.band_lsky, band, rtol=RTOL)
        np.testing.assert_allclose(h.snup, sun.daylen(sol.jday[i], lat)[3], rtol=RTOL)
    assert seen == ({True, False} if abs(lat) < 66 else seen)
    # one hour alone gives the record of the day, and a latitude without a clearness model is refused
    h, _, scal, _ = engine.hour_plan(scene, lat, sol.altitude[12], sol.azimuth[12], sol.zen[12], sol.jday[12],
                                     sol.dectime[12], sol.altmax[12], met[12, 11], met[12, 10], met[12, 14], met[12, 21],
                                     met[12, 22], met[12, 12], met[12, 9], plan[12][0].psi, plan[11][2].CI,
                                     plan[12][0].firstdaytime, 0.0, 1 / 24., plan[12][0].twater)
    assert h.rad_d == plan[12][0].rad_d and h.esky == plan[12][0].esky and scal.CI == plan[12][2].CI
    if plan[12][0].daytime:
        with pytest.raises(RuntimeError, match="latitude"):
            engine.hour_plan(scene, 90.0, sol.altitude[12], sol.azimuth[12], sol.zen[12], sol.jday[12],
                             sol.dectime[12], sol.altmax[12], 20.0, 50.0, 300.0, -999.0, -999.0, 101.3, 2.0, 0.03, 1.0,
                             1, 0.0, 1 / 24., None)
