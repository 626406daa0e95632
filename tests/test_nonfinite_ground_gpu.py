"""A ground pixel whose albedo or emissivity is not a number or infinite: it
reaches the pixels whose walks read it, at most a walk (21 pixels) away, whether
the ground view factors count their samples or add them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS, COLS = 97, 70


def _scene(field, value):
    from solweig_cuda_b200 import engine, synthetic
    s = synthetic.make_scene(ROWS, COLS, seed=11, building_cover=0.2)
    scene = engine.Scene(s.dsm, s.trees, s.dem, 1.0, landcover=s.landcover)
    ground = (scene.flags.cpu().numpy() & 1) != 0
    r, c = np.argwhere(ground)[np.abs(np.argwhere(ground) - (40, 36)).sum(axis=1).argmin()]
    getattr(scene, field)[r, c] = value
    scene._gvf_statics(engine.stream_handle())
    return scene, (r, c)


def _day(scene, met, hv):
    """GVF planes [24, 2, rows, cols] (Lup, albedo), Tmrt and the daytime hours of
    the walk-word kernel (hv 1) or the per-hour kernel (hv 0)."""
    import torch
    from solweig_cuda_b200 import _lib, batched
    day = batched.ChosenDay(scene, 48.0, 0.0, 3.0, 0.0, outputs=("tmrt",))
    cfg = _lib.SolweigDayConfig.default()
    cfg.gvf_hours = hv
    day.set_config(cfg)
    tmrt = day.run_day(met)["tmrt"].clone()
    torch.cuda.synchronize()
    at, n = day.work_offsets()["gvf"], scene.pixels
    gvf = day.work[at:at + 12 * 24 * n].view(torch.float32).view(24, 3, ROWS, COLS)[:, :2].clone()
    return gvf, tmrt, [h.daytime for h, _, _ in day.plan(met)]


@pytest.mark.parametrize("field", ["alb", "emis"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_reaches_the_walks_that_read_it(cuda, field, value):
    """The walk-word kernel is finite exactly where the per-hour kernel is, and
    the values there agree to the rounding of their sums."""
    import torch
    from solweig_cuda_b200 import synthetic
    scene, (r, c) = _scene(field, value)
    met = synthetic.make_met(doy=100, latitude=48.0, longitude=0.0, seed=2)
    g0, t0, days = _day(scene, met, 0)
    g1, t1, _ = _day(scene, met, 1)
    assert torch.equal(torch.isfinite(t1), torch.isfinite(t0))
    eps, plane = 40 * 2.0 ** -24, 0 if field == "emis" else 1
    for h, d in enumerate(days):
        if not d:
            continue
        for k in (0, 1):
            ok = torch.isfinite(g0[h, k])
            assert torch.equal(torch.isfinite(g1[h, k]), ok), (h, k)
            a, b = g0[h, k][ok], g1[h, k][ok]
            torch.testing.assert_close(b, a, rtol=eps, atol=eps * max(1.0, float(a.abs().max())))
        bad = (~torch.isfinite(g1[h, plane])).nonzero().cpu().numpy()
        assert len(bad) and np.abs(bad - (r, c)).max() <= 21


@pytest.mark.parametrize("field", ["alb", "emis"])
def test_gradient_forward(cuda, field):
    """The gradient's forward with the same fields is not a number where the day is."""
    import torch
    from solweig_cuda_b200 import grad, synthetic
    scene, _ = _scene(field, float("nan"))
    met = synthetic.make_met(doy=100, latitude=48.0, longitude=0.0, seed=2)
    _, tmrt, _ = _day(scene, met, 0)
    dg = grad.DayGradient(scene, 48.0, 0.0, 3.0, 0.0, objective="tmrt")
    tau = torch.full(scene.shape, 0.03, device=scene.device)
    daily = dg.forward(scene.alb, scene.emis, tau, met)
    assert torch.equal(torch.isnan(daily), torch.isnan(tmrt).any(dim=0))
    assert not bool(torch.isnan(daily).all())
