"""Calls of the engine that its own day runners do not make: the plan of a day as a
list and hour by hour, host work beside the wall aspect, the rays' step count."""
import types

import numpy as np
import pytest


def _plans():
    from solweig_cuda_b200 import engine, synthetic
    scene = types.SimpleNamespace(layout=engine.SkyLayout(2), tgk_wall=0.37, tstart_wall=-3.41, tmaxlst_wall=15.0,
                                  scale=1.0, amaxvalue=20.0, shape=(40, 60), landcover=1)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    args = (scene, met, 53.0, 0.0, 3.0, 0.0)
    return engine.plan_day(*args), engine.plan_hours(*args)


def _key(hour):
    h, ray, scal = hour
    return h.daytime, h.rad_tot, h.lum[7], None if ray is None else ray.dz.tobytes(), scal.esky


def test_a_plan_reads_like_a_list_of_its_hours():
    plan, hours = _plans()
    whole = [_key(h) for h in plan]
    assert len(whole) == len(plan) == 24 and [_key(h) for h in hours] == whole
    for part in (slice(2, 9), slice(None, None, 5), slice(-3, None), slice(5, 5)):
        assert [_key(h) for h in plan[part]] == whole[part]
    assert _key(plan[-1]) == whole[-1] and [_key(h) for h in reversed(plan)] == whole[::-1]
    assert [_key(h) for h in plan + plan[:2]] == whole + whole[:2]
    assert [_key(h) for h in plan[:2] + plan] == whole[:2] + whole
    with pytest.raises(IndexError):
        plan[24]


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [True, False])
def test_host_work_runs_once_beside_the_aspect(cuda, walls):
    import torch
    from solweig_cuda_b200 import engine, synthetic
    dsm = synthetic.make_scene(60, 70, seed=3).dsm.astype(np.float64) if walls else np.zeros((60, 70))
    dev = torch.from_numpy(dsm).to(cuda)
    heights = engine.wall_heights_device(dev, 3.0)
    done = []
    got = engine.wall_aspect_device(dsm, dev, heights, 1.0, host_work=lambda: done.append(1))
    assert done == [1]
    assert torch.equal(got, engine.wall_aspect_device(dsm, dev, heights, 1.0))


@pytest.mark.gpu
def test_svf_steps_counts_the_rays(cuda):
    from solweig_cuda_b200 import engine, rays, synthetic
    c = synthetic.make_scene(48, 64, seed=3)
    scene = engine.Scene(c.dsm, c.trees, c.dem, 1.0, landcover=c.landcover)
    assert scene.svf_steps == rays.svf_rays(2, scene.shape, scene.amaxvalue, 1.0)[2].sum()


@pytest.mark.gpu
def test_a_scene_and_its_days_on_another_stream_are_the_same(cuda):
    """Statics of a scene built on a side stream and days run on one, while the
    current stream is idle and while it is not."""
    import torch
    from solweig_cuda_b200 import engine, synthetic
    c = synthetic.make_scene(150, 131, seed=5)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    busy = torch.zeros(1 << 26, device=cuda)

    def build(stream, work):
        res = {}
        torch.cuda.synchronize()
        for _ in range(work):
            busy.add_(1.0)
        scene = engine.Scene(c.dsm, c.trees, c.dem, 1.0, landcover=c.landcover, stream=stream)
        torch.cuda.synchronize()
        for name in ("walls", "aspect", "masks", "svf32", "gvf_face", "gvf_walks", "gvf_nosh"):
            res[name] = getattr(scene, name).cpu().numpy()
        for runner in (engine.DayRunner, engine.DayRunner64):
            run = runner(scene, 53.0, 0.0, 3.0, 0.0)
            torch.cuda.synchronize()
            for _ in range(work):
                busy.add_(1.0)
            out = run.run_day(met, stream=stream)
            torch.cuda.synchronize()
            res.update({(runner.__name__, k): v.cpu().numpy() for k, v in out.items()})
        return res

    want = build(None, 0)
    side = torch.cuda.Stream()
    for work in (0, 0, 50):
        got = build(side, work)
        for name, v in want.items():
            assert np.array_equal(got[name], v, equal_nan=True), (name, work)
