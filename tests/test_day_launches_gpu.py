"""Kernels of a batched day against ``day_launches``, by the nodes of its graph."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relief", [False, True])
@pytest.mark.parametrize("statics", [False, True])
def test_launches_of_a_day(cuda, relief, statics):
    import numpy as np
    import torch
    from solweig_cuda_b200 import _lib, batched, engine, synthetic
    rt = pytest.importorskip("cuda.bindings.runtime")
    s = synthetic.make_scene(48, 70, seed=3)
    up = np.float32(1.1) if relief else np.float32(0)  # heights that float32 does not hold exactly
    scene = engine.Scene(s.dsm + up, s.trees, s.dem + up, 1.0, landcover=s.landcover)
    assert (scene.geo32 is None) == relief
    if not statics:
        scene.struct.gvf_nosh = None
    day = batched.ChosenDay(scene, 53.0, 0.0, 3.0, 0.0)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=2)
    want = {k: v.clone() for k, v in day.run_day(met).items()}
    for no_ceiling in (0, 1):
        for window in (0, 1, 2):
            for hours in (0, 1):
                cfg = _lib.SolweigDayConfig.default()
                cfg.no_ceiling, cfg.sweep_window, cfg.gvf_hours = no_ceiling, window, hours
                day.set_config(cfg)
                torch.cuda.synchronize()
                g = torch.cuda.CUDAGraph(keep_graph=True)
                with torch.cuda.graph(g):
                    day._sequence()
                err, _, n = rt.cudaGraphGetNodes(rt.cudaGraph_t(g.raw_cuda_graph()))
                assert int(err) == 0
                err, nodes, n = rt.cudaGraphGetNodes(rt.cudaGraph_t(g.raw_cuda_graph()), n)
                kinds = [rt.cudaGraphNodeGetType(node)[1] for node in nodes]
                kernels = sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)
                assert kernels == day.launches_per_day, (no_ceiling, window, hours)
                g.instantiate()
                g.replay()
                torch.cuda.synchronize()
                if hours:
                    for k, v in want.items():
                        assert torch.equal(day.out[k].view(torch.int32), v.view(torch.int32)), (no_ceiling, window, k)
