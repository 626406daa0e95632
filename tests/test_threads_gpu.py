"""Days of several threads at once, each with walks, hours and a stream of its own: a
kernel's shared-memory limit, one for all threads, fits every one of them."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_days_of_different_shapes_in_threads(cuda):
    import torch
    from solweig_cuda_b200 import batched, engine, synthetic
    cases = []
    for pixel, hours in ((1.0, 24), (2.0, 6), (4.0, 3), (0.5, 24), (0.6, 12)):
        s = synthetic.make_scene(40, 45, seed=3, pixel_size=pixel)
        scene = engine.Scene(s.dsm, s.trees, s.dem, pixel, landcover=s.landcover)
        met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=2)[24 - hours:]
        day = batched.ChosenDay(scene, 53.0, 0.0, 3.0, 0.0, hours=hours, use_graph=False)
        want = {k: v.clone() for k, v in day.run_day(met).items()}
        cases.append((day, want))
    torch.cuda.synchronize()
    failed = []

    def run(day, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20000):
                    day._sequence()
                torch.cuda.current_stream().synchronize()
                for k, v in want.items():
                    if not torch.equal(day.out[k].view(torch.int32), v.view(torch.int32)):
                        failed.append(k)
        except RuntimeError as e:
            failed.append(str(e))

    threads = [threading.Thread(target=run, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:3]
