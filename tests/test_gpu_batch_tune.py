"""A tuned batch is no slower than an untuned one: the launches' own choice of
rows per work item is among the tiles that tops_batch_autotune times."""
import pytest

pytestmark = pytest.mark.gpu


def test_tuned_batch_is_no_slower(T):
    import torch
    scenes = [T.Scene(n_bursts=2, lines_per_burst=300, samples_per_burst=w, overlap_lines=30,
                      dem_lines=160, dem_pixels=160, seed=w) for w in (512, 640)]
    plans = []
    for S in scenes:
        P = T.Pair(S.swath[0], S.swath[1], S.dem.shape)
        di = S.dem_info
        P.set_dem(S.dem, di.lat0, di.lon0, di.dlat, di.dlon, T.scene_windows(S))
        P.upload(S.slc[0], S.slc[1])
        plans.append(P)
    B = T.Batch(plans)
    s = torch.cuda.current_stream().cuda_stream

    def time_run():
        t = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                B.run(s, graph=True)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        return sorted(t)[len(t) // 2]

    time_run()
    untuned = time_run()
    B.autotune(s)
    tuned = time_run()
    B.close()
    for P in plans:
        P.close()
    print(f"untuned {untuned * 250:.0f} us, tuned {tuned * 250:.0f} us")
    # of a few equal tiles the fastest by two runs: within their noise
    assert tuned < 1.25 * untuned, (untuned, tuned)
