"""The event kernel's first lanes and its queue.

The first lanes are dealt to the warps one by one when one lane is long, the
rest come from the work queue.  The tallies do not depend on it: a grid of one
warp per SM gives the same ones, to the last record, as the full grid with a
thread for every lane, at lane counts around the threads and twice them; and
both agree with the history loop (same draws; its multiply-adds may contract
otherwise, which parts a history in a million)."""
import numpy as np
import pytest

import mcpet
from mcpet import inputs
import scenes

pytestmark = pytest.mark.gpu
THREADS = 32          # a block of one warp, one block per SM


def _lanes(which):
    import torch
    t = THREADS * torch.cuda.get_device_properties(0).multi_processor_count
    return {"1": 1, "31": 31, "33": 33, "T-1": t - 1, "T": t, "T+1": t + 1, "2T-1": 2 * t - 1, "2T": 2 * t,
            "2T+1": 2 * t + 1, "3T+5": 3 * t + 5}[which]


def _scene(workdir, n, hot, **kw):
    """A water block with one lane in each of its first n voxels (about 3
    decays each; the hot one holds most of the run's decays, which spreads
    the first lanes over the warps)."""
    shape = (26, 26, 26)
    mat, rho = np.full(shape, 2, np.int32), np.ones(shape, np.float32)
    act = np.zeros(shape, np.float32)
    act.ravel()[:n] = np.random.default_rng(n).uniform(1, 5, n)
    if hot:
        act.ravel()[n // 2] = 400.0 + n / 16
    return scenes.scene_from_arrays(workdir, mat, rho, act, (0.4, 0.4, 0.4), threads_per_block=1, **kw)


KINDS = {
    "sinogram": dict(),
    "psf": dict(tally_psf_sinogram=0, psf_size=200000),
    "dose": dict(material_dose=True, voxel_dose=True, dose_roi=(1, 26, 1, 26, 1, 26)),
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("hot", [False, True], ids=["even", "hot"])
@pytest.mark.parametrize("lanes", [mcpet.LANES_REFERENCE, mcpet.LANES_BALANCED], ids=["reference", "balanced"])
@pytest.mark.parametrize("count", ["1", "31", "33", "T-1", "T", "T+1", "2T-1", "2T", "2T+1", "3T+5"])
def test_tallies_do_not_depend_on_the_lanes_place(workdir, count, lanes, hot, kind):
    if kind != "sinogram" and count not in ("33", "T+1", "3T+5"):
        pytest.skip("the other tallies at three counts")
    with _scene(workdir, _lanes(count), hot, **KINDS[kind]) as sc:
        o = dict(lane_mode=lanes, histories_per_lane=1 << 20)
        assert sc.lane_plan(lanes, 1 << 20)["total_lanes"] == _lanes(count)
        a = sc.run(mcpet.RunOptions(block_threads=THREADS, blocks_per_sm=1, **o))
        b = sc.run(mcpet.RunOptions(**o))
        c = sc.run(mcpet.RunOptions(algorithm=mcpet.ALGORITHM_HISTORIES, **o))
        assert a.total_histories == b.total_histories == c.total_histories and a.detected == b.detected
        for k in ("trues", "scatter", "image_trues", "image_scatter", "spectrum", "material_dose", "voxel_dose"):
            x, y, z = getattr(a, k), getattr(b, k), getattr(c, k)
            assert (x is None) == (y is None)
            if x is not None:
                np.testing.assert_array_equal(x, y, err_msg=k)
                if not k.endswith("dose"):
                    assert np.abs(x.astype(np.int64) - z).sum() <= 0.001 * x.sum(dtype=np.int64) + 2, k
        if kind == "psf":
            assert a.psf_count == b.psf_count
            np.testing.assert_array_equal(scenes.psf_records(a.psf), scenes.psf_records(b.psf))


@pytest.mark.parametrize("count", ["33", "T+1", "3T+5"])
def test_batch_equals_runs_alone(workdir, count):
    """Two scenes of different lane counts in one launch."""
    o = mcpet.RunOptions(lane_mode=mcpet.LANES_REFERENCE, block_threads=THREADS, blocks_per_sm=1)
    with _scene(workdir, _lanes(count), False, seed=11) as a, _scene(workdir, 40, True, seed=12) as b:
        alone = [s.run(o) for s in (a, b)]
        both = mcpet.Scene.run_batch([a, b], o)
        for x, y in zip(alone, both):
            assert x.total_histories == y.total_histories and x.detected == y.detected
            for k in ("trues", "scatter", "image_trues", "image_scatter", "spectrum"):
                np.testing.assert_array_equal(getattr(x, k), getattr(y, k), err_msg=k)


@pytest.mark.parametrize("batch", [False, True], ids=["one", "batch"])
def test_autotuner_samples_start_like_the_run(workdir, batch):
    """8000 lanes of 50 decays: each 1/8000 of the decays (1/16000 of two
    scenes'), above the line of a spread start (1/16384) in the run and in a
    sample of a fifth of it."""
    shape = (20, 20, 20)
    mat, rho = np.full(shape, 2, np.int32), np.ones(shape, np.float32)
    act = np.full(shape, 50.0, np.float32)
    o = mcpet.RunOptions(lane_mode=mcpet.LANES_REFERENCE)
    sc = [scenes.scene_from_arrays(workdir, mat, rho, act, (0.5, 0.5, 0.5), threads_per_block=1, seed=21 + k)
          for k in range(2 if batch else 1)]
    tal = [mcpet.device_tallies_for(s) for s in sc]
    if batch:
        mcpet.Scene.run_batch_device(sc, tal, o)
    else:
        sc[0].run_device(tal[0], o)
    assert [mcpet.probe_start(s) for s in sc] == [1] * len(sc)
    _, info = mcpet.autotune(sc, tal, o, sample_decays=8.0e4 * len(sc))
    assert abs(info["sample_fraction"] - 0.2) < 1e-6
    assert [mcpet.probe_start(s) for s in sc] == [1] * len(sc)
    for s in sc:
        s.close()
