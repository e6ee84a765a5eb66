"""The event kernel's first lanes and its queue.

Where one lane is long against the launch (more than 1/16384 of its decays) the
first lanes are dealt to the warps one by one, longest first, and the rest come
from the work queue; elsewhere the queue deals every lane.  The tallies do not
depend on it: a grid of one warp per SM gives the same ones, to the last
record, as the full grid, at lane counts around the threads of the small grid
and above those of any grid; a scene that starts spread alone gives the same
ones packed in a batch; and all agree with the history loop (same draws; its
multiply-adds may contract otherwise, which parts a history in a million).
Each test states which start its scene takes and checks it."""
import numpy as np
import pytest

import mcpet
from mcpet import inputs
import scenes

pytestmark = pytest.mark.gpu
THREADS = 32          # a block of one warp, one block per SM
SPREAD, PACKED = 1, 0


def _lanes(which):
    import torch
    t = THREADS * torch.cuda.get_device_properties(0).multi_processor_count
    return {"1": 1, "31": 31, "33": 33, "T-1": t - 1, "T": t, "T+1": t + 1, "3T+5": 3 * t + 5,
            "26^3": 26 ** 3,            # just below the line when all lanes are alike
            "68^3": 68 ** 3}[which]     # more than 2048 threads on each of 148 SMs


def _scene(workdir, n, activity, **kw):
    """A water cube with one lane in each of its first n voxels, about 3
    decays each.  alike: the same in all; uneven: 1 to 5; hot: uneven, and one
    voxel among them with 400."""
    side = 26 if n <= 26 ** 3 else 68
    shape = (side,) * 3
    mat, rho = np.full(shape, 2, np.int32), np.ones(shape, np.float32)
    act = np.zeros(shape, np.float32)
    act.ravel()[:n] = 3.0 if activity == "alike" else np.random.default_rng(n).uniform(1, 5, n)
    if activity == "hot":
        act.ravel()[n // 2] = 400.0
    if kw.get("voxel_dose"):
        kw["dose_roi"] = (1, side) * 3
    return scenes.scene_from_arrays(workdir, mat, rho, act, (10.4 / side,) * 3, threads_per_block=1, **kw)


KINDS = {
    "sinogram": dict(),
    "psf": dict(tally_psf_sinogram=0, psf_size=1000000),
    "dose": dict(material_dose=True, voxel_dose=True),
}
# lanes, activity, start: fewer than 16384 lanes spread whatever their activity
CASES = [(c, "uneven", SPREAD) for c in ("1", "31", "33", "T-1", "T", "T+1", "3T+5")]
CASES += [(c, "hot", SPREAD) for c in ("33", "T", "3T+5", "68^3")]
CASES += [("26^3", "alike", PACKED), ("68^3", "alike", PACKED)]
RUNS = [("sinogram",) + c for c in CASES]
RUNS += [(k,) + c for k in ("psf", "dose") for c in CASES if c[0] in ("T+1", "68^3") or c[2] == PACKED]


@pytest.mark.parametrize("lanes", [mcpet.LANES_REFERENCE, mcpet.LANES_BALANCED], ids=["reference", "balanced"])
@pytest.mark.parametrize("kind, count, activity, start", RUNS, ids=["-".join(r[:3]) for r in RUNS])
def test_tallies_do_not_depend_on_the_lanes_place(workdir, kind, count, activity, start, lanes):
    with _scene(workdir, _lanes(count), activity, **KINDS[kind]) as sc:
        o = dict(lane_mode=lanes, histories_per_lane=1 << 20)
        assert sc.lane_plan(lanes, 1 << 20)["total_lanes"] == _lanes(count)
        a = sc.run(mcpet.RunOptions(block_threads=THREADS, blocks_per_sm=1, **o))
        assert mcpet.probe_start(sc) == start
        b = sc.run(mcpet.RunOptions(**o))
        assert mcpet.probe_start(sc) == start
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


@pytest.mark.parametrize("lanes", [mcpet.LANES_REFERENCE, mcpet.LANES_BALANCED], ids=["reference", "balanced"])
@pytest.mark.parametrize("first, second, starts", [
    (("33", "uneven"), ("33", "hot"), (SPREAD, SPREAD, SPREAD)),
    (("T+1", "uneven"), ("33", "hot"), (SPREAD, SPREAD, SPREAD)),
    (("33", "uneven"), ("68^3", "alike"), (SPREAD, PACKED, PACKED)),
    (("T+1", "uneven"), ("68^3", "alike"), (SPREAD, PACKED, PACKED)),
    (("T", "hot"), ("68^3", "hot"), (SPREAD, SPREAD, SPREAD)),
], ids=lambda v: "-".join(map(str, v)))
def test_batch_equals_runs_alone(workdir, first, second, starts, lanes):
    """Two scenes in one launch, which starts as its lanes together ask for:
    a scene that spreads alone is packed beside many lanes."""
    o = mcpet.RunOptions(lane_mode=lanes, histories_per_lane=1 << 20)
    with _scene(workdir, _lanes(first[0]), first[1], seed=11) as a, \
            _scene(workdir, _lanes(second[0]), second[1], seed=12) as b:
        alone = [s.run(o) for s in (a, b)]
        assert (mcpet.probe_start(a), mcpet.probe_start(b)) == starts[:2]
        both = mcpet.Scene.run_batch([a, b], o)
        assert mcpet.probe_start(a) == mcpet.probe_start(b) == starts[2]
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
