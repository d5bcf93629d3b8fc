"""The tiled kernels' candidate evaluation (lower bounds over the heaviest
taps first, survivors in lane groups) against the generic kernels, which sum
every candidate in the reference's order: every byte of the results equal."""
import numpy as np
import pytest

from painttween_gb300 import _abi, synthetic

from _harness import FILTER_MODES, assert_array_equal, assert_offsets_equal, config_params

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _inputs(w, h, kind):
    ex = synthetic.make_exemplar(44, 38, seed=w)
    clip = synthetic.make_clip(w, h, 2, 2, seed=h)
    rng = np.random.default_rng(w * h)
    if kind == "culled":  # candidates rejected before their energy: far texels and unpainted ones
        ex["dist_trans"] = rng.uniform(0, 90, ex["dist_trans"].shape).astype(np.float32)
        ex["output"][:, 10:18, 3] = 0.2
    if kind == "flat":  # every patch distance zero: no threshold, all ties
        for a in (ex["base"], ex["output"], *(f["rgba"] for f in clip)):
            a[...] = 0.5
    return ex, clip


@pytest.mark.parametrize("fm", FILTER_MODES)
@pytest.mark.parametrize("r", [2, 3, 4])
@pytest.mark.parametrize("w,h,kind", [(16, 16, "plain"), (31, 19, "flat"), (33, 21, "culled"), (70, 37, "plain"),
                                      (65, 33, "negative")])
def test_candidates_match_generic_kernels(w, h, kind, r, fm):
    from painttween_gb300 import Synthesizer
    p = config_params(r=r, levels=2, iterations=2, filter_mode=fm)
    p.temporalCoherenceWeight, p.hysteresisWeight = 0.5, 0.25
    p.distTransWeight, p.styleObjIdWeight = 0.01, 0.05
    if kind == "negative":  # partial sums may fall: nothing may be rejected early
        p.canvasOutputWeight = -0.5
    ex, clip = _inputs(w, h, kind)
    got = {}
    for name, tiled, lanes in (("generic", 0, 0), ("two lanes a pixel", 1, 1), ("four lanes a pixel", 1, 2)):
        s = Synthesizer(device=0)
        try:
            s.set_tiled_kernels(tiled)
            s.set_propagate_lanes(lanes)
            s.setup(p, w, h, 44, 38, 1)
            s.set_style(0, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
            for i, fr in enumerate(clip):
                s.set_frame_dict(i, fr)
            got[name] = s.synthesize_animation(0, 1)
        finally:
            s.close()
    for name in got:
        for f in (0, 1):
            assert_offsets_equal(got[name][f][1], got["generic"][f][1], 1.0, "%s frame %d" % (name, f))
            assert_array_equal(got[name][f][0], got["generic"][f][0], "%s output frame %d" % (name, f))


@pytest.mark.parametrize("r", [2, 3, 4])
@pytest.mark.parametrize("w,h", [(640, 129), (1030, 270), (512, 512)])
def test_active_tile_lists_change_nothing(w, h, r):
    """Levels with enough tiles for the lists, most of them culled: change
    tracking (which uses the lists) against none."""
    from painttween_gb300 import Synthesizer
    p = config_params(r=r, levels=3, iterations=2)
    p.temporalCoherenceWeight = 0.5
    p.distTransCull = 12
    ex, clip = _inputs(w, h, "plain")
    got = []
    for on in (1, 0):
        s = Synthesizer(device=0)
        try:
            s.set_incremental(on)
            s.setup(p, w, h, 44, 38, 1)
            s.set_style(0, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
            for i, fr in enumerate(clip):
                s.set_frame_dict(i, fr)
            got.append(s.synthesize_animation(0, 1))
            res = [s.get_frame_residual(f) for f in (0, 1)]
            got[-1] = {f: got[-1][f] + (res[f],) for f in (0, 1)}
        finally:
            s.close()
    for f in (0, 1):
        assert_offsets_equal(got[0][f][1], got[1][f][1], 1.0, "frame %d" % f)
        assert_array_equal(got[0][f][0], got[1][f][0], "output frame %d" % f)
        assert_array_equal(got[0][f][2], got[1][f][2], "residual frame %d" % f)
