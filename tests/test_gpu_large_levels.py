"""The kernel shapes of large levels, which small tests do not reach: scatter
with two lanes a pixel (above 2048 pixels an SM), the residual with one lane a
pixel (exact filter: two) and the lists of active tiles (above 1024), for each
radius, filter and temporal direction, against the generic kernels; and
without change tracking, where every residual is computed in full.  Every byte
equal: all of them form each patch distance by the same operations."""
import numpy as np
import pytest

from painttween_gb300 import Synthesizer, synthetic

from _harness import FILTER_MODES, assert_array_equal, assert_offsets_equal, config_params

pytestmark = pytest.mark.gpu

SCATTER_LIMIT, RESIDUAL_LIMIT = 2048, 1024  # pixels an SM, above which the level takes the large shapes


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _inputs(w, h):
    """Odd-sized tiles at the edges, idle ones inside (far from the discs),
    candidates that are rejected before their distance."""
    ex = synthetic.make_exemplar(61, 47, seed=w)
    ex["dist_trans"] = np.random.default_rng(h).uniform(0, 60, ex["dist_trans"].shape).astype(np.float32)
    ex["output"][:, 20:24, 3] = 0.2
    return ex, synthetic.make_clip(w, h, 3, 2, seed=h)


def _clip(p, w, h, ex, clip, tiled, tracked):
    s = Synthesizer(device=0)
    try:
        s.set_tiled_kernels(tiled)
        s.set_incremental(tracked)
        s.setup(p, w, h, 61, 47, 1)
        s.set_style(0, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
        for i, fr in enumerate(clip):
            s.set_frame_dict(i, fr)
        got = s.synthesize_animation(0, 1)
        return {f: got[f] + (s.get_frame_residual(f),) for f in got}
    finally:
        s.close()


@pytest.mark.parametrize("fm", FILTER_MODES)
@pytest.mark.parametrize("r", [2, 3, 4])
@pytest.mark.parametrize("w,h,limit", [(157, 1003, RESIDUAL_LIMIT), (643, 491, SCATTER_LIMIT)])
def test_large_shapes_match_generic_kernels(w, h, limit, r, fm):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert w * h > limit * sms, "not a large level on this device"
    p = config_params(r=r, levels=2, iterations=2, filter_mode=fm)
    p.temporalCoherenceWeight, p.hysteresisWeight = 0.5, 0.25
    p.distTransWeight, p.styleObjIdWeight = 0.01, 0.05
    p.distTransCull = 40
    ex, clip = _inputs(w, h)
    want = _clip(p, w, h, ex, clip, 0, 0)
    for name, tracked in (("tracked", 1), ("untracked", 0)):
        got = _clip(p, w, h, ex, clip, 1, tracked)
        for f in want:
            assert_offsets_equal(got[f][1], want[f][1], 1.0, "%s frame %d" % (name, f))
            assert_array_equal(got[f][0], want[f][0], "%s output frame %d" % (name, f))
            assert_array_equal(got[f][2], want[f][2], "%s residual frame %d" % (name, f))


@pytest.mark.parametrize("fm", FILTER_MODES)
@pytest.mark.parametrize("r", [2, 4])
def test_large_still_matches_generic_kernels(r, fm):
    """Without temporal terms."""
    w, h = 643, 491
    p = config_params(r=r, levels=2, iterations=2, filter_mode=fm)
    ex, clip = _inputs(w, h)
    got = {}
    for tiled in (0, 1):
        s = Synthesizer(device=0)
        try:
            s.set_tiled_kernels(tiled)
            s.setup(p, w, h, 61, 47, 1)
            s.set_style(0, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
            s.set_frame_dict(0, clip[0])
            got[tiled] = s.synthesize_frame(0) + (s.get_frame_residual(0),)
        finally:
            s.close()
    assert_offsets_equal(got[1][1], got[0][1])
    assert_array_equal(got[1][0], got[0][0], "output")
    assert_array_equal(got[1][2], got[0][2], "residual")
