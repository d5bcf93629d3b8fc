"""The random level's scratch: bounded however many draws a level takes, and
none of it needed, so that a memory budget which holds the level's own buffers
suffices.  The stream in windows against the oracle's serial draw and against
a context without a budget."""
import numpy as np
import pytest

from painttween_gb300 import Synthesizer, TexSynth, _abi, synthetic

from _harness import Pair, assert_array_equal, assert_offsets_equal, config_params

pytestmark = pytest.mark.gpu

SCRATCH = 6 << 20


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _bare_exemplar(share, seed=9):
    ex = synthetic.make_exemplar(64, 64, seed=seed)
    rng = np.random.default_rng(seed)
    ex["output"][..., 3] = np.where(rng.uniform(size=(64, 64)) < share, 0.2, 1.0)
    return ex


def _level(t, pair, p):
    """The level's inputs, its random level, and the offsets from it fetched."""
    t.initialize(pair.W, pair.H, pair.EW, pair.EH, 1)
    t.set_params(p)
    t.initialize_exemplars(pair.EW, pair.EH, 1)
    s, fp = pair.sp, pair.fps[0]
    t.upload_image_color4(0, _abi.LAYER_EXEMPLAR_BASE, s["base"][0], 0)
    t.upload_image_color4(0, _abi.LAYER_EXEMPLAR_OUTPUT, s["output"][0], 0)
    t.upload_image_float(0, _abi.LAYER_EXEMPLAR_ORIENTATION, s["orient"][0], 0)
    t.upload_image_float(0, _abi.LAYER_EXEMPLAR_DIST_TRANS, s["dt"][0], 0)
    t.upload_image_int(0, _abi.LAYER_EXEMPLAR_OBJECT_IDS, s["ids"][0], 0)
    t.upload_image_color4(0, _abi.LAYER_INPUT_COLOR, fp["rgba"][0])
    t.upload_image_float(0, _abi.LAYER_INPUT_ORIENTATION, fp["orient"][0])
    t.upload_image_int(0, _abi.LAYER_INPUT_ID, fp["ids"][0])
    t.upload_image_float2(0, _abi.LAYER_INPUT_VEL_B, fp["velb"][0])
    t.upload_image_float2(0, _abi.LAYER_INPUT_VEL_F, fp["velf"][0])
    t.upload_image_float(0, _abi.LAYER_INPUT_DIST_TRANS, fp["dt"][0])
    t.upload_image_float2(0, _abi.LAYER_INPUT_SCALE, fp["scale"][0])
    t.create_random_level(0, 0)
    t.randomize_offsets(0)
    return t.get_offsets(0)


# 1024 x 1024: some 4, 6 and 30 windows of the stream
@pytest.mark.parametrize("w,h,bare", [(1024, 1024, 0.0), (1024, 1024, 0.5), (1024, 1024, 0.93), (128, 128, 0.5)])
def test_scratch_is_bounded_and_not_needed(w, h, bare):
    pair = Pair(w, h, 64, 64, config_params(), style=_bare_exemplar(bare))
    try:
        pair.load_style(0)
        pair.load_frame(0, 0)
        pair.random_level(0, 0)
        pair.both("randomize_offsets", 0)
        pair.compare(0, "random level", residual=False)
        want = pair.g.get_offsets(0)
        # the same calls with the counter generator, which draws without the stream
        counter = pair.p.copy()
        counter.rngMode = _abi.RNG_COUNTER
        t = TexSynth(device=0)
        try:
            _level(t, pair, counter)
            own = t.device_bytes
        finally:
            t.close()
        free = TexSynth(device=0)
        try:
            _level(free, pair, pair.p)
            assert free.device_bytes <= own + SCRATCH
        finally:
            free.close()
        # none of it, a small window's, and a quarter of the largest
        for extra in (0, 64 << 10, 2 << 20) if w * h < 1 << 18 or bare == 0.0 else (64 << 10, 2 << 20):
            t = TexSynth(device=0, hbm_budget=own + extra)
            try:
                assert_offsets_equal(_level(t, pair, pair.p), want, 1.0, "%d bytes to spare" % extra)
            finally:
                t.close()
    finally:
        pair.close()


def _keyed(w, h, budget):
    p = config_params(r=2, levels=2, iterations=1)
    p.interpolateKeyFrame, p.numStyles = 1, 2
    s = Synthesizer(device=0, hbm_budget=budget)
    try:
        s.setup(p, w, h, w, h, 2)
        for i in range(2):
            ex = synthetic.make_exemplar(w, h, seed=3 + i)
            ex["output"][:, 10:60, 3] = 0.2
            s.set_style(i, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
        for i, fr in enumerate(synthetic.make_clip(w, h, 2, 3, seed=5)):
            s.set_frame_dict(i, fr)
        s.set_keyframes([0, 2])
        return s.synthesize_animation(0, 2), s.device_bytes
    finally:
        s.close()


def test_keyed_clip_under_a_budget():
    """A budget short by most of the scratch: smaller windows, the same frames."""
    got, held = _keyed(128, 96, 0)
    tight, _ = _keyed(128, 96, held - (200 << 10))
    for f in got:
        assert_offsets_equal(tight[f][1], got[f][1], 1.0, "frame %d" % f)
        assert_array_equal(tight[f][0], got[f][0], "output frame %d" % f)
