"""The random level drawn in parallel segments of glibc's stream against the
oracle's serial draw: whole levels without retries, retries from few to all
pixels (past what the drawn stream suffices for), partly transparent images."""
import numpy as np
import pytest

from painttween_gb300 import synthetic

from _harness import Pair, config_params

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    return gpu_lib


# a segment has 496 draws, 124 pixels without retries; 31 x 4 is one exactly
@pytest.mark.parametrize("w,h", [(2, 2), (31, 4), (25, 5), (97, 61), (200, 128)])
@pytest.mark.parametrize("bare", [0.0, 0.02, 0.5, 1.0])
def test_random_level_matches_serial_draw(w, h, bare):
    rng = np.random.default_rng(w + h)
    ex = synthetic.make_exemplar(40, 36, seed=9)
    clip = [synthetic.make_still(w, h, 2, seed=w)]
    if bare:
        ex["output"][..., 3] = np.where(rng.uniform(size=(36, 40)) < bare, 0.2, 1.0)
        clip[0]["rgba"][..., 3] = np.where(rng.uniform(size=(h, w)) < 0.3, 0.5, 1.0)
    pair = Pair(w, h, 40, 36, config_params(), style=ex, clip=clip)
    try:
        pair.load_style(0)
        pair.load_frame(0, 0)
        pair.random_level(0, 0)
        pair.both("randomize_offsets", 0)
        pair.compare(0, "random level", residual=False)
    finally:
        pair.close()


def test_random_level_seeds():
    pair = Pair(96, 80, 64, 64, config_params())
    try:
        for level, frame in ((1, 1), (1, 5), (2, 7)):
            pair.load_style(level)
            pair.load_frame(0, level)
            from oracle import oracle as O
            fp = pair.fps[0]
            rnd = O.random_level(frame * level, level, 64, 64, fp["rgba"][level], fp["orient"][level],
                                 pair.sp["output"][level], pair.sp["orient"][level], False, True)
            pair.o.upload_random(rnd)
            pair.g.create_random_level(level, frame)
            pair.both("randomize_offsets", level)
            pair.compare(level, "level %d frame %d" % (level, frame), residual=False)
    finally:
        pair.close()
