"""The lists of active tiles are a help, not a need: a clip runs within a
memory budget that holds all its buffers but them."""
import pytest

from painttween_gb300 import PaintTweenError, Synthesizer, synthetic

from _harness import assert_array_equal, assert_offsets_equal, config_params

pytestmark = pytest.mark.gpu

W, H, R = 1030, 270, 2  # above the line from which a level has lists (1024 pixels an SM)
LISTS = 4 * 18432       # three lists and the marks: 33 x 135 tiles of 32 x 2 pixels, 4 bytes each
STEP = LISTS // 8


def _clip(budget, tracked):
    """The clip's frames and the memory held, or None where the budget does not suffice."""
    p = config_params(r=R, levels=2, iterations=1)
    ex = synthetic.make_exemplar(44, 38, seed=4)
    s = Synthesizer(device=0, hbm_budget=budget)
    try:
        s.set_incremental(tracked)
        s.setup(p, W, H, 44, 38, 1)
        s.set_style(0, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
        for i, fr in enumerate(synthetic.make_clip(W, H, 2, 2, seed=6)):
            s.set_frame_dict(i, fr)
        return s.synthesize_animation(0, 1), s.device_bytes
    except PaintTweenError as e:
        assert e.status == 7  # PT_ERR_BUDGET
        return None
    finally:
        s.close()


def _size_class(n):
    """An allocation of n bytes as the context rounds it: to eighths of a power of two."""
    step = (1 << (n.bit_length() - 1)) // 8
    return -(-n // step) * step


def test_clip_without_memory_for_tile_lists(gpu_lib):
    got, held = _clip(0, 1)
    # the least that the clip needs without change tracking, and with it the planes of tap values
    low, high = held // 2, held
    while high - low > STEP:
        mid = (low + high) // 2
        if _clip(mid, 0):
            high = mid
        else:
            low = mid
    need = high + _size_class((2 * R + 1) ** 2 * W * H * 4)
    for budget in (need, need + LISTS // 2):  # room for none of the lists, for some
        tight = _clip(budget, 1)
        assert tight is not None
        for f in got:
            assert_offsets_equal(tight[0][f][1], got[f][1], 1.0, "frame %d" % f)
            assert_array_equal(tight[0][f][0], got[f][0], "output frame %d" % f)
