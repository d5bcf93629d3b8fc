"""The one-launch separable Gaussian against the oracle's two passes, at the
edges of its 64 x 32 tiles, with a pitch, and in place (two launches)."""
import numpy as np
import pytest

from oracle import oracle as O

from _harness import assert_array_equal

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    return gpu_lib


@pytest.mark.parametrize("inplace", [False, True])
@pytest.mark.parametrize("w,h,pad,radius", [(1, 1, 0, 15), (63, 31, 3, 1), (64, 32, 0, 15), (65, 33, 64, 7),
                                            (200, 97, 1, 4), (7, 130, 0, 12)])
def test_blur_matches_oracle(w, h, pad, radius, inplace):
    torch = pytest.importorskip("torch")
    from painttween_gb300 import TexSynth
    img = np.random.default_rng(w * h + radius).uniform(-2, 5, (h, w)).astype(np.float32)
    ref = O.convolve_separable(img, radius)
    src = torch.full((h, w + pad), 77.0, device="cuda")
    src[:, :w] = torch.from_numpy(img).cuda()
    dst = src if inplace else torch.full_like(src, 55.0)
    torch.cuda.synchronize()
    t = TexSynth(device=0)
    t.convolve_separable(src.data_ptr(), dst.data_ptr(), w, h, w + pad, radius)
    t.synchronize()
    t.close()
    got = dst.cpu().numpy()
    assert_array_equal(got[:, :w], ref, "blur %dx%d r=%d" % (w, h, radius))
    assert (got[:, w:] == (77.0 if inplace else 55.0)).all()
