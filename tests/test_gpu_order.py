"""The depth order of the depth-of-field blur with NaN depths (pixels without
a hit): csrc/stable_order.cu against the oracle, which runs std::stable_sort."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from raym0nade_gb300 import api  # noqa: E402
from tests.golden.make_golden import PHOTO_POST, photo_records  # noqa: E402
from tests.test_gpu_post import np_, photo_from_records  # noqa: E402


# sizes about a chunk of 7, a half of one tile of 1792 and several merge
# levels, odd (the last merge from the back) and even
@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (3, 1), (7, 1), (5, 3), (64, 56), (61, 59), (128, 61), (97, 151)])
@pytest.mark.parametrize("nan", ["some", "top", "bottom", "bands", "all"])
def test_nan_depth_order(port, w, h, nan):
    rec = photo_records(w, h, 31 + w)
    r = rec.reshape(-1, 40)
    n = w * h
    i = np.arange(n)
    miss = {"some": np.random.default_rng(w).random(n) < 0.3, "top": i < 0.4 * n, "bottom": i >= 0.6 * n,
            "bands": (i // 13) % 3 == 0, "all": i >= 0}[nan]
    r[:, 22:25] = np.round(r[:, 22:25] * 8) / 8  # ties
    r[miss, 22:25] = np.nan
    post = dict(PHOTO_POST, coc=9.0)
    ph = photo_from_records(rec, post)
    got = np_(ph.post_process(api.Full | api.DoDepthFieldBlur))
    _, want = port.photo(rec, 8, api.Full | api.DoDepthFieldBlur, **post)
    assert np.array_equal(got, want, equal_nan=True)


def test_a_pixel_without_a_hit_is_reached_when_full(port):
    """A pixel without a hit gets its own NaN colour, however much weight its
    neighbours have given it before its turn in the order: beside a near wall,
    blurred wide, the far one's pixels receive more than the 0.99 they take."""
    w, h = 96, 80
    rec = photo_records(w, h, 3)
    r = rec.reshape(-1, 40)
    rng = np.random.default_rng(1)
    x = np.arange(w * h) % w
    r[:, 22:24] = 0.0
    r[:, 24] = np.where(x < w // 2, 0.3, 2.0) + 1e-3 * rng.random(w * h)
    miss = (np.abs(x - w // 2 - 4) < 8) & (rng.random(w * h) < 0.04)
    r[miss, 22:25] = np.nan
    post = dict(PHOTO_POST, coc=10.0)
    ph = photo_from_records(rec, post)
    got = np_(ph.post_process(api.Full | api.DoDepthFieldBlur))
    _, want = port.photo(rec, 8, api.Full | api.DoDepthFieldBlur, **post)
    assert np.isnan(want).any(-1).sum() == miss.sum()
    assert np.array_equal(got, want, equal_nan=True)
