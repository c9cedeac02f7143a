"""The inpainting passes at the edges of their mask words (32 columns) and row
groups (32 rows), on masks that exercise what they special-case: strips and
groups without holes, holes reaching through several groups and words, and
nearly nothing but holes.  Through rvsb_inpaint_sources_noalloc, against the
scan model that test_inpaint_model.py proves equal to the literal sweeps;
integer sources, exact equality."""
import numpy as np
import pytest

import rvsb
from inpaint_model import inpaint_sources

pytestmark = pytest.mark.gpu


def _masks(h, w, seed):
    rng = np.random.default_rng(seed)
    yield rng.random((h, w)) < 0.1
    yield rng.random((h, w)) < 0.9
    band = np.zeros((h, w), bool)  # borders and a bar across, thicker than a group where the size allows
    band[: h // 2 - 1] = True
    band[:, : w // 3] = True
    band[:, w - w // 4:] = True
    yield band
    one = np.ones((h, w), bool)  # a single source
    one[rng.integers(h), rng.integers(w)] = False
    yield one
    yield np.zeros((h, w), bool)


@pytest.mark.parametrize("w,h", [(2, 2), (30, 34), (32, 32), (34, 30), (64, 66), (66, 96), (130, 98), (1026, 34)])
def test_sources_at_word_and_group_edges(w, h):
    import torch
    for k, hole in enumerate(_masks(h, w, 100 * w + h)):
        src = torch.full((h, w, 2), -7, dtype=torch.int32, device="cuda")
        rvsb.inpaint_sources_noalloc(torch.from_numpy(hole.astype(np.uint8)).cuda(), w, h, src)
        torch.cuda.synchronize()
        got = src.cpu().numpy()
        ys, xs = np.mgrid[0:h, 0:w]
        np.testing.assert_array_equal(got[~hole], np.stack([xs, ys], -1)[~hole])
        np.testing.assert_array_equal(got[hole], np.asarray(inpaint_sources(hole))[hole], err_msg=f"mask {k}")
