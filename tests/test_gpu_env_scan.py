"""The sampler build's scans at the sizes where their split changes: one cell,
a block's 256 cells and one around them, the last size of four cells a thread
(131,072), and the largest map; against the host's table by the same criteria
as the other sampler tests."""
import numpy as np
import pytest

from test_gpu_env_sampler import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (255, 1), (16, 16), (257, 1), (512, 256), (513, 256), (1024, 1024)])
@pytest.mark.parametrize("kind", ["uniform", "peaked"])
def test_scan_sizes(w, h, kind):
    rng = np.random.Generator(np.random.PCG64(w * 7 + h))
    img = rng.uniform(0.1, 2, (h, w, 3)) if kind == "uniform" else np.exp(3 * rng.standard_normal((h, w, 3)))
    _check(img.astype(np.float32), w, h)
