"""The product against golden outputs of the reference's own kernels (tests/golden): match lists
and denoised planes or stacked accumulators are bit for bit the reference's, for the hard
threshold and the Wiener pass, radius 0 to 2, CBM3D, and the other metrics and transforms."""
import glob
import json
import os

import numpy as np
import pytest

import ref_configs as rc
from gpu_common import run_product

pytestmark = pytest.mark.gpu
FILES = sorted(glob.glob(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "*.npz")))


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f)[:-4] for f in FILES])
def test_product_equals_reference_golden(path):
    z = np.load(path)
    spec = rc.RefSpec(**{k: (tuple(v) if isinstance(v, list) else v) for k, v in json.loads(str(z["spec"])).items()})
    (mine,), lists = run_product(spec, z["src"])
    assert np.array_equal(lists, z["matches"])
    want = z["out"][..., :spec.w]
    for p in range(mine.shape[0]):
        if not spec.chroma or (spec.proc_mask >> p) & 1:
            assert np.array_equal(mine[p], want[p]), f"plane {p}"
