"""PLS-LDA prediction of more rows than 32-bit offsets reach: the rows to predict
have no limit of their own, and rows x 8 padded columns passes 2^31 floats here.
The rows repeat a small set, so the predictions repeat the small set's, which the
CPU restatement gives."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = (1 << 28) + 4099


def test_prediction_past_32_bit_offsets(kg, orc):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[1] < 64 << 30:
        pytest.skip("needs 20 GB of device memory")
    rng = np.random.default_rng(8)
    lab = rng.integers(1, 4, 400).astype(np.int32)
    x = (rng.standard_normal((400, 1)) + 1.5 * lab[:, None]).astype(np.float32)
    few = (rng.standard_normal((1009, 1)) * 2 + 3).astype(np.float32)
    kw = dict(max_components=1, fixed_components=1)
    want = orc.plsldapredict(x, lab, few, components=1)
    assert len(np.unique(want)) == 3
    assert np.array_equal(kg.PLSLDAPredict(x, lab, few, **kw), want)
    times = -(-ROWS // len(few))
    got = kg.PLSLDAPredict(x, lab, np.tile(few, (times, 1))[:ROWS], **kw)
    assert np.array_equal(got, np.tile(want, times)[:ROWS])
