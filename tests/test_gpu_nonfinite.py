"""Activations that are not finite: an overflow upstream stays visible in the product, however many rows it has and
whichever kernel takes them, and only in its own row."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty", helpers.FORMATS)
@pytest.mark.parametrize("half", [True, False])
def test_rows_that_are_not_finite(ty, half):
    helpers.build_library()
    import torch
    import lazyweights_b200 as lw
    n, k = 128, 1024
    q, side, sym, w, rng = helpers.seeded_case(ty, n, k, seed=11)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    with lw.CodedMatrix(blob, n, sym.shape[1], ty, side) as mat:
        for m in (1, 2, 8, 20, 80):   # one row, fused rows, tensor-core rows, decoded weights
            for columns, value in ((slice(0, k), np.nan), (slice(96, 128), np.nan), (100, np.inf), (slice(0, k), -np.inf)):
                x = rng.standard_normal((m, k)).astype(np.float32)
                x[m // 2, columns] = value
                xt = torch.from_numpy(x).cuda()
                y = mat.linear("m", xt.half() if half else xt).cpu().numpy()
                assert not np.isfinite(y[m // 2]).any(), (m, value)
                assert np.isfinite(np.delete(y, m // 2, 0)).all(), (m, value)
    assert lw.lib().lw_kernel_error() == 0
