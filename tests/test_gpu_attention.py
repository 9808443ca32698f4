"""Attention of passes of several tokens against the one-token kernel, over the same cached keys and values."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


# query heads per kv head: 1, 2, 3, 4 and 8, i.e. tiles of 8, 16 and 32 query rows, whole and ragged
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(4, 4, 128), (4, 2, 128), (12, 4, 128), (8, 2, 64), (8, 1, 128), (16, 16, 96)])
def test_tiles_of_query_rows(tmp_path, heads, kv_heads, head_dim):
    helpers.build_library()
    import lazyweights_b200 as lw
    from lazyweights_b200 import modelgen
    shape = dict(n_layers=1, hidden=512, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, inter=512, vocab=256, eps=1e-5, theta=1e4)
    modelgen.write_model(str(tmp_path / "m"), shape, "Q6_K", seed=heads)
    n = 140                                                    # passes end on both sides of the 64-position chunks
    ids = np.random.default_rng(2).integers(0, shape["vocab"], n).astype(np.int32)
    with lw.Bundle(str(tmp_path / "m"), max_ctx=256, max_batch=8) as b:
        step = np.stack([b.forward(ids[i:i + 1]) for i in range(n)])
        for m in (2, 3, 5, 8):
            b.reset()
            got = np.concatenate([b.forward(ids[i:i + m], all_logits=True) for i in range(0, n, m)])
            # one layer: the keys and values of both runs come from products within helpers.GEMV_TOL of each other
            for i in range(n):
                assert helpers.rel_err(got[i], step[i]) <= helpers.GEMV_TOL, (m, i)
        b.set_pos(63)                                          # a pass over the chunk boundary, from a rewound cache
        assert helpers.rel_err(b.forward(ids[63:66], all_logits=True), step[63:66]) <= helpers.GEMV_TOL
        assert b.kernel_error() == 0
