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


def _model(tmp_path, heads, kv_heads, head_dim):
    from lazyweights_b200 import modelgen
    shape = dict(n_layers=1, hidden=512, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, inter=512, vocab=256, eps=1e-5, theta=1e4)
    modelgen.write_model(str(tmp_path / "m"), shape, "Q6_K", seed=heads + kv_heads)
    return str(tmp_path / "m")


# up to 18 chunks; spans of one, two and four chunks, tiles of 8, 16 and 32 rows, several tiles per kv head
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 32, 64), (32, 8, 128), (48, 16, 64), (8, 8, 96), (2, 2, 128)])
def test_tiles_and_single_tokens_agree_bit_for_bit(tmp_path, heads, kv_heads, head_dim):
    """A query's attention is the same whatever kernel serves it: a whole run of passes through the tiled kernel and
    one through the kernel with a block per token, over the same products, give the same logits to the last bit."""
    helpers.build_library()
    import lazyweights_b200 as lw
    path = _model(tmp_path, heads, kv_heads, head_dim)
    ids = np.random.default_rng(4).integers(0, 256, 1150).astype(np.int32)
    sizes = [64, 64, 37, 8, 8, 8, 3, 2, 1, 5, 64, 64, 64, 64, 64, 64, 64, 64, 64, 64, 64, 7, 7, 64, 8, 8, 2, 2, 64, 5, 3, 60]
    runs = []
    try:
        for tiled in (1, 0):
            assert lw.lib().lw_debug_set(b"attn_rows", tiled) == 0
            with lw.Bundle(path, max_ctx=2048, max_batch=64) as b:   # a handle each: captured passes keep their kernels
                pos, out = 0, []
                for m in sizes:
                    out.append(np.atleast_2d(b.forward(ids[pos:pos + m], all_logits=True)))
                    pos += m
                runs.append(np.concatenate(out))
    finally:
        lw.lib().lw_debug_set(b"reset", 0)
    assert np.isfinite(runs[0]).all()
    assert np.array_equal(runs[0], runs[1])
    assert lw.lib().lw_kernel_error() == 0


def test_tokens_of_a_pass_do_not_change_a_query(tmp_path):
    """Passes of two to eight tokens: the products of these row counts are the same arithmetic per row, and attention does
    not depend on the other tokens of the pass, so neither do the logits.  Eight query heads per kv head: the pass of eight
    tokens has two tiles of rows, the others one, with other spans of chunks from 640 positions on."""
    helpers.build_library()
    import lazyweights_b200 as lw
    ids = np.random.default_rng(5).integers(0, 256, 840).astype(np.int32)
    with lw.Bundle(_model(tmp_path, 128, 16, 32), max_ctx=1024, max_batch=8) as b:
        runs = []
        for m in (2, 3, 5, 8):
            b.reset()
            runs.append(np.concatenate([b.forward(ids[i:i + m], all_logits=True) for i in range(0, 840, m)]))
        for got in runs[1:]:
            assert np.array_equal(got, runs[0])
        assert b.kernel_error() == 0


@pytest.mark.parametrize("window", [1, 50, 64, 100, 130])
def test_sliding_window(tmp_path, window):
    """Passes of several tokens under a sliding window against single tokens under the same window: while the window is not
    full, across the pass in which it becomes full, and after; every position of the pass has its own first position."""
    helpers.build_library()
    import lazyweights_b200 as lw
    n = 280
    ids = np.random.default_rng(6).integers(0, 256, n).astype(np.int32)
    with lw.Bundle(_model(tmp_path, 8, 2, 128), max_ctx=512, max_batch=8) as b:
        b.set_window(window)
        step = np.stack([b.forward(ids[i:i + 1]) for i in range(n)])
        for m in (2, 3, 8, 8):               # the second time the passes of eight are captured and replayed
            b.reset()
            got = np.concatenate([np.atleast_2d(b.forward(ids[i:i + m], all_logits=True)) for i in range(0, n, m)])
            assert np.isfinite(got).all()
            # one layer: the keys and values of both runs come from products within helpers.GEMV_TOL of each other
            for i in range(n):
                assert helpers.rel_err(got[i], step[i]) <= helpers.GEMV_TOL, (m, i)
        b.set_pos(n - 1)
        cut = b.forward(ids[n - 1:n])
        b.set_window(0)
        b.set_pos(n - 1)
        assert not np.array_equal(b.forward(ids[n - 1:n]), cut)
        assert b.kernel_error() == 0
