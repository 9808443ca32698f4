"""Products of several rows at the sizes where their kernels can go wrong: edges of the token tiles, row counts that are
no multiple of the weight tiles, K that splits or does not, activations that need a range factor."""
import numpy as np
import pytest

from oracle import lw_oracle as orc
from tests import helpers

pytestmark = pytest.mark.gpu
# fp16 weights and activations: each factor of a term is off by at most 2^-11 of itself, so a sum of products of
# independent signs is off by about 2^-11 sqrt(2) of its own size; 1e-3 of the largest result is the bar of every product.
TOL = helpers.GEMV_TOL


@pytest.fixture(scope="module")
def lw():
    helpers.build_library()
    import torch
    assert torch.cuda.is_available()
    import lazyweights_b200 as pkg
    yield pkg
    assert pkg.lib().lw_kernel_error() == 0


# N 64: half a weight tile; 192: one and a half; 320: two and a half; K 256: four slabs, no split; 14336: many
@pytest.mark.parametrize("ty,n,k,rows", [("Q6_K", 64, 256, (65, 128)), ("Q4_K", 192, 512, (65, 80, 255, 256, 257)),
                                         ("Q5_K", 320, 768, (17, 127, 129, 511, 512, 513)), ("IQ4_XS", 128, 14336, (66, 200)),
                                         ("Q4_K", 4096, 2048, (300,))])
@pytest.mark.parametrize("half", [True, False])
def test_decode_and_gemm(lw, ty, n, k, rows, half):
    import torch
    q, side, sym, w, rng = helpers.seeded_case(ty, n, k, seed=n + k)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    with lw.CodedMatrix(blob, n, sym.shape[1], ty, side) as mat:
        for m in rows:
            x = rng.standard_normal((m, k)).astype(np.float16 if half else np.float32)
            if not half:
                x[m // 2] *= 1e6   # beyond fp16: this row is scaled by a power of two on the way in and back on the way out
            y = torch.full((m + 1, n), -7.0, device="cuda")
            mat.linear("m", torch.from_numpy(x).cuda(), out=y[:m])
            y = y.cpu().numpy()
            assert (y[m] == -7.0).all()
            ref = orc.gemv_f64(w, x.astype(np.float32))
            for r in (0, m // 2, m - 1):
                assert helpers.rel_err(y[r], ref[r]) <= TOL, (m, r)
            rest = [r for r in range(m) if r != m // 2]
            assert helpers.rel_err(y[rest], ref[rest]) <= TOL, m
            if not half:   # 4-byte aligned activations
                z = torch.empty(m * k + 1, device="cuda")
                z[1:] = torch.from_numpy(x).cuda().reshape(-1)
                assert torch.equal(mat.linear("m", z[1:].reshape(m, k)), torch.from_numpy(y[:m]).cuda())


# Q5_K pair layouts: narrow codes get a 10-bit pair code (groups of four), codes all over the range an 11-bit one
@pytest.mark.parametrize("n,k,wide", [(64, 512, False), (192, 1536, False), (256, 2048, True)])
def test_q5k_pair_code_lengths(lw, n, k, wide):
    import torch
    q, side, sym, w, rng = helpers.seeded_case("Q5_K", n, k, seed=n * 3 + k)
    if wide:
        q[:16] = rng.integers(0, 32, (16, k), dtype=np.uint8)   # nearly every pair occurs: ten bits would be a fixed width
        sym, w = orc.symbols_of("Q5_K", q), orc.dequant("Q5_K", q, side)
    assert lw.bundle.host_pairs(q, "Q5_K", side)["index_bits"] == (11 if wide else 10)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    with lw.CodedMatrix(blob, n, k, "Q5_K", side) as mat:
        assert np.array_equal(mat.decode_codes("m").cpu().numpy(), q)
        assert np.array_equal(mat.decode_weights("m").cpu().numpy().view(np.uint16), w.astype(np.float16).view(np.uint16))
        for m in (1, 3, 8, 20):
            x = rng.standard_normal((m, k)).astype(np.float32)
            y = mat.linear("m", torch.from_numpy(x).cuda()).cpu().numpy()
            assert helpers.rel_err(y, orc.gemv_f64(w, x)) <= TOL, m


# Activations at an address that only their own type allows: every kernel has its wide loads, every row count its kernel
@pytest.mark.parametrize("ty,n,k", [("Q4_K", 256, 1024), ("Q6_K", 256, 1536), ("Q5_K", 192, 256)])
@pytest.mark.parametrize("half", [True, False])
def test_unaligned_activations(lw, ty, n, k, half):
    import torch
    q, side, sym, w, rng = helpers.seeded_case(ty, n, k, seed=n + 5 * k)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    with lw.CodedMatrix(blob, n, sym.shape[1], ty, side) as mat:
        for m in (1, 2, 8, 9, 16, 33, 64, 65, 300):
            x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16 if half else np.float32)).cuda()
            want = mat.linear("m", x)
            for off in (1, 2):
                z = torch.empty(m * k + off, dtype=x.dtype, device="cuda")
                z[off:] = x.reshape(-1)
                assert torch.equal(mat.linear("m", z[off:].reshape(m, k)), want), (m, off)


def test_scratch_reused_back_to_back(lw):
    """Products in a row on one handle write and read the same scratch, each kernel set up while the one before still
    runs: every result is the one that the product gives alone."""
    import torch
    q, side, sym, w, rng = helpers.seeded_case("Q4_K", 512, 2048, seed=77)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    with lw.CodedMatrix(blob, 512, sym.shape[1], "Q4_K", side) as mat:
        xs = [torch.from_numpy(rng.standard_normal((m, 2048)).astype(np.float32)).cuda() for m in (8, 9, 33, 33, 64, 80, 80, 200)]
        want = []
        for x in xs:
            want.append(mat.linear("m", x).clone())
            torch.cuda.synchronize()
        order = rng.integers(0, len(xs), 300)
        got = [mat.linear("m", xs[i]) for i in order]
        for i, y in zip(order, got):
            assert torch.equal(y, want[i])


# Sizes whose tiles are 256 weight rows: the last one ragged (64 rows, i.e. one of its two blocks of 128 half full and the
# other empty), K split over several planes and not, one, two and three token tiles
@pytest.mark.parametrize("ty,n,k,rows,half", [("Q4_K", 4160, 14336, (80, 300), True), ("Q6_K", 9536, 4096, (257, 600), False)])
def test_gemm_with_tall_tiles(lw, ty, n, k, rows, half):
    import torch
    q, side, sym, w, rng = helpers.seeded_case(ty, n, k, seed=n + k)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    wt = torch.from_numpy(w).cuda().double()
    with lw.CodedMatrix(blob, n, sym.shape[1], ty, side) as mat:
        for m in rows:
            x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16 if half else np.float32)).cuda()
            y = torch.full((m + 1, n), -7.0, device="cuda")
            mat.linear("m", x, out=y[:m])
            assert (y[m] == -7.0).all()
            ref = x.double() @ wt.T
            assert ((y[:m] - ref).abs().amax(1) / ref.abs().amax(1)).max() <= TOL, m
