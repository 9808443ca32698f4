"""Products that a caller has captured into a CUDA graph: the scratch that the graph holds stays where it is, whatever is
run on the handle between capture and replay."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


# 33 rows: decode + tcgen05; 80 rows: decode to weights and GEMM; 20 rows of 256 columns: the same, the shape the fused kernel refuses
@pytest.mark.parametrize("ty,n,k,rows", [("Q4_K", 512, 1024, 33), ("Q6_K", 256, 1536, 80), ("Q5_K", 192, 256, 20)])
def test_replay_after_a_larger_product(ty, n, k, rows):
    helpers.build_library()
    import torch
    import lazyweights_b200 as lw
    q, side, sym, w, rng = helpers.seeded_case(ty, n, k, seed=n + k)
    blob, _, _ = lw.bundle.encode_huf8(sym)
    with lw.CodedMatrix(blob, n, sym.shape[1], ty, side) as mat:
        x = torch.from_numpy(rng.standard_normal((rows, k)).astype(np.float32)).cuda()
        y = torch.empty((rows, n), device="cuda")
        want = mat.linear("m", x).clone()                       # allocates what the product needs
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            mat.linear("m", x, out=y)
        for more in (300, 700, 2500):                           # larger activations, then more row factors
            big = torch.from_numpy(rng.standard_normal((more, k)).astype(np.float32)).cuda()
            first = mat.linear("m", big)
            y.zero_()
            graph.replay()
            assert torch.equal(y, want), more
            assert torch.equal(mat.linear("m", big), first), more
    assert lw.lib().lw_kernel_error() == 0
