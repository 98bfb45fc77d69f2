"""Top-k / top-p sampling around the vocabulary size from which a row is shared by a cluster of blocks: the same tokens as
the plain rule, with slices of the vocabulary that hold no mass, draws at both ends, and ties that cross slices."""
import pytest
import torch

from test_kernels_gpu import ops_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8192, 8193, 8225, 151936])
def test_rows_shared_by_blocks(V):
    cu, pl = ops_pair("float32")
    g = torch.Generator().manual_seed(V)
    R = 20
    lg = torch.randn(R, V, generator=g) * 3
    lg[2, 100:] = -float("inf")              # only the first slice holds mass
    lg[3, :V - 5] = -float("inf")            # only the last one
    lg[4, 40:V - 40] = -float("inf")         # both ends
    lg[5] = 1.0                              # all equal: ties across every slice
    lg[6] = (lg[6] / 3).round()
    temp = torch.full((R,), 0.9)
    temp[7] = 0.0
    top_k = torch.tensor([0, 5, 0, 3, 60, 0, 1000, 7, 0, 1] + [0, 40] * 5, dtype=torch.int32)
    top_p = torch.tensor([0.9, 1.0, 0.5, 1.0, 0.99, 0.37, 0.8, 0.9, 1.0, 0.5] + [0.95, 0.3] * 5)
    u = torch.rand(R, generator=g, dtype=torch.float64)
    u[[2, 10, 11]] = 0.0
    u[[3, 4, 12]] = 1.0 - 2.0 ** -53
    out, ref = torch.empty(R, dtype=torch.int32, device="cuda"), torch.empty(R, dtype=torch.int32)
    cu.sample_filtered(lg.cuda(), temp.cuda(), top_k.cuda(), top_p.cuda(), u.cuda(), out)
    pl.sample_filtered(lg, temp, top_k, top_p, u, ref)
    assert out.cpu().tolist() == ref.tolist()
    # a row's token does not depend on the rows beside it
    for r in (0, 5, 6, 13):
        one = torch.empty(1, dtype=torch.int32, device="cuda")
        cu.sample_filtered(lg[r:r + 1].cuda(), temp[r:r + 1].cuda(), top_k[r:r + 1].cuda(), top_p[r:r + 1].cuda(), u[r:r + 1].cuda(), one)
        assert int(one) == int(ref[r])


@pytest.mark.parametrize("V", [12288, 12289, 24577, 98305])
def test_a_token_does_not_depend_on_the_blocks_of_its_row(V):
    """Rows of one vocabulary in steps of every size at which the blocks per row change: one token per row, whoever computes
    it, with ties that cross slices, slices without mass and a row whose largest logit is not a number."""
    cu, pl = ops_pair("float32")
    blocks = [cu.core.fz_sample_blocks(r, V) for r in (1, 14, 15, 32, 33, 74, 75, 96, 97)]
    assert blocks == {12288: [1] * 9, 12289: [2] * 6 + [1] * 3, 24577: [4] * 4 + [2] * 2 + [1] * 3,
                      98305: [8, 8, 4, 4, 2, 2, 4, 4, 1]}[V]
    g = torch.Generator().manual_seed(V)
    R = 97
    lg = torch.randn(R, V, generator=g) * 3
    lg[1] = 1.0
    lg[2] = (lg[2] / 3).round()
    lg[3, 100:] = -float("inf")
    lg[4, :V - 5] = -float("inf")
    lg[5, V // 2] = float("nan")
    temp = torch.full((R,), 0.9)
    temp[6] = 0.0
    top_k = torch.tensor([0, 0, 40, 0, 7, 0, 9] * 14, dtype=torch.int32)[:R]
    top_p = torch.tensor([0.95, 0.6, 1.0, 0.9] * 25)[:R]
    u = torch.rand(R, generator=g, dtype=torch.float64)
    ref = torch.empty(R, dtype=torch.int32)
    rest = [r for r in range(R) if r != 5]
    part = torch.empty(len(rest), dtype=torch.int32)
    pl.sample_filtered(lg[rest], temp[rest], top_k[rest], top_p[rest], u[rest], part)
    ref[rest], ref[5] = part, V // 2
    dev = [t.cuda() for t in (lg, temp, top_k, top_p, u)]
    for n in (R, 96, 75, 74, 33, 32, 15, 14, 1):
        out = torch.empty(n, dtype=torch.int32, device="cuda")
        cu.sample_filtered(*(t[:n].contiguous() for t in dev), out)
        assert out.cpu().tolist() == ref[:n].tolist(), f"{n} rows"
