"""The float32 path's product at the sizes where its rules change hands: few rows and tiles of rows, one chunk of k and
many, one group of chunks and eight. Every result against 64-bit arithmetic within a bound from the order of the sums, and
the same bits whoever computes it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def cuda():
    from fusezap_core_b200.kernels import cuda_ops
    return cuda_ops("float32")


@pytest.mark.parametrize("N,K", [(1, 1), (9, 33), (96, 31), (130, 1024), (64, 1028), (4097, 136), (200, 2050), (896, 4864), (16385, 256)])
def test_linear(N, K):
    cu = cuda()
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn(200, K, generator=g, device="cuda")
    w = torch.randn(N, K, generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda")
    exact = a.double() @ w.double().T + bias.double()
    # a chain of K / 32 (rounded up to a multiple of 32) fmaf, at most 32 + 8 additions and the bias, each rounding by
    # 2^-24 of a partial sum that is at most the sum of magnitudes
    steps = 32 * -(-K // 1024) + 41
    bound = steps * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double())
    full = torch.empty(200, N, device="cuda")
    cu.linear(a, w, bias, full)
    assert bool(((full.double() - exact).abs() <= bound).all())
    for rows in (1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 129):
        part = torch.full((rows + 1, N), float("nan"), device="cuda")
        cu.linear(a[7:7 + rows].contiguous(), w, bias, part[:rows])
        assert torch.equal(part[:rows], full[7:7 + rows]), f"{rows} rows"
        assert bool(part[rows].isnan().all()), f"{rows} rows: written beyond the last"
    # operands off the 16-byte boundaries: read one by one, the same bits
    off_a, off_w = torch.empty(5 * K + 1, device="cuda")[1:].view(5, K), torch.empty(N * K + 1, device="cuda")[1:].view(N, K)
    off_a.copy_(a[:5])
    off_w.copy_(w)
    part = torch.empty(5, N, device="cuda")
    cu.linear(off_a, off_w, bias, part)
    assert torch.equal(part, full[:5])
    # an infinity stays in its own row and column
    bad = a[:20].clone()
    bad[3, K // 2] = float("inf")
    out = torch.empty(20, N, device="cuda")
    cu.linear(bad, w, bias, out)
    assert torch.equal(out[:3], full[:3]) and torch.equal(out[4:], full[4:20]) and not bool(out[3].isfinite().any())
