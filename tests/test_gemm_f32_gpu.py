"""The staged float32 product against float64: row counts around its tiles, widths and depths that leave rows, columns and
steps over, row strides; and that a row's result is the same bits whatever the number of rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [4, 60, 100, 516])
@pytest.mark.parametrize("N", [1, 33, 130, 700, 6144])
def test_rows_of_float32_products(N, K):
    from flambeau_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    most = 330
    a, w = torch.randn(most, K + 8, generator=g, device="cuda")[:, :K], torch.randn(N, K + 4, generator=g, device="cuda")[:, :K]
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    whole = None
    for M in (most, 301, 129, 128, 65, 64, 33, 17, 16, 9, 8, 1):
        out = torch.full((M, N), float("nan"), device="cuda")
        ops.gemm_simt(a[:M], w, out)
        # at most K / 2 + 2 roundings of 2^-24 of what has been added up, which the sum of the terms' sizes bounds
        assert bool(((out.double() - want[:M]).abs() <= (K / 2 + 2) * 2.0 ** -24 * size[:M]).all())
        whole = out if whole is None else whole
        assert torch.equal(out, whole[:M]), "a row's bits depend on the number of rows"
