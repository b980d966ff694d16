"""The two-SM product at row counts that its token tiles (32 to 256 rows wide) divide evenly, by one row more and by one less:
whole sums, shares of K, sums added to the output, activations; features and steps left over."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [129, 160, 161, 192, 224, 225, 257, 300, 384, 385, 513, 537, 577, 1029])
@pytest.mark.parametrize("N,K", [(2560, 520), (3112, 1096)])
def test_row_counts(M, N, K):
    from flambeau_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    err = K * 2.0 ** -23 * size                         # K additions of float32, cut off in the tensor cores
    for most in (1, 4):
        slabs = torch.full((most, M, N), float("nan"), device="cuda")
        parts = ops.gemm_tc(x, w, slabs[0], status, slabs=slabs)
        assert 1 <= parts <= most and bool(((slabs[:parts].double().sum(0) - want).abs() <= err).all())
    acc = torch.ones(M, N, device="cuda")
    if ops.gemm_tc_add(x, w, acc, status):
        assert bool(((acc.double() - 1 - want).abs() <= err + 2.0 ** -23 * (1 + want.abs())).all())
    half = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc(x, w, half, status)
    assert bool(((half.double() - want).abs() <= err + 2.0 ** -8 * want.abs()).all())
    ops.gemm_tc_act(x, w, half, status, "relu_squared")
    ref = torch.relu(want).square()
    assert bool(((half.double() - ref).abs() <= err * (2 * want.abs() + err) + 2.0 ** -8 * (ref + err * (2 * want.abs() + err))).all())
    gated = torch.empty(M, N // 2, device="cuda")
    ops.gemm_tc_gated(x, w, gated, status)
    a, b, e = want[:, 0::2], want[:, 1::2], err
    ref = torch.nn.functional.silu(a) * b               # (silu's slope is below 1.1)
    assert bool(((gated.double() - ref).abs() <= 1.1 * e[:, 0::2] * (b.abs() + e[:, 1::2]) + a.abs() * e[:, 1::2] + 2.0 ** -20 * ref.abs() + 1e-30).all())
    assert int(status) == 0
