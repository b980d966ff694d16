"""The grouped product of two SMs (row tiles of 32) against float64: runs of tiles longer and shorter than a unit, groups that
come back, skipped tiles, more units than a CTA lists, widths and depths that leave features and steps over, every epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def product(x, w, group, out, **more):
    from flambeau_b200.kernels import ops
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    tiles = torch.tensor(group, dtype=torch.int32, device="cuda")
    if "activation" in more:
        ops.gemm_tc_grouped_gated(x, w, tiles, 32, out, status, more["activation"])
    else:
        ops.gemm_tc_grouped(x, w, tiles, 32, out, status, more.get("plain"))
    assert int(status) == 0
    return out


PATTERNS = {"sorted": [0] * 6 + [1] * 8 + [2] * 9 + [3] + [4] * 17 + [-1] * 3, "mixed": [2, 2, -1, 0, 2, 1, 1, -1, -1, 4, 3, 3, 3],
            "stretches": [0] * 31 + [1] * 2 + [2] * 64 + [3] * 25 + [-1] * 40 + [4] * 41 + [0] + [1] * 7 + [-1],        # (a CTA lists 32 tiles at a time)
            "one": [1], "none": [-1, -1], "many": [i % 5 for i in range(450)] + [3] * 12 + [-1, 0]}


@pytest.mark.parametrize("pattern", list(PATTERNS))
@pytest.mark.parametrize("N,K", [(64, 64), (200, 72), (256, 512), (1800, 328)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_tiles_of_groups(pattern, N, K, dtype):
    group = PATTERNS[pattern]
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(32 * len(group), K, generator=g, device="cuda").bfloat16()
    w = torch.randn(5, N, K, generator=g, device="cuda").bfloat16()
    of = torch.tensor(group, device="cuda").repeat_interleave(32)
    want = torch.empty(len(of), N, dtype=torch.float64, device="cuda")
    size = torch.empty_like(want)
    for e in range(5):
        want[of == e], size[of == e] = x[of == e].double() @ w[e].double().T, x[of == e].double().abs() @ w[e].double().abs().T
    kept = of >= 0
    out = product(x, w, group, torch.full((len(of), N), 7.0, dtype=getattr(torch, dtype), device="cuda"))
    # a float32 sum of K terms (cut off in the tensor cores), then the output's rounding
    bound = K * 2.0 ** -23 * size + (0 if dtype == "float32" else 2.0 ** -8 * want.abs())
    assert bool(((out.double() - want).abs() <= bound)[kept].all()) and bool((out[~kept] == 7.0).all())
    if dtype == "bfloat16":
        act = product(x, w, group, torch.full_like(out, 7.0), plain="relu_squared")
        ref = torch.relu(want).square()
        assert bool(((act.double() - ref).abs() <= 2 * bound * (want.abs() + bound))[kept].all()) and bool((act[~kept] == 7.0).all())
    gated = product(x, w, group, torch.full((len(of), N // 2), 7.0, dtype=out.dtype, device="cuda"), activation="silu")
    a, b, e = want[:, 0::2], want[:, 1::2], K * 2.0 ** -23 * size
    ref = torch.nn.functional.silu(a) * b
    # silu's slope is below 1.1
    bound = 1.1 * e[:, 0::2] * (b.abs() + e[:, 1::2]) + a.abs() * e[:, 1::2] + (2.0 ** -20 if dtype == "float32" else 2.0 ** -8) * ref.abs() + 1e-30
    assert bool(((gated.double() - ref).abs() <= bound)[kept].all()) and bool((gated[~kept] == 7.0).all())
