"""The float32 product on the tensor cores (every float32 as three bfloat16 numbers) against float64: row counts around its
token tiles, widths and depths that leave rows, columns, sums and shares of K over, rows on any border; that a row's result
is the same bits whatever the number of rows; what infinities, NaN and the smallest numbers become."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ROWS = (330, 301, 257, 129, 128, 113, 112, 64, 17, 16, 9, 1)


def product(a, w, out=None):
    from flambeau_b200.engine.runtime import Workspace
    from flambeau_b200.kernels import ops
    out = torch.full((a.shape[0], w.shape[0]), float("nan"), device="cuda") if out is None else out
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert ops.f32_tc_supported(a, w, out)
    ops.gemm_f32_tc(a, w, out, status, Workspace("cuda"))
    assert int(status) == 0
    return out


@pytest.mark.parametrize("K", [512, 516, 548, 1060, 2048])
@pytest.mark.parametrize("N", [64, 129, 700, 6144, 18900])
def test_rows(N, K):
    from flambeau_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w = torch.randn(ROWS[0], K + 5, generator=g, device="cuda")[:, :K], torch.randn(N, K + 4, generator=g, device="cuda")[:, :K]
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    whole = product(a, w)
    # What is left out of a product is below 2^-25 of it.  A term passes at most four cut-off sums of the tensor cores
    # (2^-23 each) and one addition per 64 and per 512 of K.
    assert bool(((whole.double() - want).abs() <= (5 + K / 64 + K / 512) * 2.0 ** -23 * size).all())
    plain = torch.empty_like(whole)
    ops.gemm_simt(a, w, plain)
    assert (whole.double() - want).norm() <= (plain.double() - want).norm()
    for M in ROWS[1:]:
        assert torch.equal(product(a[:M], w), whole[:M]), "a row's bits depend on the number of rows"
    assert torch.equal(product(a[:9].contiguous(), w), whole[:9])                 # (rows on 16-byte borders)


@pytest.mark.parametrize("M", [40, 3])                                            # (in one CTA, and K split over several)
@pytest.mark.parametrize("N", [20000, 256])
def test_numbers_without_parts(M, N):
    from flambeau_b200.kernels import ops
    K = 1024
    g = torch.Generator(device="cuda").manual_seed(M)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    for r, f in ((0, 0.0), (1, 1e-33), (2, 1e36)):
        a[r] *= f
    if M > 3:
        a[4, 7], a[5, 9], a[6, 0] = float("inf"), float("nan"), -float("inf")
        a[8], a[9], a[10] = 3.39e38, 1e-42, 1e38
    w[10, 3], w[11], w[12], w[13, 100] = -float("inf"), w[11] * 1e-35, 1.0, float("nan")
    got, want = product(a, w), torch.empty(M, N, device="cuda")
    ops.gemm_simt(a, w, want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fine = torch.isfinite(want)
    assert torch.equal(got[~fine & ~torch.isnan(want)], want[~fine & ~torch.isnan(want)])
    size = a.double().abs() @ w.double().abs().T
    err = (got.double() - want.double()).abs()
    # (both lie within their own bounds of the exact values; below the normal range half of the smallest number an addition)
    assert bool((err[fine] <= ((5 + K / 64 + K / 512) * 2.0 ** -23 + (K / 2 + 2) * 2.0 ** -24) * size[fine] + K * 2.0 ** -149).all())


def test_engines_on_two_streams():
    """Products whose shares of K meet in scratch, on two streams at a time: the scratch is an arena's, not the device's."""
    from flambeau_b200.engine.runtime import Workspace
    from flambeau_b200.kernels import ops
    M, N, K, times = 8, 512, 8192, 60
    g = torch.Generator(device="cuda").manual_seed(0)
    side = []
    for _ in range(2):
        a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
        side.append((a, w, product(a, w), torch.zeros(times, M, N, device="cuda"), Workspace("cuda"), torch.cuda.Stream(),
                     torch.zeros(1, dtype=torch.int32, device="cuda")))
    assert ops.lib().fb_gemm_f32_tc_scratch_floats(M, N, K, Workspace.COUNTERS) > 0, "K is to be split"
    torch.cuda.synchronize()
    for i in range(times):
        for a, w, _, outs, ws, stream, status in side:
            with torch.cuda.stream(stream):
                ops.gemm_f32_tc(a, w, outs[i], status, ws)
    torch.cuda.synchronize()
    for _, _, want, outs, ws, _, status in side:
        assert int(status) == 0 and not bool(ws.counters.any())
        assert torch.equal(outs, want.expand_as(outs))


def test_contexts_without_an_arena():
    """What has no arena to split its rows in is multiplied on the CUDA cores, as before."""
    from types import SimpleNamespace
    from flambeau_b200.kernels import ops
    a, w = torch.randn(3, 512, device="cuda"), torch.randn(64, 512, device="cuda")
    out, want = torch.empty(3, 64, device="cuda"), torch.empty(3, 64, device="cuda")
    ops.linear(a, w, out, SimpleNamespace(runtime=SimpleNamespace(status=torch.zeros(1, dtype=torch.int32, device="cuda"))))
    ops.gemm_simt(a, w, want)
    assert torch.equal(out, want)
