"""Differential attention over portions with maps of 64 and values of 128, the sizes of the tcgen05 kernel, on that kernel and
with it switched off (the mma.sync kernel): one to 32 query heads a key/value head, portions around the edges of its 128 rows and 64-key tiles, windows, pages of 8 to 64 keys, with and
without a gate per head; planted keys at the windows' edges, poison in every slot that was not written."""
import pytest
import torch

import zedivik_tiny as zt
from test_zedivik_gpu import rel_err

pytestmark = pytest.mark.gpu

SEQS = [(0, 130), (70, 64), (37, 33), (200, 1), (129, 200), (5, 17)]


@pytest.fixture(params=[True, False], ids=["tcgen05", "mma_sync"])
def portion_kernel(request):
    from flambeau_b200.kernels import ops
    ops.set_attention_tc(request.param)
    yield request.param
    ops.set_attention_tc(True)


def portions(case, gate, out_scale, nh, nkv, window, scale, lam, eps):
    from flambeau_b200.kernels import ops
    out = torch.full((case.n, nh * 128), float("nan"), dtype=torch.bfloat16, device="cuda:0")
    status = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    ops.diff_attention_mma(case.q_d, out, gate, case.cache, case.seq_q_start, case.seq_q_len, case.seq_pos_start, len(SEQS),
                           case.max_q_len, case.max_kv_len, case.any_short, case.any_long, nh, nkv, 64, 128, window, scale, lam,
                           eps, out_scale, status)
    assert int(status.item()) == 0 and bool(torch.isfinite(out.float()).all())
    return out


@pytest.mark.parametrize("geometry", [(8, 2, 0, 16), (4, 4, 33, 16), (12, 1, 100, 64), (32, 1, 40, 8), (3, 1, 64, 32)], ids=str)
@pytest.mark.parametrize("gated", [True, False])
def test_portions_of_two_maps(portion_kernel, geometry, gated):
    nh, nkv, window, page = geometry
    case = zt.PagedCase(SEQS, nh=nh, nkv=nkv, kd=64, vd=128, window=window, page_size=page, dtype=torch.bfloat16, device="cuda:0",
                        seed=nh + window)
    scale, lam, diff, eps = 0.3, 0.62, 0.35, 1e-5
    out = portions(case, case.gate_d if gated else None, 1.0 - diff, nh, nkv, window, scale, lam, eps)
    want = case.expected(scale=scale, lam=lam, diff=diff, eps=eps)
    if not gated:
        want = (want.view(case.n, nh, 128) / case.gate_d.double().cpu()[:, :, None]).view(case.n, -1)
    assert rel_err(out, want) < 8e-3                   # the tolerance of the other arrangements' tests


def test_the_switch_reaches_differential_portions():
    """The two kernels move their reference points at other keys, so some of 800,000 roundings differ; the same bits would
    mean that both runs took one kernel."""
    from flambeau_b200.kernels import ops
    case = zt.PagedCase(SEQS, nh=16, nkv=4, kd=64, vd=128, window=0, page_size=16, dtype=torch.bfloat16, device="cuda:0", seed=5)
    outs = []
    for on in (True, False):
        ops.set_attention_tc(on)
        try:
            outs.append(portions(case, None, 0.65, 16, 4, 0, 0.125, 0.62, 1e-5))
        finally:
            ops.set_attention_tc(True)
    assert not torch.equal(*outs)


def exact(case, scale, lam, diff, eps):
    """The difference of the two maps' outputs, normed, in float64 on the GPU; no gate, no window."""
    rows = []
    for s, (ctx, n) in enumerate(case.seqs):
        q, k, v = (t[s].cuda() for t in (case.q, case.k, case.v))
        seen = torch.arange(ctx + n, device="cuda")[None] <= torch.arange(ctx, ctx + n, device="cuda")[:, None]
        o = torch.empty(n, case.nh, case.vd, dtype=torch.float64, device="cuda")
        for h in range(case.nh):
            g = h // (case.nh // case.nkv)
            a = [torch.softmax(((q[:, h, m] @ k[:, g, m].T) * scale).masked_fill(~seen, float("-inf")), -1) @ v[:, g] for m in (0, 1)]
            d = a[0] - lam * a[1]
            o[:, h] = d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * (1.0 - diff)
        rows.append(o.reshape(n, -1))
    return torch.cat(rows)


def test_weights_lose_no_more_than_on_the_mma_sync_kernel():
    """Uneven weights: how many results are not the rounding of the exact ones.  Every weight's own error makes some results
    cross a border between two bfloat16 numbers; the largest weight of a row, which counts most, has none where it is 1."""
    from flambeau_b200.kernels import ops
    case = zt.PagedCase([(300, 700)], nh=16, nkv=4, kd=64, vd=128, window=0, page_size=16, dtype=torch.bfloat16, device="cuda:0",
                        seed=4, plant=False)
    want, wrong = exact(case, 0.3, 0.62, 0.35, 1e-5).float().bfloat16(), []
    for on in (True, False):
        ops.set_attention_tc(on)
        try:
            out = torch.empty((case.n, 16 * 128), dtype=torch.bfloat16, device="cuda:0")
            status = torch.zeros(1, dtype=torch.int32, device="cuda:0")
            ops.diff_attention_mma(case.q_d, out, None, case.cache, case.seq_q_start, case.seq_q_len, case.seq_pos_start, 1,
                                   case.max_q_len, case.max_kv_len, False, True, 16, 4, 64, 128, 0, 0.3, 0.62, 1e-5, 0.65, status)
            assert int(status.item()) == 0
            wrong.append(int((out != want).sum()))
        finally:
            ops.set_attention_tc(True)
    # (counts of rare events: three standard deviations of their difference)
    assert wrong[0] <= wrong[1] + 3.0 * sum(wrong) ** 0.5, wrong
