"""Float32 attention on the tensor cores (heads of 128) against float64, where its tiles end: CTAs of 128 rows and of the 32 up to
which other warps help to fetch, groups that do not divide 128, tiles of 64 keys, stretches of 256, windows, page sizes that tiles
do not fit, compact tables, and numbers without three bfloat16 parts."""
import pytest
import torch

from test_attention_gpu import Scene

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(sc, nh, nkv, window, extras, spoil=None, all_or_nothing=()):
    """The kernel's rows, those of float64 and what a row may miss them by.  all_or_nothing: keys of the first request whose scores are
    so large that their weights are 1 or 0 whatever is lost of them."""
    from flambeau_b200.kernels import ops
    k, v = [x.clone() for x in sc.k], [x.clone() for x in sc.v]
    k_pool, v_pool = sc.k_pool.clone(), sc.v_pool.clone()
    if spoil:
        spoil(k, v)
        for s, (cached, new) in enumerate(sc.seqs):
            for t in range(cached + new):
                page = int(sc.table[s, t // sc.ps - (int(sc.table_base[s]) if sc.table_base is not None else 0)]) if not window else -1
                if page >= 0:
                    k_pool[page, :, t % sc.ps], v_pool[page, :, t % sc.ps] = k[s][t], v[s][t]
    g, n = torch.Generator().manual_seed(3), sc.q_flat.shape[0]
    sinks = torch.randn(nh, generator=g) if extras else None
    gate = torch.randn(2, n, nh + 3, generator=g) if extras else None
    out, status = torch.full((n, nh * 128), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    lens = [m for _, m in sc.seqs]
    dev_gate = gate.to(DEV) if extras else None
    ops.paged_attention_f32(
        sc.q_flat.to(DEV), out, k_pool.to(DEV), v_pool.to(DEV), sc.table.to(DEV), sc.seq_q_start.to(DEV), sc.seq_q_len.to(DEV),
        sc.seq_pos_start.to(DEV), len(lens), max(lens), max(c + m for c, m in sc.seqs), True, True, nh, nkv, 128, window, 128 ** -0.5,
        status, vd=128, sinks=sinks.to(DEV) if extras else None, seq_lens=lens,
        table_base=sc.table_base.to(DEV) if sc.table_base is not None else None,
        head_gate=(dev_gate[0][:, :nh], 2, dev_gate.stride(0)) if extras else None)
    assert int(status.item()) == 0
    want, bound = [], []
    for s, (cached, new) in enumerate(sc.seqs):
        G, T = nh // nkv, cached + new
        q, kk, vv = sc.q[s].double(), k[s].double().repeat_interleave(G, 1), v[s].double().repeat_interleave(G, 1)
        t, p = torch.arange(T), torch.arange(cached, T)
        seen = (t[None] <= p[:, None]) & ((t[None] > p[:, None] - window) if window else torch.ones(1, 1, dtype=torch.bool))
        scores = torch.einsum("qhd,thd->hqt", q, kk) * 128 ** -0.5
        scores = scores.masked_fill(~seen, -torch.inf)
        if extras:
            scores = torch.cat([scores, sinks.double()[:, None, None].expand(nh, new, 1)], -1)
        weights = scores.softmax(-1)[..., :T]
        o = torch.einsum("hqt,thd->qhd", weights.masked_fill(~seen, 0.0), vv)
        # A score is off by what eight blocks of 16 products lose, of the sum of their magnitudes; so is a weight, twice (its sum too);
        # a sum of 64 weighted values loses as many roundings again, of the values' sum of magnitudes.
        size = torch.einsum("qhd,thd->hqt", q.abs(), kk.abs()) * 128 ** -0.5
        if s == 0:
            size[..., list(all_or_nothing)] = 0.0
        off = 2.0 ** -23 * (2 * 8 * size.masked_fill(~seen, 0.0).amax(-1) + 64)
        most = torch.einsum("hqt,thd->qhd", weights.masked_fill(~seen, 0.0), vv.abs())
        factor = torch.sigmoid(gate[:, sc_rows(sc, s), :nh].double().sum(0))[..., None] if extras else 1.0
        want.append(o * factor)
        bound.append((off.transpose(0, 1)[..., None] * most + T * 2.0 ** -149) * factor)      # (below the normal range half a step a sum)
    return out.view(n, nh, 128).double().cpu(), torch.cat(want), torch.cat(bound)


def sc_rows(sc, s):
    start = int(sc.seq_q_start[s])
    return slice(start, start + sc.seqs[s][1])


SEQS = {"tiles": [(0, 1), (63, 1), (255, 2), (192, 65)], "few": [(700, 8), (64, 9), (0, 7)], "portion": [(37, 129)], "decode": [(900, 1), (31, 1)]}


@pytest.mark.parametrize("options", ["plain", "window", "extras"])
@pytest.mark.parametrize("seqs", list(SEQS))
@pytest.mark.parametrize("heads", [(1, 1), (4, 1), (6, 2), (64, 1)], ids=str)
def test_against_float64(heads, seqs, options):
    nh, nkv = heads
    window = 90 if options == "window" else 0
    sc = Scene(SEQS[seqs], nh, nkv, 128, window, torch.float32, page_size={1: 16, 4: 24, 3: 5, 64: 128}[nh // nkv], seed=nh, compact=bool(window))
    got, want, bound = run(sc, nh, nkv, window, options == "extras")
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / bound).max())


def test_a_key_without_parts():
    """A key of 1e20: its score is the largest there is, or the least, and its weight all or nothing."""
    def spoil(k, v):
        k[0][70] *= 1e20
    sc = Scene([(300, 90), (0, 50)], 4, 2, 128, 0, torch.float32, seed=5)
    got, want, bound = run(sc, 4, 2, 0, False, spoil, all_or_nothing=[70])
    assert bool(((got - want).abs() <= bound).all())


def test_a_value_without_parts():
    """A value of 1e25 beside ordinary ones and behind some rows' positions."""
    def spoil(k, v):
        v[0][200] *= 1e25
        v[1][40] *= 1e25
    sc = Scene([(300, 90), (0, 50)], 4, 2, 128, 0, torch.float32, seed=5)
    got, want, bound = run(sc, 4, 2, 0, False, spoil)
    assert bool(((got - want).abs() <= bound).all()) and float(want[90:130].abs().max()) < 1e3


@pytest.mark.parametrize("power", [-60, -83, -100, -110, -121])
@pytest.mark.parametrize("beside", ["nothing", "zeros", "ordinary channels", "a value of 1e17"])
def test_results_scale_with_the_values(power, beside):
    """Values smaller by a power of two give the same bits as much smaller, down to where a value's lowest part lies below
    bfloat16's range, whatever lies beside them in their tile."""
    def spoil(factor):
        def change(k, v):
            for x in v:
                x[..., :64] *= factor
            if beside == "zeros":
                v[0][..., 40:], v[1][..., ::2] = 0.0, 0.0
            elif beside == "a value of 1e17":
                v[0][250, :, 100], v[1][20, :, 100] = 1e17, -1e17
            elif beside == "nothing":
                v[0][..., 64:], v[1][..., 64:] = v[0][..., :64], v[1][..., :64]
        return change
    sc = Scene([(300, 90), (0, 50)], 4, 2, 128, 0, torch.float32, seed=5)
    got, whole = (run(sc, 4, 2, 0, False, spoil(2.0 ** p))[0][..., :64] for p in (power, 0))
    # (below the normal range half a step of 2^-149 for each rounding: of the value, two a tile of seven, three a stretch of two)
    assert bool(((got - whole * 2.0 ** power).abs() <= 11 * 2.0 ** -149).all()), float(((got - whole * 2.0 ** power).norm() / got.norm()))


def test_numbers_that_a_row_does_not_see():
    sc = Scene([(100, 60)], 4, 2, 128, 0, torch.float32, seed=6)

    def later(k, v):
        k[0][140], v[0][141] = float("nan"), float("inf")       # rows before position 140 do not see them
    (got, _, _), (_, want, bound) = run(sc, 4, 2, 0, False, later), run(sc, 4, 2, 0, False)
    assert bool(((got - want).abs() <= bound)[:40].all()) and bool(got[40:].isnan().all())
