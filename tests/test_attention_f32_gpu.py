"""The tiled float32 attention against the kernel that takes a row and head at a time, over every form both accept: head and
value sizes, groups of 1 to 64 query heads, portions beside decoded tokens, stretches of keys that are merged, windows that
keep first keys, sinks, caps, gates as shares, slopes, a missing page, and a later token's NaN that earlier rows must not see."""
import pytest
import torch

from test_attention_gpu import Scene

pytestmark = pytest.mark.gpu
DEV = "cuda"

SIZES = [(32, 8, 128, 128), (4, 2, 24, 24), (6, 3, 40, 72), (32, 1, 64, 64), (2, 1, 256, 256), (64, 1, 20, 12), (3, 3, 4, 4), (34, 2, 128, 64)]
SEQS = {"mixed": [(0, 1), (500, 1), (37, 70), (129, 200), (5, 4), (63, 65)], "decoding": [(900, 1), (31, 1), (32, 1)], "portion": [(0, 33)]}


def both(sc, vd, options, poison=None, drop_page=None, slope=None):
    from flambeau_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    v_pool = torch.randn(*sc.k_pool.shape[:3], vd, generator=g)
    k, v, table = sc.k_pool.nan_to_num(0.0).to(DEV), v_pool.to(DEV), sc.table.clone()
    if poison is not None:                             # a position of the last sequence whose value is not a number
        v[int(sc.table[-1, poison // sc.ps]), :, poison % sc.ps] = float("nan")
    if drop_page is not None:
        table[drop_page] = -1
    table, q = table.to(DEV), sc.q_flat.to(DEV)
    n = q.shape[0]
    kw = dict(vd=vd)
    if "window" in options:
        kw.update(keep_first=7)
    if "extras" in options:
        gate = torch.randn(2, n, sc.nh + 3, generator=g).to(DEV)
        kw.update(softcap=20.0, sinks=torch.randn(sc.nh, generator=g).to(DEV), head_gate=(gate[0][:, :sc.nh], 2, gate.stride(0)),
                  score_slopes=(-torch.rand(sc.nh, generator=g) * 0.05).to(DEV))
    if slope is not None:
        kw.update(score_slopes=torch.full((sc.nh,), slope, device=DEV))
    window, scale = 50 if "window" in options else 0, 2.0 * sc.hd ** -0.5
    outs, flags = [], []
    lens = [m for _, m in sc.seqs]
    G = sc.nh // sc.nkv
    for tiled in (False, True):
        out, status = torch.full((n, sc.nh * vd), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        if tiled:
            short = [G <= 16 and m * G <= 16 for m in lens]
            ops.paged_attention_f32(q, out, k, v, table, sc.seq_q_start.to(DEV), sc.seq_q_len.to(DEV), sc.seq_pos_start.to(DEV),
                                    len(lens), max(lens), max(c + m for c, m in sc.seqs), any(short), not all(short), sc.nh, sc.nkv,
                                    sc.hd, window, scale, status, **kw)
        else:
            ops.paged_attention_simt(q, out, k, v, table, sc.positions.to(DEV), sc.row_seq.to(DEV), sc.nh, sc.nkv, sc.hd, window,
                                     scale, status, **kw)
        outs.append(out.double().cpu())
        flags.append(int(status.item()))
    return outs, flags


@pytest.mark.parametrize("options", ["plain", "window", "extras", "window extras"])
@pytest.mark.parametrize("seqs", list(SEQS))
@pytest.mark.parametrize("sizes", SIZES, ids=str)
def test_tiles_equal_rows(sizes, seqs, options):
    nh, nkv, hd, vd = sizes
    sc = Scene(SEQS[seqs], nh, nkv, hd, 0, torch.float32, seed=hd)
    (a, b), flags = both(sc, vd, options)
    assert flags == [0, 0] and bool(torch.isfinite(b).all())
    # two orders of float32 sums over at most 900 keys and 256 channels
    assert float((a - b).abs().max() / a.abs().max()) < 5e-6


def test_a_later_value_that_is_no_number_and_a_missing_page():
    sc = Scene([(3, 90)], 8, 2, 64, 0, torch.float32, seed=1)
    (a, b), _ = both(sc, 64, "plain", poison=60)
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and bool(torch.isfinite(b[:57]).all()) and bool(torch.isnan(b[57:]).all())
    (a, b), flags = both(sc, 64, "plain", drop_page=(0, 2))
    assert flags[0] == flags[1] != 0 and float((a - b).abs().max() / a.abs().max()) < 5e-6


def test_a_seen_value_that_is_no_number_reaches_every_row_that_sees_it():
    """Scores fall by 20 a position, so most rows weigh the key at position 10 by exactly 0; it is seen all the same, in tiles
    that a row sees whole and in those it does not."""
    sc = Scene([(3, 90)], 8, 2, 64, 0, torch.float32, seed=2)
    (a, b), _ = both(sc, 64, "plain", poison=10, slope=-20.0)
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and bool(torch.isfinite(b[:7]).all()) and bool(torch.isnan(b[7:]).all())


def test_more_sequences_times_heads_than_a_grid_has_rows():
    """33,000 decoded tokens of two key/value heads (three sequences over and over); the row-wise kernel takes them in one
    launch."""
    sc, n = Scene([(0, 1), (5, 1), (2, 1)], 2, 2, 4, 0, torch.float32, seed=3, page_size=4), 33000
    sc.seqs, sc.table = sc.seqs * (n // 3), sc.table.repeat(n // 3, 1)
    sc.positions, sc.seq_pos_start, sc.seq_q_len = (t.repeat(n // 3) for t in (sc.positions, sc.seq_pos_start, sc.seq_q_len))
    sc.row_seq = sc.seq_q_start = torch.arange(n, dtype=torch.int32)
    sc.q_flat = torch.randn(n, sc.nh * sc.hd, generator=torch.Generator().manual_seed(4))
    (a, b), flags = both(sc, 4, "plain")
    assert flags == [0, 0] and float((a - b).abs().max() / a.abs().max()) < 5e-6


def rows_of(sc, keep, longest, seq_lens=True, cut=None, window=0, vd=None):
    """The tiled kernel's output for the sequences `keep` of a scene, alone in a step; cut: (sequence, rows) whose portion is only
    its rows from there on."""
    from flambeau_b200.kernels import ops
    vd = vd or sc.hd
    g = torch.Generator().manual_seed(7)
    v = torch.randn(*sc.k_pool.shape[:3], vd, generator=g).to(DEV)
    lens, starts = sc.seq_q_len[keep].clone(), [int(sc.seq_q_start[s]) for s in keep]
    pos = sc.seq_pos_start[keep].clone()
    if cut is not None:
        lens[0], starts[0], pos[0] = lens[0] - cut, starts[0] + cut, pos[0] + cut
    rows = torch.cat([torch.arange(a, a + int(m)) for a, m in zip(starts, lens)])
    q_start = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    q = sc.q_flat[rows].to(DEV)
    out, status = torch.full((len(rows), sc.nh * vd), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    G = sc.nh // sc.nkv
    short = [G <= 16 and m * G <= 16 for m in lens.tolist()]
    sinks = torch.randn(sc.nh, generator=g).to(DEV)
    ops.paged_attention_f32(q, out, sc.k_pool.nan_to_num(0.0).to(DEV), v, sc.table[keep].to(DEV), q_start.to(DEV), lens.to(DEV), pos.to(DEV),
                            len(keep), int(lens.max()), longest, any(short), not all(short), sc.nh, sc.nkv, sc.hd, window, sc.hd ** -0.5,
                            status, vd=vd, sinks=sinks, keep_first=40 if window else 0, seq_lens=lens.tolist() if seq_lens else None)
    assert int(status.item()) == 0 and bool(torch.isfinite(out).all())
    return out, q_start.tolist(), lens.tolist()


@pytest.mark.parametrize("window", [0, 700, 90])
@pytest.mark.parametrize("sizes", [(8, 2, 64, 64), (32, 8, 128, 128), (16, 1, 256, 256), (20, 1, 20, 12), (3, 3, 40, 72)], ids=str)
def test_a_row_has_the_same_bits_whatever_shares_its_step(sizes, window):
    """Decoded tokens and portions alone, together, beside many others, with other bounds on the longest context (which decide
    over how many CTAs the keys are cut), and the last row of a portion as a token of its own."""
    nh, nkv, hd, vd = sizes
    seqs = [(2600, 1), (511, 1), (256, 300), (1000, 71), (37, 5), (0, 1)]      # (an odd number of rows, heads and stretches once)
    sc = Scene(seqs, nh, nkv, hd, 0, torch.float32, seed=hd)
    everyone = list(range(len(seqs)))
    whole, start, lens = rows_of(sc, everyone, 2601, window=window, vd=vd)
    for s in everyone:
        mine = whole[start[s]:start[s] + lens[s]]
        for keep, longest in (([s], sum(seqs[s])), ([s], 32768), ([s] + everyone[::2] + everyone, 4000)):
            got, at, _ = rows_of(sc, keep, max(longest, max(sum(seqs[k]) for k in keep)), seq_lens=longest != 4000, window=window, vd=vd)
            assert torch.equal(got[at[0]:at[0] + lens[s]], mine), (s, keep, longest)
        if lens[s] > 1:
            for cut in (lens[s] - 1, lens[s] // 3):
                got, _, _ = rows_of(sc, [s], 2601, cut=cut, window=window, vd=vd)
                assert torch.equal(got, mine[cut:]), (s, cut)


def test_replayed_decode_steps_across_the_ends_of_stretches(tmp_path):
    """Two requests decode past positions 256 and 512 from one captured graph, whose stretches were laid out for the longest
    context that the engine allows: the same bits as step by step without graphs and in another company."""
    import tiny
    from flambeau_b200.engine.batch import Entry
    from flambeau_b200.engine.step import Engine, EngineOptions
    cfg = dict(tiny.CONFIGS["A"], sliding_window=None)
    folder = tiny.make_folder(tmp_path / "m", cfg, seed=3, dtype="float32")
    toks = tiny.random_requests(cfg, [262, 518], seed=5)
    got = {}
    for graphs, longest in ((True, 3000), (False, 3000), (False, 600)):
        engine = Engine.from_folder(folder, EngineOptions(dtype="float32", cache_tokens=6400, max_requests=2, max_step_tokens=1024,
                                                          max_seq_len=longest, cuda_graphs=graphs))
        engine.step([Entry("a", toks["r0"][:250], [249]), Entry("b", toks["r1"][:506], [505])])
        got[graphs, longest] = [engine.step([Entry("a", [toks["r0"][250 + t]], [0]), Entry("b", [toks["r1"][506 + t]], [0])]).clone()
                                for t in range(12)]
        engine.runtime.check_status("decode")
    for steps in list(got.values())[1:]:
        for x, y in zip(got[True, 3000], steps):
            assert torch.equal(x, y)
    alone = Engine.from_folder(folder, EngineOptions(dtype="float32", cache_tokens=6400, max_requests=2, max_step_tokens=1024,
                                                     max_seq_len=3000, cuda_graphs=False))
    alone.step([Entry("b", toks["r1"][:100], [])])
    alone.step([Entry("b", toks["r1"][100:506], [405])])
    for t in range(12):
        assert torch.equal(alone.step([Entry("b", [toks["r1"][506 + t]], [0])])[0], got[True, 3000][t][1])
